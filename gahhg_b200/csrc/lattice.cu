// lattice.cu - exact-label query index and query kernel.
//
// The reference answers a query by descending the hexagon hierarchy from 42
// level-0 cells (kernel_PISP, source/GPISPAHHG.cu:1422-1504): about ten
// dependent levels of plane tests per point.  Here the same question is
// answered from a lattice over longitude/latitude that is indexed directly
// from the input coordinates // (the lattice itself, and how it is built: lattice_build.cu.)
//
// A query reads lon/lat (16 B), computes the top cell with two FP64
// multiply-adds, follows inner nodes by exact power-of-two scaling, and
//   - in a cell without edges writes the cell's label (no trigonometry);
//   - in a leaf counts crossings of arc(R, q) with the leaf's edges:
//       s2 = orient(A,B,q) = q.(A x B), s3 = orient(R,q,A) = q.(A x R),
//       s4 = orient(R,q,B) = q.(B x R), s1 = orient(A,B,R) stored exactly;
//     each sign is first taken in FP32 (q from __sincosf, vectors rounded to
//     FP32) against a forward error bound, then in FP64 on the canonical q,
//     then exactly (exact_pred.cuh).  Labels are therefore those of the exact
//     oracle; the FP32 stage only decides when its bound proves the sign.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

#include "exact_pred.cuh"
#include "lattice.cuh"
#include "local_frame.cuh"

namespace gahhg {

namespace {

constexpr int TPB = 256;
inline int blocks_for(long long n) { return (int)std::max(1LL, (n + TPB - 1) / TPB); }

// ------------------------------------------------------------- query ----

struct PointCtx {
    double lon, lat;      // input longitude and FakeLL latitude (canonical XYZ)
    double lon_r, lat_r;  // the same point with lon in [-180, 180], lat in [-90, 90]
    bool have64;
    double q[3];
    __device__ void need64()
    {
        if (!have64) {
            gahhg_canon_vertex_xyz(lon, lat, q);
            have64 = true;
        }
    }
};

// exact sign of orient(x, y, z) given a failed FP32 stage; `code` reports a
// decided label (vertex rule / coincident center) through *early.
__device__ __forceinline__ int sign_escalate(const double* x, const double* y, const double* z,
                                             unsigned long long* cnt64, unsigned long long* cntx)
{
    int s = exact::orient_fp64(x, y, z);
    if (cnt64) atomicAdd(cnt64, 1ull);
    if (s != 0) return s;
    if (cntx) atomicAdd(cntx, 1ull);
    return exact::orient_exact(x, y, z);
}

__device__ uint8_t leaf_label(const QueryView& Q, uint32_t leaf, PointCtx& P, bool fp32, unsigned long long* ctr)
{
    const LeafRec L = Q.leaves[leaf];
    double LR[3];
    gahhg_canon_vertex_xyz(L.lon, L.lat, LR);
    local_frame::Frame f;
    local_frame::Tests ft;
    if (fp32) fp32 = fabs(P.lon) <= 540.0 && local_frame::frame_at(P.lon, P.lat, L.lon, L.lat, L.sb, L.cb, f);
    if (fp32) local_frame::tests_of(f, ft);
    if (!fp32) P.need64();
    unsigned long long* c64 = ctr ? ctr + 0 : nullptr;
    unsigned long long* cx = ctr ? ctr + 1 : nullptr;
    int par = 0;
    for (int k = 0; k < L.cnt; k++) {
        const uint32_t es = __ldg(Q.eids + L.off + k);
        const int e = (int)(es & 0x7fffffffu);
        const int s1 = (es >> 31) ? 1 : -1;
        // the record holds (A, B) when s1 = +1, else (B, A): see local_frame.cuh
        int s2 = 0, ea = 0, eb = 0;
        if (fp32) {
            const float4 r = __ldg(Q.recs + L.off + k);
            s2 = s1 * local_frame::sign_edge(ft, r.x, r.y, r.z, r.w);
            const float x1 = s1 > 0 ? r.x : r.z, x2 = s1 > 0 ? r.y : r.w;
            const float y1 = s1 > 0 ? r.z : r.x, y2 = s1 > 0 ? r.w : r.y;
            ea = local_frame::sign_end(ft, x1, x2);
            eb = local_frame::sign_end(ft, y1, y2);
        }
        double A[3], B[3];
        bool haveAB = false;
        auto needAB = [&]() {
            if (!haveAB) {
                const D3 a = Q.pv[Q.pe[2 * e]], b = Q.pv[Q.pe[2 * e + 1]];
                A[0] = a.x;
                A[1] = a.y;
                A[2] = a.z;
                B[0] = b.x;
                B[1] = b.y;
                B[2] = b.z;
                haveAB = true;
            }
        };
        if (s2 == 0) {
            P.need64();
            needAB();
            if (exact::same(P.q, A) || exact::same(P.q, B)) return CELL_IN;  // vertex rule
            if (exact::same(P.q, LR)) return L.label;                       // q is the center
            s2 = sign_escalate(A, B, P.q, c64, cx);
        }
        if (s2 == s1) continue;
        // s3 = orient(R, q, A); crossing needs s3 == s2
        int s3 = ea;
        if (s3 == 0) {
            P.need64();
            needAB();
            if (exact::same(P.q, A) || exact::same(P.q, B)) return CELL_IN;
            if (exact::same(P.q, LR)) return L.label;
            s3 = sign_escalate(LR, P.q, A, c64, cx);
        }
        if (s3 != s2) continue;
        int s4 = eb;
        if (s4 == 0) {
            P.need64();
            needAB();
            if (exact::same(P.q, A) || exact::same(P.q, B)) return CELL_IN;
            if (exact::same(P.q, LR)) return L.label;
            s4 = sign_escalate(LR, P.q, B, c64, cx);
        }
        if (s4 == -s2) par ^= 1;
    }
    return (uint8_t)(par ? 3 - L.label : L.label);
}

// Programmatic dependent launch (sm_90+): a kernel launched with
// programmatic stream serialization may start while its predecessor drains;
// it waits here until the predecessor's grid has completed and its memory is
// visible.  Predecessors allow the start when a block has finished its main
// loop: allowing it at their beginning made the waiting blocks of the next
// tier hold registers through the whole pass (14 % slower on near-edge
// points), allowing it at the end only hides the launch of the next tier.
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ------------------------------------------- summary staging by bulk copy --
//
// The coarse summary (up to 16 KB) goes to shared memory by one bulk copy
// (TMA, untiled cp.async.bulk global -> shared, completion counted on an
// mbarrier in bytes; no multicast) issued by one thread, instead of a load
// per word by every thread.  Both addresses are 16-byte aligned (pool
// allocations are 256-byte aligned, the shared arrays are declared so) and
// the size is rounded up to 16 bytes (the summary's allocation holds at least
// 1,024 words).  Every wait is bounded; a wait that runs out is counted in
// g_tma_timeouts and the block falls back to loading the summary itself into
// memory no pending copy can write (see the kernels), so labels never depend
// on a copy completing.

__device__ unsigned int g_tma_timeouts;
constexpr int MBAR_POLL_LIMIT = 1 << 20;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One thread: the copy of `bytes` from global `src` to shared `dst`,
// completing the barrier's current phase.
__device__ __forceinline__ void bulk_stage(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    // earlier generic-proxy reads of dst (ordered by the block barrier) come
    // before the async-proxy write
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Bounded wait for the phase with the given parity; false when it ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit = MBAR_POLL_LIMIT)
{
    for (int i = 0; i < limit; i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__host__ __device__ __forceinline__ uint32_t summary_bytes(int swords) { return ((uint32_t)swords * 4u + 15u) & ~15u; }

// ------------------------------------------------------ escalation tiers --
//
// The crossing tests of the queued points run in tiers, each its own launch
// over the points the previous tier could not decide, so that no warp carries
// the registers or waits on the branches of a rarer, costlier tier:
//   tier 1: every sign from the certified FP32 filter in the leaf's local
//           frame (local_frame.cuh);
//   tier 2: the canonical FP64 point, the vertex and center rules, and every
//           sign from the FP64 filter on translated rows (orient_fp64_near);
//   tier 3: the complete test (FP64 filter, then exact arithmetic with
//           simulation of simplicity), leaf_label above.
// Every sign a tier returns is exact, so a label does not depend on the tier
// that produced it.
constexpr uint8_t LABEL_DEFER = 0xFF;

// Tier 1 runs every edge of the leaf: a decided edge adds its crossing to
// the parity, an undecided one is noted in `mask` (bit k for record k < 31)
// and the FP64 tier evaluates only those, starting from the parity of the
// decided ones (bit 31).  The label is exact either way: the crossing parity
// is the XOR of independent per-edge tests.  MASK_ALL asks tier 2 for every
// edge (a record beyond the 31st undecided, or the offset refused).
constexpr uint32_t MASK_ALL = 0xFFFFFFFFu;

// Records whose loads tier 1 issues together (one group covers a leaf of
// the default leaf size): the first group goes out before the offset's
// arithmetic, so its latency hides behind the sines and cosines.
constexpr int T1_GROUP = 4;
// Blocks per SM of tier 1: five (48 registers, 20 bytes spilled) ran C2 at
// 21.0-21.1 Gpts/s against 20.5 at four (56 registers); five with groups of
// two (no spills) 20.5, six with groups of two (40 registers) 20.8.
constexpr int T1_BLOCKS = 5;

// A record of tier 1: from global memory through the read-only path, or
// from a copy in shared memory (SHARED).
template <bool SHARED>
__device__ __forceinline__ float4 t1_record(const float4* p)
{
    if constexpr (SHARED) return *p;
    else return __ldg(p);
}

// Tier 1 on the leaf L whose records start at rec (global memory, or the
// staged copy in shared memory when SHARED).
template <bool SHARED>
__device__ __forceinline__ uint8_t leaf_label_fp32_at(const float4* rec, const LeafRec& L, const PointCtx& P,
                                                    uint32_t& mask)
{
    const int cnt = L.cnt;
    float4 r[T1_GROUP];
#pragma unroll
    for (int j = 0; j < T1_GROUP; j++) r[j] = j < cnt ? t1_record<SHARED>(rec + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    local_frame::Frame f;
    if (!(fabs(P.lon) <= 540.0) || !local_frame::frame_at(P.lon, P.lat, L.lon, L.lat, L.sb, L.cb, f)) {
        mask = MASK_ALL;
        return LABEL_DEFER;
    }
    local_frame::Tests t;
    local_frame::tests_of(f, t);
    int par = 0;
    uint32_t und = 0;
    bool all = false;
    for (int k0 = 0; k0 < cnt; k0 += T1_GROUP) {
        if (k0 > 0) {
#pragma unroll
            for (int j = 0; j < T1_GROUP; j++)
                r[j] = k0 + j < cnt ? t1_record<SHARED>(rec + k0 + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < T1_GROUP; j++) {
            const int k = k0 + j;
            if (k >= cnt) break;
            const int x = local_frame::record_crossing(t, r[j].x, r[j].y, r[j].z, r[j].w);
            if (x > 0) par ^= 1;
            if (x < 0) {
                if (k < 31)
                    und |= 1u << k;
                else
                    all = true;
            }
        }
    }
    if (all) {
        mask = MASK_ALL;
        return LABEL_DEFER;
    }
    if (und) {
        mask = und | ((uint32_t)par << 31);
        return LABEL_DEFER;
    }
    return (uint8_t)(par ? 3 - L.label : L.label);
}

__device__ __forceinline__ uint8_t leaf_label_fp32(const QueryView& Q, const LeafRec& L, const PointCtx& P,
                                                 uint32_t& mask)
{
    return leaf_label_fp32_at<false>(Q.recs + L.off, L, P, mask);
}

// Edges of a leaf whose FP64 endpoints the FP64 tier loads together: their
// loads (edge id, then three 16-byte loads of the endpoints) are all in flight
// before the first sign is evaluated, instead of one dependent chain per edge.
constexpr int T2_GROUP = 4;

// FP64 tier on the leaf's records selected by `mask` (MASK_ALL: every record,
// parity from 0; else the records of bits 0..30, parity from bit 31).
__device__ uint8_t leaf_label_fp64(const QueryView& Q, uint32_t leaf, PointCtx& P, uint32_t mask = MASK_ALL)
{
    const LeafRec L = Q.leaves[leaf];
    // the leaf's loads go out before the point's canonical XYZ is computed
    const double LR[3] = {__ldg(Q.leafR + 3 * (size_t)leaf), __ldg(Q.leafR + 3 * (size_t)leaf + 1),
                          __ldg(Q.leafR + 3 * (size_t)leaf + 2)};
    const bool all = mask == MASK_ALL;
    const int cnt = L.cnt;
    int par = all ? 0 : (int)(mask >> 31);
    uint32_t sel = all ? 0u : (mask & 0x7fffffffu);
    int kk[T2_GROUP];
    uint32_t es[T2_GROUP];
    // the next T2_GROUP records (consecutive ones, or the next set bits of
    // sel) and their edge words
    auto next_group = [&](int k0) {
#pragma unroll
        for (int j = 0; j < T2_GROUP; j++) {
            if (all) {
                kk[j] = k0 + j < cnt ? k0 + j : -1;
            } else if (sel) {
                kk[j] = __ffs(sel) - 1;
                sel &= sel - 1u;
            } else {
                kk[j] = -1;
            }
        }
#pragma unroll
        for (int j = 0; j < T2_GROUP; j++) es[j] = kk[j] >= 0 ? __ldg(Q.eids + L.off + kk[j]) : 0u;
    };
    // the first group's edge words are in flight while the point's canonical
    // XYZ is computed
    next_group(0);
    P.need64();
    for (int k0 = 0; kk[0] >= 0; k0 += T2_GROUP) {
        double2 e[T2_GROUP][3];
#pragma unroll
        for (int j = 0; j < T2_GROUP; j++) {
            if (kk[j] >= 0) {
                const double2* p = Q.ends + 3 * (size_t)(es[j] & 0x7fffffffu);
                e[j][0] = __ldg(p);
                e[j][1] = __ldg(p + 1);
                e[j][2] = __ldg(p + 2);
            }
        }
#pragma unroll
        for (int j = 0; j < T2_GROUP; j++) {
            if (kk[j] < 0) break;
            const int s1 = (es[j] >> 31) ? 1 : -1;
            const double A[3] = {e[j][0].x, e[j][0].y, e[j][1].x}, B[3] = {e[j][1].y, e[j][2].x, e[j][2].y};
            if (exact::same(P.q, A) || exact::same(P.q, B)) return CELL_IN;  // vertex rule
            if (exact::same(P.q, LR)) return L.label;                       // q is the center
            // every row is within a cap of the first: translated rows keep the bound small
            const int s2 = exact::orient_fp64_near(A, B, P.q);
            if (s2 == 0) return LABEL_DEFER;
            if (s2 == s1) continue;
            const int s3 = exact::orient_fp64_near(LR, P.q, A);
            if (s3 == 0) return LABEL_DEFER;
            if (s3 != s2) continue;
            const int s4 = exact::orient_fp64_near(LR, P.q, B);
            if (s4 == 0) return LABEL_DEFER;
            if (s4 == -s2) par ^= 1;
        }
        if (all ? k0 + T2_GROUP >= cnt : sel == 0u) break;
        next_group(k0 + T2_GROUP);
    }
    return (uint8_t)(par ? 3 - L.label : L.label);
}

// Level-0 cell of a point from its longitude and FakeLL latitude + 90
// (`laf`); false when the point lies outside the domain.
struct Loc {
    int ix, iy;
    double fu, fv;
};

// Level-0 cell of a point from its longitude and FakeLL latitude + 90
// (`laf`); false when the point lies outside the domain.  Inside the domain
// this costs two multiply-adds, two conversions and two unsigned compares;
// points beyond a non-polar latitude edge are rejected with one more compare.
__device__ __forceinline__ bool domain_locate(const QueryView& Q, double lo, double laf, Loc& L)
{
    double u = fma(lo, Q.su_lon, Q.u0), v = fma(laf, Q.su_lat, Q.v0);
    int ix = __double2int_rd(u), iy = __double2int_rd(v);
    if ((unsigned)iy >= (unsigned)Q.H) {
        if (iy < 0 ? !Q.to_south : !Q.to_north) return false;
        // a domain that reaches the pole keeps the pole in its first/last row
        const bool below = iy < 0;
        iy = below ? 0 : Q.H - 1;
        v = below ? 0.0 : fmin(v, Q.Hd);
    }
    if ((unsigned)ix >= (unsigned)Q.W) {
        if (u < 0.0) u += Q.U360;
        if (u < 0.0) u += Q.U360;
        if (u >= Q.U360) u -= Q.U360;
        if (u >= Q.U360) u -= Q.U360;
        ix = __double2int_rd(u);
        if ((unsigned)ix >= (unsigned)Q.W) {
            if (!Q.full_lon) return false;
            ix = ix < 0 ? 0 : Q.W - 1;
        }
    }
    L.ix = ix;
    L.iy = iy;
    L.fu = u - ix;
    L.fv = v - iy;
    return true;
}

// A cell fraction in [0, 1) as a 32-bit binary fraction, saturating (below 0
// gives 0, 1 and above all ones).  Its base-4 digits are the children that
// the recursion f -> 4 f - floor(4 f) (clamped to 0..3) visits: that FP64
// recursion is exact, so digit k of the fraction is its k-th child for the
// first 16 levels, and for the clamped out-of-range cases both give 0 or 3 at
// every level.  The lattice has at most MAX_DESCENT levels below the top.
constexpr int MAX_DESCENT = 16;
__device__ __forceinline__ uint32_t frac_bits(double f) { return __double2uint_rz(f * 4294967296.0); }

__device__ __forceinline__ uint32_t descend(const QueryView& Q, uint32_t w, double fu, double fv)
{
    uint32_t U = frac_bits(fu), V = frac_bits(fv);
    while ((w & KIND_MASK) == KIND_INNER) {
        w = __ldg(Q.nodes + (w & INDEX_MASK) + (V >> 30) * FAN + (U >> 30));
        U <<= 2;
        V <<= 2;
    }
    return w;
}

// block-reduced count of inside labels (statistics only)
__device__ __forceinline__ void count_inside(int v, unsigned long long* dst)
{
    __shared__ int s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_sum, v);
    __syncthreads();
    if (threadIdx.x == 0 && s_sum) atomicAdd(dst, (unsigned long long)s_sum);
}

constexpr int LOC_UNROLL = 4;
constexpr uint8_t LABEL_PENDING = 0;
// Leaf word of a queued point that pass 1 did not locate (a pure node
// without a label, which is never queued).
constexpr uint32_t LEAF_UNKNOWN = KIND_PURE;

// Pass 1: every point whose cell has no edges gets its label; the others are
// queued (index within this chunk) for pass 2.  Lean on registers and
// instructions so that many warps keep loads in flight; lon/lat and labels
// stream with an evict-first policy so the node table stays in L2.  The index
// arithmetic need not match the canonical conversion bit for bit: every cap
// carries a margin far above its rounding (see LOC_MARGIN).
// Pass 1 over points [first, first + count) of one polygon, in tiles of
// TPB * LOC_UNROLL points (tiles tile0, tile0 + tstride, ...): every point
// whose cell has no edges gets its label; the others are queued (their index
// `first + local`) for pass 2.  Lean on registers and instructions so that
// many warps keep loads in flight; lon/lat and labels stream with an
// evict-first policy so the node table stays in L2.  The index arithmetic
// need not match the canonical conversion bit for bit: every cap carries a
// margin far above its rounding (see LOC_MARGIN).
template <bool STATS, bool LOCKSTEP = false, int UNROLL = LOC_UNROLL>
__device__ __forceinline__ void locate_range(const QueryView& Q, const uint32_t* s_sum,
                                             const double2* __restrict__ ll, uint8_t* __restrict__ out,
                                             uint32_t* __restrict__ queue, uint32_t* __restrict__ leafq,
                                             unsigned int* __restrict__ qcount, long long first, int count,
                                             int tile0, int tstride, int& inside)
{
    const int lane = threadIdx.x & 31;
    const int cs = Q.cshift, cw = Q.CW;
    constexpr int TILE = TPB * UNROLL;
    for (int base = tile0 * TILE; base < count; base += tstride * TILE) {
        const bool full = base + TILE <= count;
        double2 p[UNROLL];
#pragma unroll
        for (int k = 0; k < UNROLL; k++) {
            const int i = base + k * TPB + threadIdx.x;
            p[k] = (full || i < count) ? __ldcs(ll + first + i) : make_double2(0.0, 0.0);
        }
        uint8_t lab[UNROLL];
        bool push[UNROLL];
        bool any = false;
        // LOCKSTEP: the node words of all points are loaded first and the
        // descents advance one level per round, so a thread keeps one
        // independent load per point in flight (points that mostly need the
        // node table, as around small polygons, are bound by its latency)
        uint32_t w[UNROLL];
        uint32_t fu[UNROLL], fv[UNROLL];  // cell fractions as binary fractions (frac_bits)
#pragma unroll
        for (int k = 0; k < UNROLL; k++) {
            const int i = base + k * TPB + threadIdx.x;
            const double lo = p[k].x;
            const double laf = p[k].y + 90.0;  // the reference's FakeLL latitude + 90
            lab[k] = LABEL_PENDING;
            push[k] = false;
            w[k] = KIND_PURE;
            if (full || i < count) {
                if (laf >= 0.0 && laf <= 180.0 && fabs(lo) <= 540.0) {
                    Loc L;
                    if (!domain_locate(Q, lo, laf, L)) {
                        lab[k] = (uint8_t)Q.outside;
                    } else {
                        const int c = (L.iy >> cs) * cw + (L.ix >> cs);
                        const uint32_t code = (s_sum[c >> 4] >> ((c & 15) << 1)) & 3u;
                        if (code < 2u) {
                            lab[k] = (uint8_t)(code + 1u);  // coarse cell without edges: most points end here
                        } else if (LOCKSTEP) {
                            w[k] = __ldg(Q.nodes + (size_t)L.iy * Q.W + L.ix);
                            fu[k] = frac_bits(L.fu);
                            fv[k] = frac_bits(L.fv);
                        } else {
                            const uint32_t d = descend(Q, __ldg(Q.nodes + (size_t)L.iy * Q.W + L.ix), L.fu, L.fv);
                            if ((d & KIND_MASK) == KIND_PURE)
                                lab[k] = (uint8_t)(d & 3u);
                            else
                                push[k] = true;
                            w[k] = d;
                        }
                    }
                } else {
                    // unusual coordinates go to pass 2; non-finite input stays undefined
                    push[k] = isfinite(lo) && isfinite(laf);
                }
            }
            if (!LOCKSTEP) any |= push[k];
        }
        if (LOCKSTEP) {
            bool inner = true;
            while (inner) {
                inner = false;
#pragma unroll
                for (int k = 0; k < UNROLL; k++)
                    if ((w[k] & KIND_MASK) == KIND_INNER) {
                        w[k] = __ldg(Q.nodes + (w[k] & INDEX_MASK) + (fv[k] >> 30) * FAN + (fu[k] >> 30));
                        fu[k] <<= 2;
                        fv[k] <<= 2;
                        inner = true;
                    }
            }
#pragma unroll
            for (int k = 0; k < UNROLL; k++) {
                if (lab[k] == LABEL_PENDING && !push[k]) {
                    const int i = base + k * TPB + threadIdx.x;
                    if (full || i < count) {
                        if ((w[k] & KIND_MASK) == KIND_PURE) {
                            if (w[k] != KIND_PURE) lab[k] = (uint8_t)(w[k] & 3u);  // KIND_PURE alone: no node read
                        } else {
                            push[k] = true;
                        }
                    }
                }
                any |= push[k];
            }
        }
        if (__any_sync(0xffffffffu, any)) {
            // one atomic on the queue counter per warp and tile: every thread of
            // the grid pushes through this one counter, and where most points
            // are queued (points near the edges) the counter itself limits pass 1
            // (one per block and tile, which takes block-wide barriers, made
            // uniform points 14 % slower and near-edge points 2 % faster)
            unsigned int total = 0;
#pragma unroll
            for (int k = 0; k < UNROLL; k++) total += __popc(__ballot_sync(0xffffffffu, push[k]));
            unsigned int pos = 0;
            if (lane == 0) pos = atomicAdd(qcount, total);
            pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
            for (int k = 0; k < UNROLL; k++) {
                const unsigned int mk = __ballot_sync(0xffffffffu, push[k]);
                if (push[k]) {
                    const unsigned int at = pos + __popc(mk & ((1u << lane) - 1u));
                    queue[at] = (uint32_t)(first + base + k * TPB + threadIdx.x);
                    // w is the leaf word, or KIND_PURE (LEAF_UNKNOWN) for an unlocated point
                    if (leafq) leafq[at] = w[k];
                }
                pos += __popc(mk);
            }
        }
#pragma unroll
        for (int k = 0; k < UNROLL; k++) {
            const int i = base + k * TPB + threadIdx.x;
            if (full || i < count) __stcs(out + first + i, lab[k]);
            if (STATS) inside += lab[k] == CELL_IN;
        }
    }
}

template <bool STATS>
__global__ void __launch_bounds__(TPB) k_locate(const double2* __restrict__ ll, int n, uint8_t* __restrict__ out,
                                               QueryView Q, uint32_t* __restrict__ queue,
                                               uint32_t* __restrict__ leafq, unsigned int* __restrict__ qcount,
                                               unsigned long long* ctr, int poll_limit)
{
    extern __shared__ __align__(16) uint32_t s_sum[];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_late;
    if (threadIdx.x == 0) {
        s_late = 0;
        mbar_init(&s_bar);
        bulk_stage(s_sum, Q.summary, summary_bytes(Q.swords), &s_bar);
    }
    __syncthreads();
    if (!mbar_wait(&s_bar, 0, poll_limit)) s_late = 1;
    __syncthreads();
    const bool late = s_late != 0;
    // after a wait that ran out the block reads the summary from global
    // memory and never touches s_sum, which the pending copy still targets
    if (late && threadIdx.x == 0) atomicAdd(&g_tma_timeouts, 1u);
    int inside = 0;
    locate_range<STATS>(Q, late ? Q.summary : s_sum, ll, out, queue, leafq, qcount, 0, n, blockIdx.x, gridDim.x,
                        inside);
    if (late) mbar_wait(&s_bar, 0);  // the copy in flight ends before the block does (bounded)
    allow_dependents();
    if (STATS && ctr) count_inside(inside, ctr + 3);
}

// The leaf of a queued point (the point context filled in), or its label
// with KIND_PURE when its cell has no edges.
// The point's context, and its node word: `known` when pass 1 located the
// point (any leaf it finds serves: every leaf cap holds its points with a
// margin above the locate arithmetic's rounding), else a descent from the top.
__device__ __forceinline__ uint32_t point_leaf(const QueryView& Q, double2 p, PointCtx& P,
                                              uint32_t known = LEAF_UNKNOWN)
{
    P.lat = gahhg_canon_query_lat(p.y);
    P.lon = p.x;
    P.have64 = false;
    double lo = P.lon, la = P.lat;
    if (!(fabs(lo) <= 540.0 && fabs(la) <= 90.0)) {
        // unusual input: locate from the canonical XYZ itself
        P.need64();
        la = asin(fmin(1.0, fmax(-1.0, P.q[1]))) / RAD;
        lo = atan2(P.q[0], P.q[2]) / RAD;
    }
    Loc L;
    double lr = lo;
    if (lr > 180.0) lr -= 360.0;
    if (lr > 180.0) lr -= 360.0;
    if (lr < -180.0) lr += 360.0;
    if (lr < -180.0) lr += 360.0;
    P.lon_r = lr;
    P.lat_r = la;
    if (known != LEAF_UNKNOWN) return known;
    const bool in = domain_locate(Q, lo, la + 90.0, L);
    return in ? descend(Q, __ldg(Q.nodes + (size_t)L.iy * Q.W + L.ix), L.fu, L.fv) : Q.outside;
}

// One point through the untiered path (escalations inline, counted per test).
template <bool FP32>
__device__ __forceinline__ uint8_t leaf_point(const QueryView& Q, double2 p, unsigned long long* ctr)
{
    PointCtx P;
    const uint32_t w = point_leaf(Q, p, P);
    if ((w & KIND_MASK) == KIND_PURE) return (uint8_t)(w & 3u);
    if (ctr) atomicAdd(ctr + 2, 1ull);
    return leaf_label(Q, w & INDEX_MASK, P, FP32, ctr);
}

// Pass 2: exact crossing tests for the queued points.
template <bool FP32>
__global__ void __launch_bounds__(TPB) k_leaf(const double2* __restrict__ ll, uint8_t* __restrict__ out,
                                             QueryView Q, const uint32_t* __restrict__ queue,
                                             const unsigned int* __restrict__ qcount, unsigned long long* ctr)
{
    const unsigned int m = *qcount;
    int inside = 0;
    for (unsigned int t = blockIdx.x * blockDim.x + threadIdx.x; t < m; t += gridDim.x * blockDim.x) {
        const uint32_t i = queue[t];
        const uint8_t lab = leaf_point<FP32>(Q, ll[i], ctr);
        out[i] = lab;
        inside += lab == CELL_IN;
    }
    if (ctr) count_inside(inside, ctr + 3);
}

// ------------------------------------------------------------- batches --

// A run of points of one view (points are stored segment after segment, and
// chunks are in point order, so chunk starts are increasing).
struct BatchChunk {
    int view;
    int count;
    long long start;
};

constexpr int BATCH_SUMMARY_WORDS = 4096;  // 16 KB of shared memory
// Launch shapes of the batch locate: points per thread in flight (in
// lockstep) and blocks per SM (all resident; each holds 32 KB of shared
// memory, and the register budget per thread follows from the blocks).  The
// default, five points at five blocks (48 registers), took a 1,024-polygon
// C3 batch from 75.6 (8 points, two blocks) to 106.5 Gpts/s; 4 x 5 101.2,
// 6 x 4 101.8, 6 x 5 102.3, 4 x 6 91.2, 8 x 3 93.5 (labels identical): more
// warps hide more of the node descents' latency than more points per
// thread (2 x 6 spills at 40 registers and ran at 56.6).  Batches of other
// point mixes may prefer another row (4 x 4 leaves fewer lanes idle in
// chunks of few points); the batch autotuner measures them.
struct BatchShape {
    int unroll, blocks;
};
constexpr BatchShape BATCH_SHAPES[] = {{5, 5}, {4, 4}, {6, 4}, {8, 3}};
constexpr int BATCH_NSHAPES = (int)(sizeof(BATCH_SHAPES) / sizeof(BATCH_SHAPES[0]));

// Pass 1 over a batch: a persistent grid takes chunks in order from an atomic
// counter (polygons of very different sizes balance themselves), stages the
// chunk's polygon summary in shared memory and runs the single-polygon tile
// loop on it.
template <bool STATS, int UNROLL, int BLOCKS>
__global__ void __launch_bounds__(TPB, BLOCKS) k_batch_locate(const QueryView* __restrict__ views,
                                                     const BatchChunk* __restrict__ chunks, int nchunks,
                                                     unsigned int* next_chunk, const double2* __restrict__ ll,
                                                     uint8_t* __restrict__ out, uint32_t* __restrict__ queue,
                                                     uint32_t* __restrict__ leafq, unsigned int* __restrict__ qcount,
                                                     unsigned long long* ctr, int poll_limit)
{
    // s_sum receives the bulk copies; after a wait runs out the block loads
    // summaries itself into s_own, which no copy writes
    __shared__ __align__(16) uint32_t s_sum[BATCH_SUMMARY_WORDS];
    __shared__ __align__(16) uint32_t s_own[BATCH_SUMMARY_WORDS];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_chunk, s_late;
    if (threadIdx.x == 0) {
        s_late = 0;
        mbar_init(&s_bar);
    }
    uint32_t phase = 0;
    bool late = false;  // the same in every thread: read from s_late after a barrier
    int inside = 0;
    for (;;) {
        if (threadIdx.x == 0) s_chunk = (int)atomicAdd(next_chunk, 1u);
        __syncthreads();
        const int ci = s_chunk;
        if (ci >= nchunks) break;
        const BatchChunk c = chunks[ci];
        const QueryView Q = views[c.view];
        const uint32_t* sum = s_sum;
        if (!late) {
            if (threadIdx.x == 0) bulk_stage(s_sum, Q.summary, summary_bytes(Q.swords), &s_bar);
            if (!mbar_wait(&s_bar, phase, poll_limit)) s_late = 1;  // any thread's timeout switches the block
            phase ^= 1u;
            __syncthreads();
            late = s_late != 0;
        }
        if (late) {
            for (int k = threadIdx.x; k < Q.swords; k += TPB) s_own[k] = __ldg(Q.summary + k);
            sum = s_own;
            __syncthreads();
        }
        locate_range<STATS, true, UNROLL>(Q, sum, ll, out, queue, leafq, qcount, c.start, c.count, 0, 1, inside);
        __syncthreads();
    }
    if (late) {
        if (threadIdx.x == 0) atomicAdd(&g_tma_timeouts, 1u);
        mbar_wait(&s_bar, phase ^ 1u);  // the copy in flight ends before the block does (bounded)
    }
    allow_dependents();
    if (STATS && ctr) count_inside(inside, ctr + 3);
}

// Escalation queues of one pass-2 run.  cnt[0] / cnt[1] count the points
// deferred to tier 2 / tier 3 (they keep counting past the capacities);
// cnt[2] is raised when a point found its queue full: it stays unlabelled
// (pass 1 wrote LABEL_PENDING) and the final sweep gives it the complete
// test, so no tier carries the code of the tiers after it.
// Every queue of points has a parallel array of leaf words (l1 for the
// pass-1 queue): the node word pass 1 found for the point, or LEAF_UNKNOWN
// when it did not locate it, so the tiers need not descend again.
struct Tiers {
    uint32_t* q2;
    uint32_t* q3;
    uint32_t* l1;
    uint32_t* l2;
    uint32_t* l3;
    uint32_t* m2;   // per tier-2 entry: tier 1's mask of undecided records (leaf_label_fp32)
    unsigned int* cnt;
    unsigned int cap2, cap3;
    // the pass-1 queue in window order (k_part_scatter), used by the first
    // tier when *sorted == 1
    const uint32_t* spts = nullptr;
    const uint32_t* sleaf = nullptr;
    const unsigned int* sorted = nullptr;
    int sstride = 1;  // words from one ordered entry to the next (2: leaf order's interleaved pairs)
};

// The pass-1 queue as the first tier reads it: in window order when
// k_part_scatter ran, else in pass-1 order.
__device__ __forceinline__ void first_tier_source(const Tiers& T, const uint32_t*& pts, const uint32_t*& leaf,
                                                  unsigned int& stride)
{
    stride = 1;
    if (T.sorted && *(const volatile unsigned int*)T.sorted == 1u) {
        pts = T.spts;
        leaf = T.sleaf;
        stride = (unsigned int)T.sstride;
    }
}

// Where a queued point's index view comes from: one polygon...
struct OneView {
    QueryView Q;
    __device__ __forceinline__ const QueryView& of(uint32_t) const { return Q; }
};

// ...or the chunk holding it (binary search of the chunk starts).
struct ChunkViews {
    const QueryView* views;
    const BatchChunk* chunks;
    int nchunks;
    __device__ __forceinline__ const QueryView& of(uint32_t i) const
    {
        int lo = 0, hi = nchunks;  // chunks[lo].start <= i < chunks[hi].start
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(&chunks[mid].start) <= (long long)i) lo = mid;
            else hi = mid;
        }
        return views[__ldg(&chunks[lo].view)];
    }
};

// Appends i to q through counter *c, one atomic per group of converged
// threads; false when the queue is full.
__device__ __forceinline__ bool push_deferred(uint32_t i, uint32_t w, uint32_t* q, uint32_t* l, unsigned int* c,
                                              unsigned int cap, uint32_t* extra = nullptr, uint32_t x = 0u)
{
    const unsigned int act = __activemask();
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(act) - 1;
    unsigned int base = 0;
    if (lane == leader) base = atomicAdd(c, (unsigned int)__popc(act));
    base = __shfl_sync(act, base, leader);
    const unsigned int pos = base + __popc(act & ((1u << lane) - 1u));
    if (pos >= cap) return false;
    q[pos] = i;
    l[pos] = w;
    if (extra) extra[pos] = x;
    return true;
}

__device__ __forceinline__ void count_stats(unsigned long long* ctr, int inside, int boundary, int fp64, int exact)
{
    count_inside(inside, ctr + 3);
    count_inside(boundary, ctr + 2);
    count_inside(fp64, ctr + 0);
    count_inside(exact, ctr + 1);
}

// Tier 1 over the pass-1 queue.
template <class VS>
__global__ void __launch_bounds__(TPB, T1_BLOCKS) k_leaf_t1(VS vs, const double2* __restrict__ ll,
                                                         uint8_t* __restrict__ out, const uint32_t* __restrict__ queue,
                                                         const unsigned int* __restrict__ qcount, Tiers T,
                                                         unsigned long long* ctr)
{
    __shared__ unsigned int s_wcnt[TPB / 32];
    __shared__ unsigned int s_base;
    wait_for_predecessor();
    const unsigned int m = *qcount;
    const uint32_t* src = queue;
    const uint32_t* src_leaf = T.l1;
    unsigned int st;
    first_tier_source(T, src, src_leaf, st);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inside = 0, boundary = 0, fp64 = 0;
    // block-uniform loop: the deferred points of a block's round take one
    // atomic on the tier-2 counter (about half the points defer on near-edge
    // inputs, and one counter serves the whole grid)
    for (unsigned int b0 = blockIdx.x * blockDim.x; b0 < m; b0 += gridDim.x * blockDim.x) {
        const unsigned int t = b0 + threadIdx.x;
        bool defer = false;
        uint32_t i = 0, w = 0, mask = 0;
        if (t < m) {
            i = src[t * st];
            const uint32_t known = src_leaf[t * st];
            const QueryView& Q = vs.of(i);
            // the leaf record (a point pass 1 located in a leaf) is loaded
            // with the point's coordinates, not after them
            const bool in_leaf = (known & KIND_MASK) == KIND_LEAF;
            LeafRec L0;
            if (in_leaf) L0 = Q.leaves[known & INDEX_MASK];
            PointCtx P;
            w = point_leaf(Q, ll[i], P, known);
            uint8_t lab;
            if ((w & KIND_MASK) == KIND_PURE) {
                lab = (uint8_t)(w & 3u);
            } else {
                boundary++;
                lab = leaf_label_fp32(Q, in_leaf ? L0 : Q.leaves[w & INDEX_MASK], P, mask);
            }
            if (lab == LABEL_DEFER) {
                fp64++;
                defer = true;
            } else {
                out[i] = lab;
                inside += lab == CELL_IN;
            }
        }
        const unsigned int bal = __ballot_sync(0xffffffffu, defer);
        if (lane == 0) s_wcnt[warp] = __popc(bal);
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned int tot = 0;
            for (int k = 0; k < TPB / 32; k++) {
                const unsigned int c = s_wcnt[k];
                s_wcnt[k] = tot;
                tot += c;
            }
            s_base = tot ? atomicAdd(T.cnt, tot) : 0u;
        }
        __syncthreads();
        if (defer) {
            const unsigned int pos = s_base + s_wcnt[warp] + __popc(bal & ((1u << lane) - 1u));
            if (pos < T.cap2) {
                T.q2[pos] = i;
                T.l2[pos] = w;
                T.m2[pos] = mask;
            } else {
                T.cnt[2] = 1;  // the tier-3 sweep labels it
            }
        }
        __syncthreads();  // s_wcnt / s_base are rewritten next round
    }
    allow_dependents();
    if (ctr) count_stats(ctr, inside, boundary, fp64, 0);
}

// ---------------------------------- tier 1 with the edge lists staged --
//
// Over the pass-1 queue in leaf order (k_ls_*), the entries of a tile of TPB
// consecutive entries lie in a run of consecutive leaves, and leaves are
// numbered so that their records are contiguous: the tile's leaf records and
// the edge records of those leaves are two contiguous slices of the index.
// One thread copies both into shared memory (TMA: two untiled cp.async.bulk
// global -> shared, completion counted in bytes on one mbarrier; no
// multicast, the source is this GPU's index) while the block loads its
// points and their frames, and every crossing test of the tile then reads
// its leaf record and edge list from shared memory.  A tile whose slices do
// not fit the buffers, a tile holding points pass 1 did not locate, and every
// tile of a queue left in pass-1 order (below PART_MIN_QUEUE entries) read
// the index from global memory as k_leaf_t1 does.  Every wait is bounded: a
// wait that runs out makes the block stop staging (its later tiles read
// global memory, so the late copy is never read), is counted once in
// g_tma_timeouts, and before exiting the block waits (bounded again) for
// that copy.  Both slices start on 16-byte boundaries (pool allocations are
// 256-byte aligned; leaf records are 32 bytes, edge records 16) and their
// sizes are multiples of 16 bytes.  Measured on 2e7 C2 points (9.1M queued):
// 337 us against 283 us for k_leaf_t1 on the same leaf-ordered queue, whose
// per-warp gathers leaf order already makes one request per warp and leaf;
// the staging adds a block barrier and a wait per tile and copies every
// leaf of the tile's range.  It is therefore an option (pass-2 order 3).
constexpr int T1S_LEAVES = 256;  // 8 KB of leaf records per tile
constexpr int T1S_RECS = 1536;   // 24 KB of edge records per tile
constexpr int T1S_BLOCKS = 5;

__global__ void __launch_bounds__(TPB, T1S_BLOCKS) k_leaf_t1s(QueryView Q, const double2* __restrict__ ll,
                                                            uint8_t* __restrict__ out,
                                                            const uint32_t* __restrict__ queue,
                                                            const unsigned int* __restrict__ qcount, Tiers T,
                                                            unsigned long long* ctr, int polls)
{
    __shared__ __align__(16) LeafRec s_leaf[T1S_LEAVES];
    __shared__ __align__(16) float4 s_rec[T1S_RECS];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ unsigned int s_wcnt[TPB / 32];
    __shared__ unsigned int s_base;
    __shared__ uint32_t s_l0, s_r0, s_nr;  // first staged leaf, first staged record, records staged
    __shared__ int s_nl;                   // leaves staged for the tile (0: none)
    __shared__ int s_broken;               // a wait ran out: no more staging
    if (threadIdx.x == 0) {
        mbar_init(&s_bar);
        s_broken = 0;
    }
    __syncthreads();
    wait_for_predecessor();
    const unsigned int m = *qcount;
    const uint32_t* src = queue;
    const uint32_t* src_leaf = T.l1;
    unsigned int st;
    first_tier_source(T, src, src_leaf, st);
    const bool sorted = src_leaf != T.l1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inside = 0, boundary = 0, fp64 = 0;
    uint32_t phase = 0;  // parity of the barrier's current phase
    // Thread 0 works a tile ahead so that a tile's copy goes out as the tile
    // starts: while the block labels tile k it loads the first and last leaf
    // words of tile k + 1, and after the labels those leaves' record
    // offsets (the bounds, state 1; 2 when the slices do not fit).
    // (thread 0's state is kept in shared memory, off the other threads'
    // registers)
    const unsigned int bstep = gridDim.x * blockDim.x;
    __shared__ uint32_t s_nw0, s_nw1;                 // next tile's first and last leaf words
    __shared__ uint32_t s_bL0, s_bL1, s_br0, s_br1;  // its leaves and record range
    __shared__ int s_bstate;                          // 0 not known, 1 staged, 2 not staged
    auto tile_words = [&](unsigned int b) {
        s_nw0 = src_leaf[b * st];
        s_nw1 = src_leaf[(min(b + TPB, m) - 1) * st];
    };
    auto tile_bounds = [&]() {
        const uint32_t w0 = s_nw0, w1 = s_nw1;
        s_bstate = 2;
        if ((w0 & KIND_MASK) != KIND_LEAF || (w1 & KIND_MASK) != KIND_LEAF) return;
        const uint32_t L0 = w0 & INDEX_MASK, L1 = w1 & INDEX_MASK;
        if (L1 < L0 || L1 - L0 >= (uint32_t)T1S_LEAVES) return;
        const uint32_t r0 = Q.leaves[L0].off, r1 = Q.leaves[L1].off + Q.leaves[L1].cnt;
        if (r1 < r0 || r1 - r0 > (uint32_t)T1S_RECS) return;
        s_bL0 = L0;
        s_bL1 = L1;
        s_br0 = r0;
        s_br1 = r1;
        s_bstate = 1;
    };
    if (threadIdx.x == 0) s_bstate = 0;
    if (threadIdx.x == 0 && sorted && blockIdx.x * blockDim.x < m) tile_words(blockIdx.x * blockDim.x);
    for (unsigned int b0 = blockIdx.x * blockDim.x; b0 < m; b0 += bstep) {
        if (threadIdx.x == 0) {
            int nl = 0;
            if (sorted && !s_broken) {
                if (s_bstate == 0) tile_bounds();  // the first tile
                if (s_bstate == 1) {
                    const uint32_t bL0 = s_bL0, br0 = s_br0;
                    nl = (int)(s_bL1 - bL0 + 1);
                    s_l0 = bL0;
                    s_r0 = br0;
                    s_nr = s_br1 - br0;
                    const uint32_t lb = (uint32_t)nl * (uint32_t)sizeof(LeafRec);
                    const uint32_t rb = (s_br1 - br0) * (uint32_t)sizeof(float4);
                    // the previous tile's reads of the buffers (ordered by
                    // the block barrier) come before these writes
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&s_bar)),
                                 "r"(lb + rb)
                                 : "memory");
                    asm volatile(
                        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                            smem_u32(s_leaf)),
                        "l"(Q.leaves + bL0), "r"(lb), "r"(smem_u32(&s_bar))
                        : "memory");
                    if (rb)
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
                            "[%3];" ::"r"(smem_u32(s_rec)),
                            "l"(Q.recs + br0), "r"(rb), "r"(smem_u32(&s_bar))
                            : "memory");
                }
            }
            s_nl = nl;
            s_bstate = 0;
            if (sorted && b0 + bstep < m) tile_words(b0 + bstep);
        }
        // every thread's point and frame while the copy is in flight
        const unsigned int t = b0 + threadIdx.x;
        bool defer = false;
        uint32_t i = 0, w = 0, mask = 0;
        PointCtx P;
        if (t < m) {
            i = src[t * st];
            w = point_leaf(Q, ll[i], P, src_leaf[t * st]);
        }
        __syncthreads();
        const int nl = s_nl;
        bool staged = false;
        if (nl) {
            staged = mbar_wait(&s_bar, phase, polls);
            phase ^= 1u;
            if (!staged) atomicOr(&s_broken, 1);  // any thread whose wait ran out
        }
        if (t < m) {
            uint8_t lab;
            if ((w & KIND_MASK) == KIND_PURE) {
                lab = (uint8_t)(w & 3u);
            } else {
                boundary++;
                const uint32_t li = (w & INDEX_MASK) - s_l0;  // wraps above nl below the first leaf
                bool done = false;
                if (staged && li < (uint32_t)nl) {
                    const LeafRec L = s_leaf[li];
                    const uint32_t ro = L.off - s_r0;
                    if (ro <= s_nr && (uint32_t)L.cnt <= s_nr - ro) {
                        lab = leaf_label_fp32_at<true>(s_rec + ro, L, P, mask);
                        done = true;
                    }
                }
                if (!done) lab = leaf_label_fp32(Q, Q.leaves[w & INDEX_MASK], P, mask);
            }
            if (lab == LABEL_DEFER) {
                fp64++;
                defer = true;
            } else {
                out[i] = lab;
                inside += lab == CELL_IN;
            }
        }
        if (threadIdx.x == 0 && sorted && b0 + bstep < m) tile_bounds();  // the next tile's, ahead of its start
        const unsigned int bal = __ballot_sync(0xffffffffu, defer);
        if (lane == 0) s_wcnt[warp] = __popc(bal);
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned int tot = 0;
            for (int k = 0; k < TPB / 32; k++) {
                const unsigned int c = s_wcnt[k];
                s_wcnt[k] = tot;
                tot += c;
            }
            s_base = tot ? atomicAdd(T.cnt, tot) : 0u;
        }
        __syncthreads();
        if (defer) {
            const unsigned int pos = s_base + s_wcnt[warp] + __popc(bal & ((1u << lane) - 1u));
            if (pos < T.cap2) {
                T.q2[pos] = i;
                T.l2[pos] = w;
                T.m2[pos] = mask;
            } else {
                T.cnt[2] = 1;  // the tier-3 sweep labels it
            }
        }
        __syncthreads();  // s_wcnt / s_base and the staged slices are rewritten next round
    }
    allow_dependents();
    if (threadIdx.x == 0 && s_broken) {
        atomicAdd(&g_tma_timeouts, 1u);
        mbar_wait(&s_bar, phase ^ 1u);  // the copy whose wait ran out
    }
    if (ctr) count_stats(ctr, inside, boundary, fp64, 0);
}

// Tier 2's shape: blocks of 128 threads, five per SM (96 registers, about
// 60 bytes spilled) hold 20 warps per SM where 256-thread blocks at 110
// registers held 16: FP64-filter queries of C2 (tier 2 over the whole
// pass-1 queue) 15.8 -> 16.6 Gpts/s; six blocks (80 registers, 200 bytes
// spilled) 12.8; the FP32 filter's tier 2 is unchanged by any of them.
constexpr int T2_TPB = 128;
constexpr int T2_BLOCKS = 5;

// Tier 2 over the tier-1 queue, or (FROM_PASS1, FP64-filter queries) over
// the pass-1 queue itself.
template <class VS, bool FROM_PASS1>
__global__ void __launch_bounds__(T2_TPB, T2_BLOCKS) k_leaf_t2(VS vs, const double2* __restrict__ ll, uint8_t* __restrict__ out,
                                                const uint32_t* __restrict__ src, const uint32_t* __restrict__ src_leaf,
                                                const unsigned int* __restrict__ src_count, unsigned int src_cap,
                                                Tiers T, unsigned long long* ctr)
{
    wait_for_predecessor();
    const unsigned int m = min(*src_count, src_cap);
    const uint32_t* sp = src;
    const uint32_t* sl = src_leaf;
    unsigned int st = 1;
    if (FROM_PASS1) first_tier_source(T, sp, sl, st);
    int inside = 0, boundary = 0, exact = 0;
    for (unsigned int t = blockIdx.x * blockDim.x + threadIdx.x; t < m; t += gridDim.x * blockDim.x) {
        const uint32_t i = sp[t * st];
        const QueryView& Q = vs.of(i);
        PointCtx P;
        const uint32_t w = point_leaf(Q, ll[i], P, sl[t * st]);
        uint8_t lab;
        if ((w & KIND_MASK) == KIND_PURE) {
            lab = (uint8_t)(w & 3u);
        } else {
            if (FROM_PASS1) boundary++;
            lab = leaf_label_fp64(Q, w & INDEX_MASK, P, FROM_PASS1 ? MASK_ALL : T.m2[t]);
            if (lab == LABEL_DEFER) {
                exact++;
                if (!push_deferred(i, w, T.q3, T.l3, T.cnt + 1, T.cap3)) T.cnt[2] = 1;
                continue;
            }
        }
        out[i] = lab;
        inside += lab == CELL_IN;
    }
    allow_dependents();
    if (ctr) count_stats(ctr, inside, boundary, 0, exact);
}

// Tier 3 over the tier-2 queue, then, after a queue overflow, the complete
// test for every pass-1 point still unlabelled.
template <class VS>
__global__ void __launch_bounds__(TPB) k_leaf_t3(VS vs, const double2* __restrict__ ll, uint8_t* __restrict__ out,
                                                const uint32_t* __restrict__ queue,
                                                const unsigned int* __restrict__ qcount, Tiers T,
                                                unsigned long long* ctr)
{
    wait_for_predecessor();
    const unsigned int m3 = min(T.cnt[1], T.cap3);
    const bool sweep = T.cnt[2] != 0;
    const unsigned int m = sweep ? *qcount : 0;
    int inside = 0;
    for (unsigned int t = blockIdx.x * blockDim.x + threadIdx.x; t < m3 + m; t += gridDim.x * blockDim.x) {
        uint32_t i, known;
        if (t < m3) {
            i = T.q3[t];
            known = T.l3[t];
        } else {
            i = queue[t - m3];
            if (out[i] != LABEL_PENDING) continue;
            known = T.l1[t - m3];
        }
        const QueryView& Q = vs.of(i);
        PointCtx P;
        const uint32_t w = point_leaf(Q, ll[i], P, known);
        const uint8_t lab = ((w & KIND_MASK) == KIND_PURE) ? (uint8_t)(w & 3u)
                                                            : leaf_label(Q, w & INDEX_MASK, P, false, nullptr);
        out[i] = lab;
        inside += lab == CELL_IN;
    }
    if (ctr) count_inside(inside, ctr + 3);
}

// ------------------------------------- pass-2 queue in leaf-window order --
//
// Pass 1 queues points in input order, so on inputs without spatial order
// (C2's near-edge points) the tiers' gathers of leaf and edge records sweep
// the whole index, which is larger than L2 (350-400 MB on the C1 polygon):
// nearly every record comes from DRAM, once per point.  Leaves are numbered
// so that their records are contiguous, so a window of consecutive leaves is
// a contiguous slice of the index.  Two launches put the queue in window
// order (a counting sort with a few dozen bins, block-aggregated):
//   k_part_count    entries per window (shared-memory counts, one global
//                   atomic per window and block);
//   k_part_scatter  each block ranks a tile's entries per window in shared
//                   memory, takes the tile's place in each window with one
//                   global atomic per window, and writes them there.
// The tiers' grid-stride loops then sweep the queue in order, so at any time
// the grid works in one or two windows whose records stay in L2, and tier 1
// writes the tier-2 queue in the same order.  Windows are sized at about
// PART_BYTES of index; queues below PART_MIN_QUEUE entries keep pass-1 order
// (both kernels return at once and the tiers read the pass-1 queue).
constexpr int PART_MAX = 64;
constexpr long long PART_BYTES = 24LL << 20;
constexpr unsigned int PART_MIN_QUEUE = 1u << 18;
constexpr int P_TPB = 256;
constexpr int P_ITEMS = 8;

struct PartScratch {
    unsigned int* total;   // [PART_MAX] entries per window; zero before the pass
    unsigned int* cursor;  // [PART_MAX] entries placed per window; zero before the pass
    unsigned int* done;    // set to 1 when the window-ordered arrays are complete; zero before the pass
    uint32_t* spts;        // point indices in window order
    uint32_t* sleaf;       // their leaf words
    int np;                // windows (>= 2)
    float scale;           // QueryView::part_scale
};

__device__ __forceinline__ int part_of(uint32_t w, int np, float scale)
{
    if ((w & KIND_MASK) != KIND_LEAF) return np - 1;  // a point pass 1 did not locate
    return min((int)(__uint2float_rz(w & INDEX_MASK) * scale), np - 1);
}

// Adds one per active lane to cnt[b] in shared memory, one atomic per group
// of lanes with the same b; returns the lane's rank (old value + position).
__device__ __forceinline__ unsigned int smem_rank(unsigned int* cnt, int b)
{
    const unsigned int act = __activemask();
    const unsigned int same = __match_any_sync(act, b);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(same) - 1;
    unsigned int base = 0;
    if (lane == leader) base = atomicAdd(cnt + b, (unsigned int)__popc(same));
    base = __shfl_sync(same, base, leader);
    return base + __popc(same & ((1u << lane) - 1u));
}

__global__ void __launch_bounds__(P_TPB) k_part_count(const uint32_t* __restrict__ l1,
                                                      const unsigned int* __restrict__ qcount, PartScratch S)
{
    __shared__ unsigned int s_cnt[PART_MAX];
    wait_for_predecessor();
    const unsigned int m = *qcount;
    if (m < PART_MIN_QUEUE) {
        allow_dependents();
        return;
    }
    for (int k = threadIdx.x; k < S.np; k += P_TPB) s_cnt[k] = 0;
    __syncthreads();
    for (unsigned int t = blockIdx.x * P_TPB + threadIdx.x; t < m; t += gridDim.x * P_TPB)
        smem_rank(s_cnt, part_of(l1[t], S.np, S.scale));
    __syncthreads();
    allow_dependents();
    for (int k = threadIdx.x; k < S.np; k += P_TPB)
        if (s_cnt[k]) atomicAdd(S.total + k, s_cnt[k]);
}

__global__ void __launch_bounds__(P_TPB) k_part_scatter(const uint32_t* __restrict__ queue,
                                                        const uint32_t* __restrict__ l1,
                                                        const unsigned int* __restrict__ qcount, PartScratch S)
{
    __shared__ unsigned int s_start[PART_MAX], s_cnt[PART_MAX], s_base[PART_MAX];
    wait_for_predecessor();
    const unsigned int m = *qcount;
    if (m < PART_MIN_QUEUE) {
        allow_dependents();
        return;
    }
    if (threadIdx.x == 0) {
        unsigned int run = 0;
        for (int k = 0; k < S.np; k++) {
            s_start[k] = run;
            run += S.total[k];
        }
    }
    for (int k = threadIdx.x; k < S.np; k += P_TPB) s_cnt[k] = 0;
    __syncthreads();
    constexpr int TILE = P_TPB * P_ITEMS;
    // block-uniform loop; per tile: ranks (s_cnt), barrier, the tile's place
    // in each window (s_base; s_cnt cleared), barrier, writes
    for (unsigned int base = blockIdx.x * TILE; base < m; base += gridDim.x * TILE) {
        uint32_t q[P_ITEMS], w[P_ITEMS];
        unsigned int r[P_ITEMS];
        int b[P_ITEMS];
#pragma unroll
        for (int k = 0; k < P_ITEMS; k++) {
            const unsigned int t = base + k * P_TPB + threadIdx.x;
            q[k] = t < m ? queue[t] : 0u;
            w[k] = t < m ? l1[t] : 0u;
            b[k] = part_of(w[k], S.np, S.scale);
        }
#pragma unroll
        for (int k = 0; k < P_ITEMS; k++)
            if (base + k * P_TPB + threadIdx.x < m) r[k] = smem_rank(s_cnt, b[k]);
        __syncthreads();
        for (int j = threadIdx.x; j < S.np; j += P_TPB) {
            const unsigned int c = s_cnt[j];
            if (c) s_base[j] = s_start[j] + atomicAdd(S.cursor + j, c);
            s_cnt[j] = 0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < P_ITEMS; k++) {
            if (base + k * P_TPB + threadIdx.x >= m) continue;
            const unsigned int at = s_base[b[k]] + r[k];
            if (at < m) {  // counts and entries agree; never write past the queue
                S.spts[at] = q[k];
                S.sleaf[at] = w[k];
            }
        }
    }
    allow_dependents();
    if (blockIdx.x == 0 && threadIdx.x == 0) *S.done = 1u;
}

// --------------------------------------- pass-2 queue in leaf order --
//
// The finest order: a counting sort of the pass-1 queue by leaf, so that the
// points of one leaf sit together and the warps of the first tier mostly
// take points of one leaf (their loads of the leaf's record and edge records
// are then one request per warp, served by L1 after the first).  Four
// launches:
//   k_ls_count      each entry takes its rank in its leaf (an atomic on the
//                   leaf's count; the last bucket holds points pass 1 did not
//                   locate);
//   k_ls_tile_sums  the counts' sums per tile of LS_TILE leaves;
//   k_ls_scan       each block scans one tile, starting from the sum of the
//                   tiles before it (no waits between blocks);
//   k_ls_scatter    each entry goes to its leaf's start plus its rank, point
//                   index and leaf word as one 8-byte pair (one random store
//                   per entry, where two arrays took two).
// The counts, ranks and the sorted arrays of a C2 pass fit in L2, so the
// random atomics and writes of the sort do not reach DRAM.
constexpr int LS_TPB = 256;
constexpr int LS_ITEMS = 16;
constexpr int LS_TILE = LS_TPB * LS_ITEMS;

struct LeafSortScratch {
    unsigned int* cnt;    // [nb] entries per bucket; zero before the pass
    unsigned int* start;  // [nb + 1] exclusive prefix of cnt
    unsigned int* tsum;   // [tiles] sums of cnt per tile
    unsigned int* rank;   // [queue] an entry's rank in its bucket
    uint2* sent;          // (point index, leaf word) in leaf order: one 8-byte store per entry
    unsigned int* done;   // set to 1 with the sorted arrays; zero before the pass
    int nb;               // buckets: leaves + 1
    int tiles;            // ceil(nb / LS_TILE)
    bool stage;           // tier 1 stages each tile's edge lists (k_leaf_t1s)
};

__device__ __forceinline__ int leaf_bucket(uint32_t w, int nb)
{
    return (w & KIND_MASK) == KIND_LEAF ? (int)min(w & INDEX_MASK, (uint32_t)(nb - 1)) : nb - 1;
}

__global__ void __launch_bounds__(LS_TPB) k_ls_count(const uint32_t* __restrict__ l1,
                                                     const unsigned int* __restrict__ qcount, LeafSortScratch S)
{
    wait_for_predecessor();
    const unsigned int m = *qcount;
    if (m >= PART_MIN_QUEUE)
        for (unsigned int t = blockIdx.x * LS_TPB + threadIdx.x; t < m; t += gridDim.x * LS_TPB)
            S.rank[t] = atomicAdd(S.cnt + leaf_bucket(l1[t], S.nb), 1u);
    allow_dependents();
}

// Block-wide sum of one value per thread (every thread gets it).
__device__ __forceinline__ unsigned int ls_block_sum(unsigned int v, unsigned int* s_w)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();  // s_w may still be read from the previous call
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned int t = 0;
#pragma unroll
    for (int k = 0; k < LS_TPB / 32; k++) t += s_w[k];
    return t;
}

__global__ void __launch_bounds__(LS_TPB) k_ls_tile_sums(const unsigned int* __restrict__ qcount, LeafSortScratch S)
{
    __shared__ unsigned int s_w[LS_TPB / 32];
    wait_for_predecessor();
    if (*qcount >= PART_MIN_QUEUE) {
        for (int tile = blockIdx.x; tile < S.tiles; tile += gridDim.x) {
            unsigned int v = 0;
            const int b0 = tile * LS_TILE;
            for (int k = threadIdx.x; k < LS_TILE; k += LS_TPB)
                if (b0 + k < S.nb) v += S.cnt[b0 + k];
            v = ls_block_sum(v, s_w);
            if (threadIdx.x == 0) S.tsum[tile] = v;
        }
    }
    allow_dependents();
}

__global__ void __launch_bounds__(LS_TPB) k_ls_scan(const unsigned int* __restrict__ qcount, LeafSortScratch S)
{
    __shared__ unsigned int s_w[LS_TPB / 32];
    __shared__ unsigned int s_wx[LS_TPB / 32];
    wait_for_predecessor();
    if (*qcount >= PART_MIN_QUEUE) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int tile = blockIdx.x; tile < S.tiles; tile += gridDim.x) {
            unsigned int before = 0;
            for (int k = threadIdx.x; k < tile; k += LS_TPB) before += S.tsum[k];
            before = ls_block_sum(before, s_w);
            // this thread's LS_ITEMS consecutive buckets
            const int b0 = tile * LS_TILE + threadIdx.x * LS_ITEMS;
            unsigned int c[LS_ITEMS], run = 0;
#pragma unroll
            for (int k = 0; k < LS_ITEMS; k++) {
                c[k] = b0 + k < S.nb ? S.cnt[b0 + k] : 0u;
                run += c[k];
            }
            // exclusive scan of the threads' totals: in the warp, then over warps
            unsigned int x = run;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            __syncthreads();  // s_wx may still be read from the previous tile
            if (lane == 31) s_wx[warp] = x;
            __syncthreads();
            unsigned int wbase = 0;
            for (int k = 0; k < warp; k++) wbase += s_wx[k];
            unsigned int at = before + wbase + x - run;
#pragma unroll
            for (int k = 0; k < LS_ITEMS; k++) {
                if (b0 + k < S.nb) S.start[b0 + k] = at;
                at += c[k];
            }
            if (b0 <= S.nb - 1 && S.nb - 1 < b0 + LS_ITEMS) S.start[S.nb] = at;  // the total
        }
    }
    allow_dependents();
}

__global__ void __launch_bounds__(LS_TPB) k_ls_scatter(const uint32_t* __restrict__ queue,
                                                       const uint32_t* __restrict__ l1,
                                                       const unsigned int* __restrict__ qcount, LeafSortScratch S)
{
    wait_for_predecessor();
    const unsigned int m = *qcount;
    if (m >= PART_MIN_QUEUE) {
        for (unsigned int t = blockIdx.x * LS_TPB + threadIdx.x; t < m; t += gridDim.x * LS_TPB) {
            const uint32_t w = l1[t];
            const unsigned int at = S.start[leaf_bucket(w, S.nb)] + S.rank[t];
            if (at < m) {  // counts and entries agree; never write past the queue
                S.sent[at] = make_uint2(queue[t], w);
            }
        }
    }
    allow_dependents();
    if (m >= PART_MIN_QUEUE && blockIdx.x == 0 && threadIdx.x == 0) *S.done = 1u;
}

// Launch with programmatic stream serialization (see wait_for_predecessor).
template <typename... KArgs, typename... Args>
void launch_dependent_tpb(void (*kernel)(KArgs...), int grid, int tpb, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(tpb);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename... KArgs, typename... Args>
void launch_dependent(void (*kernel)(KArgs...), int grid, cudaStream_t s, Args... args)
{
    launch_dependent_tpb(kernel, grid, TPB, s, args...);
}

// Tier counters (T.cnt[0..2]) must be zero.  stage_t1 (one polygon, queue
// in leaf order): tier 1 reads each tile's edge lists from shared memory
// (k_leaf_t1s).
template <class VS>
void leaf_tiers_launch(const VS& vs, const double2* ll, uint8_t* out, const uint32_t* queue,
                       const unsigned int* qcount, const Tiers& T, int precision, unsigned long long* ctr, int sms,
                       cudaStream_t s, bool stage_t1 = false)
{
    if (precision == GAHHG_QUERY_FP64_FILTER) {
        launch_dependent_tpb(k_leaf_t2<VS, true>, sms * T2_BLOCKS, T2_TPB, s, vs, ll, out, queue,
                             (const uint32_t*)T.l1, qcount, 0xffffffffu, T, ctr);
    } else {
        bool staged = false;
        if constexpr (std::is_same<VS, OneView>::value) {
            if (stage_t1) {
                launch_dependent(k_leaf_t1s, sms * T1S_BLOCKS, s, vs.Q, ll, out, queue, qcount, T, ctr,
                                 (int)knob(GAHHG_KNOB_STAGING_POLL_LIMIT));
                staged = true;
            }
        }
        if (!staged) launch_dependent(k_leaf_t1<VS>, sms * T1_BLOCKS, s, vs, ll, out, queue, qcount, T, ctr);
        launch_dependent_tpb(k_leaf_t2<VS, false>, sms * T2_BLOCKS, T2_TPB, s, vs, ll, out, (const uint32_t*)T.q2,
                             (const uint32_t*)T.l2, (const unsigned int*)T.cnt, T.cap2, T, ctr);
    }
    launch_dependent(k_leaf_t3<VS>, sms * 2, s, vs, ll, out, queue, qcount, T, ctr);
}

// Escalation queue capacities for a pass-2 queue of `points` entries.
inline void tier_caps(long long points, unsigned int* cap2, unsigned int* cap3)
{
    *cap2 = (unsigned int)(points / 2 + 1024);
    *cap3 = (unsigned int)(points / 8 + 1024);
}

}  // namespace

// ------------------------------------------------------------------ host --

gahhg_status lattice_query_with(const QueryView& Q, const double* d_lonlat, long long n, uint8_t* d_labels,
                                int precision, cudaStream_t s, uint64_t* d_counters, uint32_t* queue,
                                unsigned int* qcount, long long chunk, int device, const Tiers* tiers,
                                const PartScratch* part = nullptr, const LeafSortScratch* lsort = nullptr);

static const QueryView& make_view(const Grid* g) { return g->lattice->views[0]; }

// Windows of about PART_BYTES of the records the tiers gather per leaf.
void set_leaf_windows(QueryView& Q, long long nleaves, long long nrecs)
{
    const long long tier_bytes = nrecs * (long long)(sizeof(float4) + sizeof(uint32_t)) +
                                 nleaves * (long long)(sizeof(LeafRec) + 3 * sizeof(double));
    Q.nparts = (int)std::min<long long>(PART_MAX, std::max<long long>(1, (tier_bytes + PART_BYTES - 1) / PART_BYTES));
    if (nleaves < 2 * PART_MAX) Q.nparts = 1;
    Q.part_scale = Q.nparts > 1 ? (float)((double)Q.nparts / (double)nleaves) : 0.0f;
}

// Points per pass; the pass-2 queue holds one 4-byte index per point.
constexpr long long QUERY_CHUNK = 1LL << 27;

gahhg_status lattice_query(Grid* g, const double* d_lonlat, size_t n, uint8_t* d_labels, int precision,
                           cudaStream_t s, uint64_t* d_counters)
{
    if (n == 0) return GAHHG_OK;
    const QueryView Q = make_view(g);
    const long long chunk = std::min<long long>((long long)n, QUERY_CHUNK);
    // Words: [pass-2 queue: chunk][control: 192 (queue fill at +32, tier
    // counters at +33..35, window-order flag at +36, entries per window at
    // +64, windows' cursors at +128)][pass-2 leaf words: chunk][tier-2 queue]
    // [its leaf words][tier-3 queue][its leaf words][tier-2 masks][queue in
    // window order: points, leaf words (chunk each)].
    // One memset per pass clears the control words from the queue fill on.
    // [leaf order only: entries per leaf: nb][leaf starts: nb + 1][tile
    // sums][ranks: chunk].
    unsigned int cap2 = 0, cap3 = 0;
    tier_caps(chunk, &cap2, &cap3);
    const long long order = knob(GAHHG_KNOB_GROUPED_PASS2);
    const bool windows = order == 1 && Q.nparts > 1 && chunk >= PART_MIN_QUEUE;
    const bool leaves = (order == 2 || order == 3) && chunk >= PART_MIN_QUEUE && g->lattice->nleaves > 0 &&
                        g->lattice->nleaves < (1LL << 30);
    const int nb = leaves ? (int)g->lattice->nleaves + 1 : 0;
    const int tiles = (nb + LS_TILE - 1) / LS_TILE;
    const size_t l1_at = (size_t)chunk + 192;
    // even, so that the leaf order's (point, leaf word) pairs are 8-byte aligned
    const size_t sorted_at = (l1_at + (size_t)chunk + 3 * (size_t)cap2 + 2 * (size_t)cap3 + 1) & ~(size_t)1;
    const size_t ls_at = sorted_at + 2 * (size_t)chunk;
    const size_t words = windows ? ls_at : leaves ? ls_at + 2 * (size_t)nb + 1 + tiles + (size_t)chunk : sorted_at;
    uint32_t* queue = nullptr;
    GAHHG_TRY(pool_alloc((void**)&queue, sizeof(uint32_t) * words, g->device, s));
    unsigned int* qcount = (unsigned int*)(queue + chunk + 32);
    Tiers T;
    T.cnt = qcount + 1;
    T.l1 = queue + l1_at;
    T.q2 = T.l1 + chunk;
    T.l2 = T.q2 + cap2;
    T.q3 = T.l2 + cap2;
    T.l3 = T.q3 + cap3;
    T.m2 = T.l3 + cap3;
    T.cap2 = cap2;
    T.cap3 = cap3;
    PartScratch W;
    W.done = qcount + 4;
    W.total = queue + chunk + 64;
    W.cursor = queue + chunk + 128;
    W.spts = queue + sorted_at;
    W.sleaf = queue + sorted_at + chunk;
    W.np = Q.nparts;
    W.scale = Q.part_scale;
    LeafSortScratch LS;
    LS.done = qcount + 4;
    LS.sent = (uint2*)(queue + sorted_at);
    LS.cnt = queue + ls_at;
    LS.start = LS.cnt + nb;
    LS.tsum = LS.start + nb + 1;
    LS.rank = LS.tsum + tiles;
    LS.nb = nb;
    LS.tiles = tiles;
    LS.stage = order == 3;
    const gahhg_status st = lattice_query_with(Q, d_lonlat, (long long)n, d_labels, precision, s, d_counters,
                                               queue, qcount, chunk, g->device, &T, windows ? &W : nullptr,
                                               leaves ? &LS : nullptr);
    cudaFreeAsync(queue, s);
    return st;
}

// tiers == nullptr: one pass-2 launch with escalations inline (no queues
// beyond the pass-2 queue); else qcount[1..3] are the tier counters.
gahhg_status lattice_query_with(const QueryView& Q, const double* d_lonlat, long long n, uint8_t* d_labels,
                                int precision, cudaStream_t s, uint64_t* d_counters, uint32_t* queue,
                                unsigned int* qcount, long long chunk, int device, const Tiers* tiers,
                                const PartScratch* part, const LeafSortScratch* lsort)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    unsigned long long* ctr = (unsigned long long*)d_counters;
    for (long long off = 0; off < n; off += chunk) {
        const int m = (int)std::min<long long>(chunk, n - off);
        const double2* ll = (const double2*)d_lonlat + off;
        // the queue fill, the tier counters and, when ordering by window, the
        // flag, the counts and the cursors (the control words run up to them)
        const size_t zero_words = part ? (size_t)(part->cursor + PART_MAX - qcount) : lsort ? 5 : (tiers ? 4 : 1);
        GAHHG_CUDA_TRY(cudaMemsetAsync(qcount, 0, sizeof(unsigned int) * zero_words, s));
        if (lsort) GAHHG_CUDA_TRY(cudaMemsetAsync(lsort->cnt, 0, sizeof(unsigned int) * lsort->nb, s));
        const long long tiles = ((long long)m + TPB * LOC_UNROLL - 1) / (TPB * LOC_UNROLL);
        const int grid = (int)std::min<long long>(tiles, (long long)sms * 8);
        uint32_t* leafq = tiers ? tiers->l1 : nullptr;
        const int polls = (int)knob(GAHHG_KNOB_STAGING_POLL_LIMIT);
        auto kl = ctr ? k_locate<true> : k_locate<false>;
        kl<<<grid, TPB, summary_bytes(Q.swords), s>>>(ll, m, d_labels + off, Q, queue, leafq, qcount, ctr, polls);
        if (tiers && part) {
            // the pass-1 queue in window order, then the tiers over it
            launch_dependent_tpb(k_part_count, sms * 4, P_TPB, s, (const uint32_t*)tiers->l1,
                                 (const unsigned int*)qcount, *part);
            launch_dependent_tpb(k_part_scatter, sms * 4, P_TPB, s, (const uint32_t*)queue,
                                 (const uint32_t*)tiers->l1, (const unsigned int*)qcount, *part);
            Tiers T = *tiers;
            T.spts = part->spts;
            T.sleaf = part->sleaf;
            T.sorted = part->done;
            leaf_tiers_launch(OneView{Q}, ll, d_labels + off, queue, qcount, T, precision, ctr, sms, s);
        } else if (tiers && lsort) {
            // the pass-1 queue in leaf order, then the tiers over it
            const uint32_t* l1 = tiers->l1;
            const unsigned int* qc = qcount;
            launch_dependent_tpb(k_ls_count, sms * 8, LS_TPB, s, l1, qc, *lsort);
            launch_dependent_tpb(k_ls_tile_sums, std::min(lsort->tiles, sms * 8), LS_TPB, s, qc, *lsort);
            launch_dependent_tpb(k_ls_scan, std::min(lsort->tiles, sms * 8), LS_TPB, s, qc, *lsort);
            launch_dependent_tpb(k_ls_scatter, sms * 8, LS_TPB, s, (const uint32_t*)queue, l1, qc, *lsort);
            Tiers T = *tiers;
            T.spts = (const uint32_t*)lsort->sent;
            T.sleaf = T.spts + 1;
            T.sstride = 2;
            T.sorted = lsort->done;
            leaf_tiers_launch(OneView{Q}, ll, d_labels + off, queue, qcount, T, precision, ctr, sms, s,
                              lsort->stage);
        } else if (tiers) {
            leaf_tiers_launch(OneView{Q}, ll, d_labels + off, queue, qcount, *tiers, precision, ctr, sms, s);
        }
        else if (precision == GAHHG_QUERY_FP64_FILTER)
            k_leaf<false><<<sms * 4, TPB, 0, s>>>(ll, d_labels + off, Q, queue, qcount, ctr);
        else
            k_leaf<true><<<sms * 4, TPB, 0, s>>>(ll, d_labels + off, Q, queue, qcount, ctr);
        GAHHG_CUDA_TRY(cudaGetLastError());
    }
    return GAHHG_OK;
}

// ------------------------------------------------- allocation-free query --
//
// The same two passes as lattice_query, with the pass-2 queue in a fixed
// array in device memory instead of memory taken from the pool, for callers
// that must not allocate (see gahhg_query_device_noalloc in include/gahhg.h).
// Every device that loads this library reserves the array until the process
// exits.  All calls share it: calls that overlap on the GPU race.

constexpr long long NOALLOC_MAX_POINTS = 1LL << 21;  // 2,097,152 points per call
static __device__ __align__(256) uint32_t g_noalloc_queue[NOALLOC_MAX_POINTS + 64];

long long lattice_noalloc_max_points() { return NOALLOC_MAX_POINTS; }

// Device address of the array on the current device (the caller has made
// g->device current).  In host code `g_noalloc_queue` names a host-side
// stand-in, never the device array, so the address is asked of the runtime.
// It is looked up on every call rather than cached: after cudaDeviceReset
// (or any other teardown of the primary context) the module is loaded again
// and the array may sit at another address.  The lookup allocates nothing;
// the first one on a device loads the module there, which is why the first
// call on a device should come before any stream capture.
static gahhg_status noalloc_queue_address(int device, uint32_t** out)
{
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_queue);
    if (e != cudaSuccess || !p) {
        set_error("cudaGetSymbolAddress(g_noalloc_queue) on device %d: %s", device, cudaGetErrorString(e));
        return GAHHG_ERR_CUDA;
    }
    *out = (uint32_t*)p;
    return GAHHG_OK;
}

gahhg_status lattice_query_noalloc(Grid* g, const double* d_lonlat, size_t n, uint8_t* d_labels, int precision,
                                   cudaStream_t s)
{
    if ((long long)n > NOALLOC_MAX_POINTS) {
        set_error("gahhg_query_device_noalloc: %zu points exceed the fixed maximum of %lld per call", n,
                  NOALLOC_MAX_POINTS);
        return GAHHG_ERR_CAPACITY;
    }
    if ((uintptr_t)d_lonlat & 15u) {
        set_error("exact queries read lon/lat in 16-byte units: the device buffer must be 16-byte aligned");
        return GAHHG_ERR_ARG;
    }
    uint32_t* queue = nullptr;
    GAHHG_TRY(noalloc_queue_address(g->device, &queue));
    if (n == 0) return GAHHG_OK;
    const QueryView Q = make_view(g);
    // the queue count lives after the queue; lattice_query_with zeroes it before each pass
    unsigned int* qcount = (unsigned int*)(queue + NOALLOC_MAX_POINTS + 32);
    return lattice_query_with(Q, d_lonlat, (long long)n, d_labels, precision, s, nullptr, queue, qcount,
                              NOALLOC_MAX_POINTS, g->device, nullptr);
}

// ------------------------------------------------------- batch launcher --

size_t lattice_view_bytes() { return sizeof(QueryView); }
size_t batch_chunk_bytes() { return sizeof(BatchChunk); }

gahhg_status lattice_staging_fallbacks(int device, unsigned long long* out)
{
    GAHHG_CUDA_TRY(cudaSetDevice(device));
    unsigned int v = 0;
    GAHHG_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_tma_timeouts, sizeof(v)));
    *out = v;
    return GAHHG_OK;
}

// Chunks of at most `chunk_points` points, segment after segment.
// A segment's chunks hold at least 16 points per word of its summary, so
// staging the summary costs at most a quarter byte per point.
void batch_write_chunks(const long long* offsets, int nseg, int chunk_points, const int* swords, const int* seg_view,
                        void* out, int* nchunks)
{
    BatchChunk* v = (BatchChunk*)out;
    int n = 0;
    for (int p = 0; p < nseg; p++) {
        const long long step = std::max<long long>(chunk_points, 16LL * (swords ? swords[p] : 0));
        for (long long a = offsets[p]; a < offsets[p + 1]; a += step) {
            BatchChunk c;
            c.view = seg_view ? seg_view[p] : p;
            c.start = a;
            c.count = (int)std::min<long long>(step, offsets[p + 1] - a);
            if (v) v[n] = c;
            n++;
        }
    }
    *nchunks = n;
}

size_t batch_chunk_count_bound(long long points, int nseg, int chunk_points)
{
    return (size_t)(points / std::max(chunk_points, 1)) + (size_t)nseg + 1;
}

void batch_make_chunks(const long long* offsets, int nseg, int chunk_points, const int* swords, const int* seg_view,
                       std::vector<uint8_t>& out, int* nchunks)
{
    int n = 0;
    batch_write_chunks(offsets, nseg, chunk_points, swords, seg_view, nullptr, &n);
    out.resize((size_t)n * sizeof(BatchChunk));
    batch_write_chunks(offsets, nseg, chunk_points, swords, seg_view, out.data(), nchunks);
}

// Launches the batch locate instance of shape `shape` (statistics on when
// `ctr` is set).
template <int I>
static void batch_locate_launch(int shape, int grid, cudaStream_t s, const QueryView* views, const BatchChunk* chunks,
                                int nchunks, unsigned int* next_chunk, const double2* ll, uint8_t* out,
                                uint32_t* queue, uint32_t* leafq, unsigned int* qcount, unsigned long long* ctr,
                                int polls)
{
    if constexpr (I < BATCH_NSHAPES) {
        if (shape != I) {
            batch_locate_launch<I + 1>(shape, grid, s, views, chunks, nchunks, next_chunk, ll, out, queue, leafq,
                                       qcount, ctr, polls);
            return;
        }
        constexpr int U = BATCH_SHAPES[I].unroll, B = BATCH_SHAPES[I].blocks;
        if (ctr)
            k_batch_locate<true, U, B><<<grid, TPB, 0, s>>>(views, chunks, nchunks, next_chunk, ll, out, queue, leafq,
                                                            qcount, ctr, polls);
        else
            k_batch_locate<false, U, B><<<grid, TPB, 0, s>>>(views, chunks, nchunks, next_chunk, ll, out, queue,
                                                             leafq, qcount, ctr, polls);
    }
}

int batch_shape_count() { return BATCH_NSHAPES; }

bool batch_shape_info(int shape, int* points_per_thread, int* blocks_per_sm)
{
    if (shape < 0 || shape >= BATCH_NSHAPES) return false;
    if (points_per_thread) *points_per_thread = BATCH_SHAPES[shape].unroll;
    if (blocks_per_sm) *blocks_per_sm = BATCH_SHAPES[shape].blocks;
    return true;
}

size_t batch_queue_words(long long queue_cap)
{
    unsigned int cap2 = 0, cap3 = 0;
    tier_caps(queue_cap, &cap2, &cap3);
    return 2 * ((size_t)queue_cap + cap2 + cap3) + cap2;
}

// counters: [0] queue count, [1] next chunk, [2..4] tier counters.  The
// queue holds batch_queue_words(queue_cap) words: the pass-2 queue and its
// leaf words, then the escalation queues, each followed by its leaf words.  Everything is enqueued on `s` (no allocation, no host
// synchronisation), so it can be captured in a graph.
gahhg_status batch_query_launch(const void* d_views, const void* d_chunks, int nchunks, const double* d_lonlat,
                                uint8_t* d_labels, int precision, uint32_t* queue, long long queue_cap,
                                unsigned int* counters, uint64_t* d_stats, cudaStream_t s, int device,
                                bool zero_counters, int shape)
{
    if (nchunks == 0) return GAHHG_OK;
    static std::atomic<int> sms_cache[64];
    int sms = (device >= 0 && device < 64) ? sms_cache[device].load(std::memory_order_relaxed) : 0;
    if (!sms) {
        sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (device >= 0 && device < 64) sms_cache[device].store(sms, std::memory_order_relaxed);
    }
    const QueryView* views = (const QueryView*)d_views;
    const BatchChunk* chunks = (const BatchChunk*)d_chunks;
    unsigned long long* ctr = (unsigned long long*)d_stats;
    if (zero_counters) GAHHG_CUDA_TRY(cudaMemsetAsync(counters, 0, 5 * sizeof(unsigned int), s));
    Tiers T;
    tier_caps(queue_cap, &T.cap2, &T.cap3);
    T.l1 = queue + queue_cap;
    T.q2 = T.l1 + queue_cap;
    T.l2 = T.q2 + T.cap2;
    T.q3 = T.l2 + T.cap2;
    T.l3 = T.q3 + T.cap3;
    T.m2 = T.l3 + T.cap3;
    T.cnt = counters + 2;
    const int polls = (int)knob(GAHHG_KNOB_STAGING_POLL_LIMIT);
    if (shape < 0 || shape >= BATCH_NSHAPES) shape = 0;
    const int grid = std::min(nchunks, sms * BATCH_SHAPES[shape].blocks);  // persistent: every block resident
    batch_locate_launch<0>(shape, grid, s, views, chunks, nchunks, counters + 1, (const double2*)d_lonlat, d_labels,
                           queue, T.l1, counters, ctr, polls);
    leaf_tiers_launch(ChunkViews{views, chunks, nchunks}, (const double2*)d_lonlat, d_labels, queue, counters, T,
                      precision, ctr, sms, s);
    GAHHG_CUDA_TRY(cudaGetLastError());
    return GAHHG_OK;
}

}  // namespace gahhg
