// lattice.cu - exact-label query index and query kernel.
//
// The reference answers a query by descending the hexagon hierarchy from 42
// level-0 cells (kernel_PISP, source/GPISPAHHG.cu:1422-1504): about ten
// dependent levels of plane tests per point.  Here the same question is
// answered from a lattice over longitude/latitude that is indexed directly
// from the input coordinates (the lattice itself, and how it is built:
// lattice_build.cu).
//
// A query reads lon/lat (16 B), computes the top cell with two FP64
// multiply-adds, follows inner nodes by exact power-of-two scaling, and
//   - in a cell without edges writes the cell's label (no trigonometry);
//   - in a leaf counts crossings of arc(R, q) with the leaf's edges:
//       s2 = orient(A,B,q) = q.(A x B), s3 = orient(R,q,A) = q.(A x R),
//       s4 = orient(R,q,B) = q.(B x R), s1 = orient(A,B,R) stored exactly;
//     each sign is first taken in FP32 (in the leaf's tangent frame, from the
//     angle differences to R: local_frame.cuh) against a forward error bound,
//     then in FP64 on the canonical q, then exactly (exact_pred.cuh).  Labels
//     are therefore those of the exact oracle; the FP32 stage only decides when
//     its bound proves the sign.
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

// ------------------------------------------------------------- query ----

// A query point: input longitude and FakeLL latitude (what the canonical XYZ is made from).
struct PointCtx {
    double lon, lat;
};

__device__ __forceinline__ int sign_exactly(const double* x, const double* y, const double* z)
{
    const int s = exact::orient_fp64(x, y, z);
    return s != 0 ? s : exact::orient_exact(x, y, z);
}

__device__ __forceinline__ void load_ends(const QueryView& Q, uint32_t e, double* A, double* B)
{
    const double2* p = Q.ends + 3 * (size_t)e;
    const double2 u = __ldg(p), v = __ldg(p + 1), w = __ldg(p + 2);
    A[0] = u.x;
    A[1] = u.y;
    A[2] = v.x;
    B[0] = v.y;
    B[1] = w.x;
    B[2] = w.y;
}

// The complete crossing test of a point in a leaf: FP64 filter, then exact
// expansions with simulation of simplicity.  A call, not inlined: the few
// points that need it must not cost the others registers.
__device__ __noinline__ uint8_t leaf_label_exact(const QueryView* Qp, uint32_t leaf, double lon, double lat)
{
    const QueryView& Q = *Qp;
    const LeafRec* Lp = Q.leaves + leaf;
    const uint32_t off = Lp->off;
    const int cnt = Lp->cnt;
    const uint8_t label = Lp->label;
    const double LR[3] = {Q.aux[leaf].R[0], Q.aux[leaf].R[1], Q.aux[leaf].R[2]};
    double q[3];
    gahhg_canon_vertex_xyz(lon, lat, q);
    if (exact::same(q, LR)) {  // q is the center: its label, unless it is a vertex
        for (int k = 0; k < cnt; k++) {
            double A[3], B[3];
            load_ends(Q, __ldg(Q.eids + off + k) & 0x7fffffffu, A, B);
            if (exact::same(q, A) || exact::same(q, B)) return CELL_IN;
        }
        return label;
    }
    int par = 0;
    for (int k = 0; k < cnt; k++) {
        const uint32_t es = __ldg(Q.eids + off + k);
        const int s1 = (es >> 31) ? 1 : -1;
        double A[3], B[3];
        load_ends(Q, es & 0x7fffffffu, A, B);
        if (exact::same(q, A) || exact::same(q, B)) return CELL_IN;  // vertex rule
        const int s2 = sign_exactly(A, B, q);
        if (s2 == s1) continue;
        if (sign_exactly(LR, q, A) != s2) continue;  // a crossing needs orient(R, q, A) == s2
        if (sign_exactly(LR, q, B) == -s2) par ^= 1;
    }
    return (uint8_t)(par ? 3 - label : label);
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
// the size is rounded up to 16 bytes (in the index every summary starts at a
// multiple of four words and the last one is padded to one, so the copy reads
// no further).  Every wait is bounded; a wait that runs out is counted in
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

constexpr int SUMMARY_WORDS_MAX = 4096;  // 65,536 coarse cells of 2 bits: 16 KB
__host__ __device__ __forceinline__ uint32_t summary_bytes(int swords) { return ((uint32_t)swords * 4u + 15u) & ~15u; }

// ------------------------------------------------------ escalation tiers --
//
// The crossing tests run in tiers, so that no warp carries the registers or
// waits on the branches of a rarer, costlier tier:
//   tier 1: every sign from the certified FP32 filter in the leaf's local
//           frame (local_frame.cuh);
//   tier 2: the canonical FP64 point, the vertex and center rules, and every
//           sign from the FP64 filter on translated rows (orient_fp64_near);
//   the complete test (leaf_label_exact) for what is left.
// Every sign a tier returns is exact, so a label does not depend on the tier
// that produced it.
constexpr uint8_t LABEL_DEFER = 0xFF;

// Tier 1 runs every edge of the leaf: a decided edge adds its crossing to
// the parity, an undecided one is noted in `mask` (bit k for record k < 31)
// and the FP64 tier evaluates only those, starting from the label that the
// decided ones give (bit 31: inside).  The label is exact either way: the
// crossing parity is the XOR of independent per-edge tests.  MASK_ALL asks
// tier 2 for every edge (a record beyond the 31st undecided, or the offset
// refused).
constexpr uint32_t MASK_ALL = 0xFFFFFFFFu;

// Records beyond the leaf's own two whose loads tier 1 issues together (most
// leaves have at most four edges; groups of four: 263 us where two take 251).
constexpr int T1_GROUP = 2;

// A leaf as tier 1 reads it: four 16-byte loads of one line in flight.
struct LeafLoad {
    double lon, lat;
    uint32_t off, cnt_label;
    float sb, cb;
    float4 r0, r1;
    __device__ __forceinline__ int cnt() const { return (int)(cnt_label & 0xFFFFu); }
    __device__ __forceinline__ uint32_t label() const { return (cnt_label >> 16) & 0xFFu; }
};

template <bool SHARED>
__device__ __forceinline__ LeafLoad load_leaf(const LeafRec* p)
{
    const float4* f = reinterpret_cast<const float4*>(p);
    float4 a, b;
    LeafLoad L;
    if constexpr (SHARED) {
        a = f[0];
        b = f[1];
        L.r0 = f[2];
        L.r1 = f[3];
    } else {
        a = __ldg(f);
        b = __ldg(f + 1);
        L.r0 = __ldg(f + 2);
        L.r1 = __ldg(f + 3);
    }
    L.lon = __hiloint2double(__float_as_int(a.y), __float_as_int(a.x));
    L.lat = __hiloint2double(__float_as_int(a.w), __float_as_int(a.z));
    L.off = __float_as_uint(b.x);
    L.cnt_label = __float_as_uint(b.y);
    L.sb = b.z;
    L.cb = b.w;
    return L;
}

// A record of tier 1: from global memory through the read-only path, or
// from a copy in shared memory (SHARED).
template <bool SHARED>
__device__ __forceinline__ float4 t1_record(const float4* p)
{
    if constexpr (SHARED) return *p;
    else return __ldg(p);
}

// Tier 1 on the leaf L whose third record and on are at rec + 2 ... (global
// memory, or the staged copy in shared memory when SHARED).
template <bool SHARED>
__device__ __forceinline__ uint8_t leaf_label_fp32(const float4* rec, const LeafLoad& L, const PointCtx& P,
                                                 uint32_t& mask)
{
    const int cnt = L.cnt();
    local_frame::Frame f;
    mask = MASK_ALL;
    if (!(fabs(P.lon) <= 540.0) || !local_frame::frame_at(P.lon, P.lat, L.lon, L.lat, L.sb, L.cb, f))
        return LABEL_DEFER;
    local_frame::Tests t;
    local_frame::tests_of(f, t);
    uint32_t par = L.label() == CELL_IN;
    uint32_t und = 0;
    bool all = false;
    auto take = [&](const float4& r, int k) {
        const int x = local_frame::record_crossing(t, r.x, r.y, r.z, r.w);
        if (x > 0) par ^= 1u;
        if (x < 0) {
            if (k < 31) und |= 1u << k;
            else all = true;
        }
    };
    take(L.r0, 0);
    if (cnt > 1) take(L.r1, 1);
    for (int k0 = LEAF_INLINE; k0 < cnt; k0 += T1_GROUP) {
        float4 r[T1_GROUP];
#pragma unroll
        for (int j = 0; j < T1_GROUP; j++) r[j] = t1_record<SHARED>(rec + min(k0 + j, cnt - 1));
#pragma unroll
        for (int j = 0; j < T1_GROUP; j++)
            if (k0 + j < cnt) take(r[j], k0 + j);
    }
    if (all) return LABEL_DEFER;
    if (und) {
        mask = und | (par << 31);
        return LABEL_DEFER;
    }
    return (uint8_t)(1u + par);
}

// Records beyond the leaf's own two whose ends the FP64 tier loads together.
constexpr int T2_GROUP = 2;

// A warp's 32 aux lines in shared memory: line r's 16-byte part q lies at
// aux_slot(r, q) (the permutation keeps lanes that read the same part of their
// lines off each other's banks).
__device__ __forceinline__ int aux_slot(int r, int q) { return 8 * r + (q ^ (r & 7)); }

// Brings the lines (null: none) there by the warp together, eight lanes a
// line: an instruction touches four lines and not 32.
__device__ __forceinline__ void copy_aux(uint4* s_aux, const LeafAux* mine)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int r = 4 * j + (lane >> 3), q = lane & 7;
        const unsigned long long a = __shfl_sync(0xffffffffu, (unsigned long long)mine, r);
        if (a)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(s_aux + aux_slot(r, q))),
                         "l"(a + 16 * q)
                         : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// FP64 tier on the leaf's records selected by `mask` (MASK_ALL: every record,
// from the leaf's label; else the records of bits 0..30, from the label of
// bit 31): the leaf's aux line (in the lane's place in shared memory, or
// global memory when s_aux is null), and edge words and ends beyond its two
// edges.  q: the point's canonical XYZ.
template <bool SHARED>
__device__ __forceinline__ uint8_t leaf_label_fp64(const QueryView& Q, uint32_t leaf, const uint4* s_aux,
                                                   const double* q, uint32_t mask)
{
    const LeafAux* X = Q.aux + leaf;
    const int lane = threadIdx.x & 31;
    const uint4* xp = reinterpret_cast<const uint4*>(X);
    const uint4 xa = SHARED ? s_aux[aux_slot(lane, 0)] : __ldg(xp), xb = SHARED ? s_aux[aux_slot(lane, 1)] : __ldg(xp + 1);
    double2 e[T2_GROUP][3];
    static_assert(T2_GROUP == LEAF_INLINE, "the line's edges are the first group");
    // the line's ends go out with its header, the second edge's when it is asked for
#pragma unroll
    for (int j = 0; j < LEAF_INLINE; j++) {
        const double2* p = reinterpret_cast<const double2*>(X->ends[j]);
        const double2* sp = reinterpret_cast<const double2*>(s_aux);
        if (mask >> j & 1u)
#pragma unroll
            for (int k = 0; k < 3; k++) e[j][k] = SHARED ? sp[aux_slot(lane, 2 + 3 * j + k)] : __ldg(p + k);
    }
    const double LR[3] = {__hiloint2double((int)xa.y, (int)xa.x), __hiloint2double((int)xa.w, (int)xa.z),
                          __hiloint2double((int)xb.y, (int)xb.x)};
    const uint32_t off = xb.z;
    uint32_t par = mask >> 31, sel = mask & 0x7fffffffu;
    int left = 0;  // records after the selected ones (MASK_ALL on a long leaf)
    if (mask == MASK_ALL) {
        const int cnt = (int)(xb.w & 0xFFFFu);
        par = ((xb.w >> 16) & 0xFFu) == CELL_IN;
        left = max(0, cnt - 31);
        sel = cnt >= 31 ? 0x7fffffffu : (1u << cnt) - 1u;
    }
    // bits of the group's edges and of their signs (orient(A, B, R) > 0)
    uint32_t group = sel & 3u, signs = xb.w >> 24, k0 = 0;
    sel &= ~3u;
    for (;;) {
#pragma unroll
        for (int j = 0; j < T2_GROUP; j++) {
            if (!(group >> j & 1u)) continue;
            const int s1 = (signs >> j & 1u) ? 1 : -1;
            const double A[3] = {e[j][0].x, e[j][0].y, e[j][1].x}, B[3] = {e[j][1].y, e[j][2].x, e[j][2].y};
            if (exact::same(q, A) || exact::same(q, B)) return CELL_IN;  // vertex rule
            if (exact::same(q, LR)) return LABEL_DEFER;                  // q is the center: the complete test
            // every row is within a cell of the first: translated rows keep the bound small
            const int s2 = exact::orient_fp64_near(A, B, q);
            if (s2 == 0) return LABEL_DEFER;
            if (s2 == s1) continue;
            const int s3 = exact::orient_fp64_near(LR, q, A);
            if (s3 == 0) return LABEL_DEFER;
            if (s3 != s2) continue;
            const int s4 = exact::orient_fp64_near(LR, q, B);
            if (s4 == 0) return LABEL_DEFER;
            if (s4 == -s2) par ^= 1u;
        }
        if (!sel) {
            if (left <= 0) break;
            k0 += 31;
            const int n = min(left, 31);
            sel = n == 31 ? 0x7fffffffu : (1u << n) - 1u;
            left -= n;
        }
        group = signs = 0;
#pragma unroll
        for (int j = 0; j < T2_GROUP; j++) {
            if (!sel) break;
            const uint32_t word = __ldg(Q.eids + off + k0 + __ffs(sel) - 1);
            sel &= sel - 1u;
            group |= 1u << j;
            signs |= (word >> 31) << j;
            const double2* p = Q.ends + 3 * (size_t)(word & 0x7fffffffu);
            e[j][0] = __ldg(p);
            e[j][1] = __ldg(p + 1);
            e[j][2] = __ldg(p + 2);
        }
    }
    return (uint8_t)(1u + par);
}

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

// The label of a point whose coarse cell has no edges (or that lies outside
// the domain), 0 for a mixed cell and for unusual coordinates.  Straight to
// the coarse cell, without the top cell: a point that rounding puts beyond a
// coarse border is within the margin of both cells, and beyond the domain's
// end a partial last cell has the outside's label if it has one.  Pass 1 of a
// query over the whole sphere is bound by its instructions (62-69 % of the
// issue slots at 60 to 85 per 32 points, through the top cell, its checks and
// the tests of the domain's sides), so this is straight-line code of about 15:
// conversions that saturate at 0, one minimum per axis, the ring of the
// summary for everything outside.
__device__ __forceinline__ uint32_t coarse_label(const QueryView& Q, const uint32_t* __restrict__ sum, double lo,
                                                 double la)
{
    double u = fma(lo, Q.cu, Q.cu0);
    if (Q.cwrap) u += u < 1.0 ? Q.cu360 : 0.0;
    const double v = fma(la, Q.cv, Q.cv0);
    const unsigned int x = min(__double2uint_rz(u), (unsigned int)Q.SW - 1u);
    const unsigned int y = min(__double2uint_rz(v), (unsigned int)Q.SH - 1u);
    const unsigned int c = y * (unsigned int)Q.SW + x;
    const uint32_t w = sum[c >> 4] >> ((c & 15u) << 1);
    const bool ok = (fabs(lo) <= 180.0) & (fabs(la) <= 90.0);
    return ok ? w & 3u : 0u;
}

// A cell fraction in [0, 1) as a 32-bit binary fraction, saturating (below 0
// gives 0, 1 and above all ones).  Its base-4 digits are the children that
// the recursion f -> 4 f - floor(4 f) (clamped to 0..3) visits: that FP64
// recursion is exact, so digit k of the fraction is its k-th child for the
// first 16 levels, and for the clamped out-of-range cases both give 0 or 3 at
// every level.  The lattice has at most MAX_DESCENT levels below the top.
constexpr int MAX_DESCENT = 16;
static_assert(MAX_LEVEL <= MAX_DESCENT, "two bits of a fraction per level");
__device__ __forceinline__ uint32_t frac_bits(double f) { return __double2uint_rz(f * 4294967296.0); }

__device__ __forceinline__ uint32_t descend_bits(const QueryView& Q, uint32_t w, uint32_t U, uint32_t V)
{
    while ((w & KIND_MASK) == KIND_INNER) {
        w = __ldg(Q.nodes + (w & INDEX_MASK) + (V >> 30) * FAN + (U >> 30));
        U <<= 2;
        V <<= 2;
    }
    return w;
}

__device__ __forceinline__ uint32_t descend(const QueryView& Q, uint32_t w, double fu, double fv)
{
    return descend_bits(Q, w, frac_bits(fu), frac_bits(fv));
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
// Leaf word of a queued point that was not located (its coordinates are
// unusual, or it is out of a pure node).
constexpr uint32_t LEAF_UNKNOWN = KIND_PURE;

__device__ __forceinline__ bool usual(double lo, double laf) { return laf >= 0.0 && laf <= 180.0 && fabs(lo) <= 540.0; }

// The point's context, and its node word: `known` when it was located (any
// leaf the locate arithmetic finds serves: every cell's rectangle holds its
// points with a margin above that arithmetic's rounding), else a descent from
// the top, for unusual input from the canonical XYZ itself.
__device__ __forceinline__ uint32_t point_leaf(const QueryView& Q, double2 p, PointCtx& P,
                                              uint32_t known = LEAF_UNKNOWN)
{
    P.lat = gahhg_canon_query_lat(p.y);
    P.lon = p.x;
    if (known != LEAF_UNKNOWN) return known;
    double lo = P.lon, la = P.lat;
    if (!(fabs(lo) <= 540.0 && fabs(la) <= 90.0)) {
        double q[3];
        gahhg_canon_vertex_xyz(P.lon, P.lat, q);
        la = asin(fmin(1.0, fmax(-1.0, q[1]))) / RAD;
        lo = atan2(q[0], q[2]) / RAD;
    }
    Loc L;
    const bool in = domain_locate(Q, lo, la + 90.0, L);
    return in ? descend(Q, __ldg(Q.nodes + (size_t)L.iy * Q.W + L.ix), L.fu, L.fv) : Q.outside;
}

// ------------------------------------------------------- pass 1 (locate) --

// The pass-1 queue is filled in parts, block b into part b % parts, each with
// its own counter on a line of its own: an atomic that returns a value takes
// about 1.3 ns on one address, one after the other, so a single counter held
// queries whose points in leaves are spread over all tiles to 0.75 G tiles/s
// (1e8 uniform points on the 1,100-edge polygon, a few in every tile: 1075 us
// of locate, of which the counter was the most).  A part has room for all
// points of its blocks.
constexpr int QUEUE_PARTS = 64;
constexpr int COUNTER_STRIDE = 32;  // words between counters

// Pass 1 over one polygon.  A warp's points in mixed blocks wait in shared
// memory and descend 32 at a time: most tiles of a query over the whole sphere
// have a few of them, and descending where they stood cost a tile up to four
// chains of node loads one after the other, on a few lanes each.
constexpr int LOC_QUEUE = 32 + 32 * LOC_UNROLL;
// 32 registers, 64 warps per SM: the pass is bound by the latency of its
// streams (17 B a point; 255 us for 1e8 points at the copy rate), and warps
// hide it better than loads in flight per warp do: six blocks 354 us where
// eight take 296 (1e8 uniform points on the 1.1M-edge polygon).
constexpr int LOC_BLOCKS = 8;

// A warp's tile is LOC_UNROLL / 2 rows of 64 points, a lane's two of a row
// side by side, through 16-byte loads.  (1e8 uniform points on the 1.1M-edge
// polygon: 295 us of locate this way, 320-330 with 32-byte loads or evict-first
// hints on them; on the 1,100-edge polygon 286, and 323 with evict-first.)
template <bool STATS>
__device__ __forceinline__ void locate_points(const QueryView& Q, const uint32_t* __restrict__ sum,
                                              const double2* __restrict__ ll, int n, uint8_t* __restrict__ out,
                                              uint32_t* __restrict__ queue, uint32_t* __restrict__ leafq,
                                              unsigned int* __restrict__ qcount, uint32_t qbase, uint32_t* mixed,
                                              int& inside)
{
    constexpr int ROWS = LOC_UNROLL / 2;
    static_assert(LOC_UNROLL == 4, "rows of two points per lane, four labels in a word");
    const int lane = threadIdx.x & 31;
    int nm = 0;  // points in `mixed`, the same in every lane
    constexpr int TILE = TPB * LOC_UNROLL;
    for (int base = blockIdx.x * TILE;; base += gridDim.x * TILE) {
        const bool last = base >= n;
        if (!last) {
            const int i = base + (threadIdx.x & ~31) * LOC_UNROLL + 2 * lane;  // row r: points i + 64 r, i + 64 r + 1
            uint32_t lab = 0;   // labels, a byte each; 0: mixed (or LABEL_PENDING, the same)
            uint32_t skip = 0;  // beyond the last point
            if (base + TILE <= n) {
                double2 a[ROWS], b[ROWS];
#pragma unroll
                for (int r = 0; r < ROWS; r++) {
                    a[r] = __ldg(ll + i + 64 * r);
                    b[r] = __ldg(ll + i + 64 * r + 1);
                }
#pragma unroll
                for (int r = 0; r < ROWS; r++) {
                    const uint32_t l = coarse_label(Q, sum, a[r].x, a[r].y) | coarse_label(Q, sum, b[r].x, b[r].y) << 8;
                    lab |= l << (16 * r);
                    out[i + 64 * r] = (uint8_t)l;
                    out[i + 64 * r + 1] = (uint8_t)(l >> 8);
                }
            } else {
#pragma unroll
                for (int k = 0; k < LOC_UNROLL; k++) {
                    const int j = i + 64 * (k >> 1) + (k & 1);
                    if (j < n) {
                        const double2 q = __ldg(ll + j);
                        const uint32_t l = coarse_label(Q, sum, q.x, q.y);
                        lab |= l << (8 * k);
                        out[j] = (uint8_t)l;
                    } else {
                        skip |= 1u << (8 * k);
                    }
                }
            }
            if (STATS) inside += __popc(lab & 0x02020202u);
            const uint32_t mixed4 = ~(lab | (lab >> 1) | skip) & 0x01010101u;  // a bit per mixed point
            if (__any_sync(0xffffffffu, mixed4 != 0)) {
#pragma unroll
                for (int k = 0; k < LOC_UNROLL; k++) {
                    const bool push = (mixed4 >> (8 * k)) & 1u;
                    const unsigned int mk = __ballot_sync(0xffffffffu, push);
                    if (push) mixed[nm + __popc(mk & ((1u << lane) - 1u))] = (uint32_t)(i + 64 * (k >> 1) + (k & 1));
                    nm += __popc(mk);
                }
            }
            __syncwarp();  // (orders the labels before those that B writes, too)
        }
        while (nm >= 32 || (last && nm > 0)) {
            const int m = min(nm, 32);
            nm -= m;
            uint32_t i = 0, w = KIND_PURE | 1u;
            if (lane < m) {
                i = mixed[nm + lane];
                const double2 p = __ldg(ll + i);
                const double laf = p.y + 90.0;
                Loc L;
                if (usual(p.x, laf))
                    w = domain_locate(Q, p.x, laf, L)
                            ? descend(Q, __ldg(Q.nodes + (size_t)L.iy * Q.W + L.ix), L.fu, L.fv)
                            : Q.outside;
                else if (isfinite(p.x) && isfinite(p.y))
                    w = LEAF_UNKNOWN;  // unusual coordinates: tier 1 locates them
                else
                    w = KIND_PURE | 4u;  // non-finite input stays undefined (LABEL_PENDING)
                if ((w & KIND_MASK) == KIND_PURE && (w & 3u)) {
                    out[i] = (uint8_t)(w & 3u);
                    if (STATS) inside += (w & 3u) == CELL_IN;
                }
            }
            const bool leaf = (w & KIND_MASK) != KIND_PURE || w == LEAF_UNKNOWN;
            const unsigned int mk = __ballot_sync(0xffffffffu, leaf);
            if (mk) {
                unsigned int pos = 0;
                if (lane == 0) pos = atomicAdd(qcount, (unsigned int)__popc(mk));
                pos = __shfl_sync(0xffffffffu, pos, 0) + qbase + __popc(mk & ((1u << lane) - 1u));
                if (leaf) {
                    queue[pos] = i;
                    leafq[pos] = w;
                }
            }
            __syncwarp();
        }
        if (last) break;
    }
}

template <bool STATS>
__global__ void __launch_bounds__(TPB, LOC_BLOCKS) k_locate(const double2* __restrict__ ll, int n,
                                                           uint8_t* __restrict__ out,
                                                           const __grid_constant__ QueryView Q,
                                                           uint32_t* __restrict__ queue, uint32_t* __restrict__ leafq,
                                                           unsigned int* __restrict__ qcount, int parts,
                                                           unsigned int part_cap, unsigned long long* ctr,
                                                           int poll_limit)
{
    extern __shared__ __align__(16) uint32_t s_sum[];
    __shared__ uint32_t s_mixed[TPB / 32][LOC_QUEUE];
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
    const unsigned int part = blockIdx.x % (unsigned int)parts;
    uint32_t* mixed = s_mixed[threadIdx.x >> 5];
    int inside = 0;
    if (s_late == 0) {
        locate_points<STATS>(Q, s_sum, ll, n, out, queue, leafq, qcount + part * COUNTER_STRIDE, part * part_cap, mixed,
                             inside);
    } else {
        // after a wait that ran out the block reads the summary from global
        // memory and never touches s_sum, which the pending copy still targets
        if (threadIdx.x == 0) atomicAdd(&g_tma_timeouts, 1u);
        locate_points<STATS>(Q, Q.summary, ll, n, out, queue, leafq, qcount + part * COUNTER_STRIDE, part * part_cap,
                             mixed, inside);
        mbar_wait(&s_bar, 0);  // the copy in flight ends before the block does (bounded)
    }
    allow_dependents();
    if (STATS && ctr) count_inside(inside, ctr + 3);
}

// ----------------------------------------------------- a query, one launch --
//
// Queries that cannot fill the chip for long (INLINE_MAX) take a point from
// its coordinates to its label in one launch, without scratch and without
// counters to clear: a warp works on its own tiles of points, with queues of
// its own in shared memory between the steps, so a step runs when 32 points
// need it, on a full warp, and no step waits for other warps:
//   A  the tile's points: level-0 cell, then the coarse summary; a block of
//      cells without edges gives the label, the others are queued with their
//      cell and their place in it;
//   B  32 points in mixed blocks: node table, down to a pure node (the
//      label) or a leaf (queued);
//   C  32 points in leaves: tier 1; a label, or queued for tier 2 with the
//      mask of undecided edges (FP64-filter queries: queued as they are);
//   D  32 points: tier 2, then the complete test for what is left.
// Every step's loads are independent across the lanes.  Large queries run the
// passes as launches of their own (k_locate, k_leaf_t1, k_leaf_t2), where each
// has the registers it needs at the warps it can use; a small one paid for
// four launches, an allocation and a memset there (18 us a call).  Four blocks
// per SM (64 registers, 100 bytes spilled in tier 2) against two without:
// 1,048,576 points near the 1.1M-edge polygon's edges 102 us and 114, uniform
// ones 14 and 15.
template <int U>
struct WarpSpace {
    static constexpr int TILE = 32 * U;
    uint32_t p1[32 + TILE], c1[32 + TILE], u1[32 + TILE], v1[32 + TILE];  // B: points, cells, places in them
    uint32_t p2[64], w2[64];                                              // C: points, leaf words
    uint32_t p3[64], w3[64], m3[64];                                      // D: points, leaf words, masks
};

struct QueryCounts {
    int inside = 0, boundary = 0, fp64 = 0, exact = 0;
};

template <bool FP32, bool STATS, int U>
__device__ __forceinline__ void query_tiles(const QueryView& Q, const uint32_t* s_sum, int first, int stride, int n,
                                            const double2* __restrict__ ll, uint8_t* __restrict__ out,
                                            WarpSpace<U>& s, QueryCounts& c)
{
    const int lane = threadIdx.x & 31;
    const unsigned int below = (1u << lane) - 1u;
    int n1 = 0, n2 = 0, n3 = 0;  // queued points, the same in every lane
    for (int base = first;; base += stride) {
        const bool last = base >= n;
        if (!last) {  // A
            double2 pt[U];
#pragma unroll
            for (int k = 0; k < U; k++) {
                const int i = base + k * 32 + lane;
                pt[k] = i < n ? __ldg(ll + i) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int k = 0; k < U; k++) {
                const int i = base + k * 32 + lane;
                const bool have = i < n;
                uint8_t lab = (uint8_t)coarse_label(Q, s_sum, pt[k].x, pt[k].y);
                bool push = false;
                uint32_t cell = 0xFFFFFFFFu, fu = 0, fv = 0;  // unusual coordinates: not located
                if (lab == LABEL_PENDING) {
                    Loc L;
                    if (usual(pt[k].x, pt[k].y + 90.0)) {
                        push = domain_locate(Q, pt[k].x, pt[k].y + 90.0, L);
                        if (push) {
                            cell = (uint32_t)(L.iy * Q.W + L.ix);
                            fu = frac_bits(L.fu);
                            fv = frac_bits(L.fv);
                        } else {
                            lab = (uint8_t)Q.outside;
                        }
                    } else {
                        push = isfinite(pt[k].x) && isfinite(pt[k].y);  // non-finite input stays undefined
                    }
                }
                push = push && have;
                if (have && !push) {
                    out[i] = lab;
                    if (STATS) c.inside += lab == CELL_IN;
                }
                const unsigned int mk = __ballot_sync(0xffffffffu, push);
                if (push) {
                    const int at = n1 + __popc(mk & below);
                    s.p1[at] = (uint32_t)i;
                    s.c1[at] = cell;
                    s.u1[at] = fu;
                    s.v1[at] = fv;
                }
                n1 += __popc(mk);
            }
            __syncwarp();
        }
        for (;;) {
            const bool doB = n1 >= 32 || (last && n1 > 0);
            if (doB) {
                const int m = min(n1, 32);
                n1 -= m;
                uint32_t i = 0, w = KIND_PURE | 1u;
                if (lane < m) {
                    i = s.p1[n1 + lane];
                    const uint32_t cell = s.c1[n1 + lane];
                    w = LEAF_UNKNOWN;
                    if (cell != 0xFFFFFFFFu) {
                        w = descend_bits(Q, __ldg(Q.nodes + cell), s.u1[n1 + lane], s.v1[n1 + lane]);
                        if ((w & KIND_MASK) == KIND_PURE) {
                            const uint8_t lab = (uint8_t)(w & 3u);
                            out[i] = lab;
                            if (STATS) c.inside += lab == CELL_IN;
                        }
                    }
                }
                const bool leaf = (w & KIND_MASK) == KIND_LEAF || w == LEAF_UNKNOWN;
                const unsigned int mk = __ballot_sync(0xffffffffu, leaf);
                if (leaf) {
                    const int at = n2 + __popc(mk & below);
                    s.p2[at] = i;
                    s.w2[at] = w;
                }
                n2 += __popc(mk);
                __syncwarp();
            }
            const bool doC = n2 >= 32 || (last && n1 == 0 && n2 > 0);
            if (doC) {
                const int m = min(n2, 32);
                n2 -= m;
                bool defer = false;
                uint32_t i = 0, w = 0, mask = MASK_ALL;
                if (lane < m) {
                    i = s.p2[n2 + lane];
                    w = s.w2[n2 + lane];
                    if (FP32) {
                        LeafLoad L;
                        const bool known = (w & KIND_MASK) == KIND_LEAF;
                        if (known) L = load_leaf<false>(Q.leaves + (w & INDEX_MASK));
                        PointCtx P;
                        w = point_leaf(Q, __ldg(ll + i), P, w);
                        uint8_t lab = (uint8_t)(w & 3u);
                        if ((w & KIND_MASK) != KIND_PURE) {
                            if (STATS) c.boundary++;
                            if (!known) L = load_leaf<false>(Q.leaves + (w & INDEX_MASK));
                            lab = leaf_label_fp32<false>(Q.recs + L.off, L, P, mask);
                            defer = lab == LABEL_DEFER;
                            if (STATS) c.fp64 += defer;
                        }
                        if (!defer) {
                            out[i] = lab;
                            if (STATS) c.inside += lab == CELL_IN;
                        }
                    } else {
                        defer = true;
                    }
                }
                const unsigned int mk = __ballot_sync(0xffffffffu, defer);
                if (defer) {
                    const int at = n3 + __popc(mk & below);
                    s.p3[at] = i;
                    s.w3[at] = w;
                    if (FP32) s.m3[at] = mask;
                }
                n3 += __popc(mk);
                __syncwarp();
            }
            const bool doD = n3 >= 32 || (last && n1 == 0 && n2 == 0 && n3 > 0);
            if (doD) {
                const int m = min(n3, 32);
                n3 -= m;
                if (lane < m) {
                    const uint32_t i = s.p3[n3 + lane];
                    PointCtx P;
                    const uint32_t w = point_leaf(Q, __ldg(ll + i), P, s.w3[n3 + lane]);
                    uint8_t lab = (uint8_t)(w & 3u);
                    if ((w & KIND_MASK) != KIND_PURE) {
                        if (STATS && !FP32) c.boundary++;
                        double q[3];
                        gahhg_canon_vertex_xyz(P.lon, P.lat, q);
                        lab = leaf_label_fp64<false>(Q, w & INDEX_MASK, nullptr, q, FP32 ? s.m3[n3 + lane] : MASK_ALL);
                        if (lab == LABEL_DEFER) {
                            if (STATS) c.exact++;
                            lab = leaf_label_exact(&Q, w & INDEX_MASK, P.lon, P.lat);
                        }
                    }
                    out[i] = lab;
                    if (STATS) c.inside += lab == CELL_IN;
                }
                __syncwarp();
            }
            if (!(doB || doC || doD)) break;
        }
        if (last) break;
    }
}

__device__ __forceinline__ void count_stats(unsigned long long* ctr, const QueryCounts& c)
{
    count_inside(c.inside, ctr + 3);
    count_inside(c.boundary, ctr + 2);
    count_inside(c.fp64, ctr + 0);
    count_inside(c.exact, ctr + 1);
}

// STAGE: the coarse summary is copied to shared memory first (a query of a
// few thousand points reads the words it needs instead).
template <bool FP32, bool STATS, int U, bool STAGE>
__global__ void __launch_bounds__(TPB, U == 1 ? 2 : 4) k_query(const double2* __restrict__ ll, int n, uint8_t* __restrict__ out,
                                                 const __grid_constant__ QueryView Q, unsigned long long* ctr,
                                                 int poll_limit)
{
    extern __shared__ __align__(16) uint32_t s_sum[];
    constexpr int WARPS = TPB / 32, TILE = WarpSpace<U>::TILE;
    __shared__ WarpSpace<U> s_q[WARPS];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_late;
    bool late = false;
    if (STAGE) {
        if (threadIdx.x == 0) {
            s_late = 0;
            mbar_init(&s_bar);
            bulk_stage(s_sum, Q.summary, summary_bytes(Q.swords), &s_bar);
        }
        __syncthreads();
        if (!mbar_wait(&s_bar, 0, poll_limit)) s_late = 1;
        __syncthreads();
        late = s_late != 0;
        // after a wait that ran out the block reads the summary from global
        // memory and never touches s_sum, which the pending copy still targets
        if (late && threadIdx.x == 0) atomicAdd(&g_tma_timeouts, 1u);
    }
    QueryCounts c;
    const int warp = threadIdx.x >> 5;
    query_tiles<FP32, STATS, U>(Q, STAGE && !late ? s_sum : Q.summary, (blockIdx.x * WARPS + warp) * TILE,
                                gridDim.x * WARPS * TILE, n, ll, out, s_q[warp], c);
    if (STAGE && late) mbar_wait(&s_bar, 0);  // the copy in flight ends before the block does (bounded)
    if (STATS && ctr) count_stats(ctr, c);
}

// ------------------------------------------------------------- batches --

// A run of points of one view (points are stored segment after segment, and
// chunks are in point order, so chunk starts are increasing).
struct BatchChunk {
    int view;
    int count;
    long long start;
};

// Launch shapes of the batch locate: points a thread loads at a time and
// blocks per SM (all resident; the register budget per thread follows from the
// blocks).  Batches of other point mixes may prefer another row; the batch
// autotuner measures them.
struct BatchShape {
    int unroll, blocks;
};
constexpr BatchShape BATCH_SHAPES[] = {{5, 5}, {4, 4}, {6, 4}, {8, 3}};
constexpr int BATCH_NSHAPES = (int)(sizeof(BATCH_SHAPES) / sizeof(BATCH_SHAPES[0]));

// Pass 1 over the points of one chunk, by a block whose warps take tiles of
// 32 * U points: as locate_points, the points in mixed blocks wait in the
// warp's queue; B_DESCENTS per lane descend in lockstep (1, 2 and 3 per lane:
// 89, 79 and 80 us for the 6 x 4 shape on 28M points in 160 polygons, the
// others within 3 us).  Descending every point where it stood, five to a
// thread, the same points took 228 us in the same chunks as 150 now.
constexpr int B_DESCENTS = 2;
template <bool STATS, int U>
__device__ __forceinline__ void locate_chunk(const QueryView& Q, const uint32_t* sum, const double2* __restrict__ ll,
                                             int n, uint8_t* __restrict__ out, uint32_t first,
                                             uint32_t* __restrict__ queue, uint32_t* __restrict__ leafq,
                                             unsigned int* qcount, uint32_t* mixed, int& inside)
{
    const int lane = threadIdx.x & 31;
    int nm = 0;
    for (int base = (threadIdx.x >> 5) * 32 * U;; base += TPB * U) {
        const bool last = base >= n;
        if (!last) {
            double2 p[U];
#pragma unroll
            for (int k = 0; k < U; k++) {
                const int i = base + 32 * k + lane;
                p[k] = i < n ? __ldg(ll + i) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int k = 0; k < U; k++) {
                const int i = base + 32 * k + lane;
                const uint32_t l = coarse_label(Q, sum, p[k].x, p[k].y);
                if (i < n) out[i] = (uint8_t)l;
                if (STATS) inside += (l == CELL_IN) & (i < n);
                const bool push = l == 0 && i < n;
                const unsigned int mk = __ballot_sync(0xffffffffu, push);
                if (push) mixed[nm + __popc(mk & ((1u << lane) - 1u))] = (uint32_t)i;
                nm += __popc(mk);
            }
            __syncwarp();
        }
        while (nm >= 32 * B_DESCENTS || (last && nm > 0)) {
            const int m = min(nm, 32 * B_DESCENTS);
            nm -= m;
            uint32_t i[B_DESCENTS], w[B_DESCENTS], fu[B_DESCENTS], fv[B_DESCENTS];
#pragma unroll
            for (int d = 0; d < B_DESCENTS; d++) {
                w[d] = KIND_PURE | 4u;  // no point, or non-finite input, which stays undefined (LABEL_PENDING)
                i[d] = fu[d] = fv[d] = 0;
                if (lane + 32 * d < m) {
                    i[d] = mixed[nm + lane + 32 * d];
                    const double2 p = __ldg(ll + i[d]);
                    const double laf = p.y + 90.0;
                    Loc L;
                    if (usual(p.x, laf)) {
                        w[d] = Q.outside;
                        if (domain_locate(Q, p.x, laf, L)) {
                            w[d] = __ldg(Q.nodes + (size_t)L.iy * Q.W + L.ix);
                            fu[d] = frac_bits(L.fu);
                            fv[d] = frac_bits(L.fv);
                        }
                    } else if (isfinite(p.x) && isfinite(p.y)) {
                        w[d] = LEAF_UNKNOWN;  // unusual coordinates: tier 1 locates them
                    }
                }
            }
            bool inner = true;
            while (inner) {
                inner = false;
#pragma unroll
                for (int d = 0; d < B_DESCENTS; d++)
                    if ((w[d] & KIND_MASK) == KIND_INNER) {
                        w[d] = __ldg(Q.nodes + (w[d] & INDEX_MASK) + (fv[d] >> 30) * FAN + (fu[d] >> 30));
                        fu[d] <<= 2;
                        fv[d] <<= 2;
                        inner = true;
                    }
            }
            unsigned int mk[B_DESCENTS], total = 0;
#pragma unroll
            for (int d = 0; d < B_DESCENTS; d++) {
                const bool pure = (w[d] & KIND_MASK) == KIND_PURE;
                if (pure && (w[d] & 3u)) {
                    out[i[d]] = (uint8_t)(w[d] & 3u);
                    if (STATS) inside += (w[d] & 3u) == CELL_IN;
                }
                mk[d] = __ballot_sync(0xffffffffu, !pure || w[d] == LEAF_UNKNOWN);
                total += __popc(mk[d]);
            }
            if (total) {
                unsigned int pos = 0;
                if (lane == 0) pos = atomicAdd(qcount, total);
                pos = __shfl_sync(0xffffffffu, pos, 0) + first;
#pragma unroll
                for (int d = 0; d < B_DESCENTS; d++) {
                    if (mk[d] >> lane & 1u) {
                        const unsigned int at = pos + __popc(mk[d] & ((1u << lane) - 1u));
                        queue[at] = first + i[d];
                        leafq[at] = w[d];
                    }
                    pos += __popc(mk[d]);
                }
            }
            __syncwarp();
        }
        if (last) break;
    }
}

// Prefix sums of the chunks' queue counts, by one block of THREADS threads:
// pre[c] entries come before chunk c's, pre[nchunks] in all.  And zeros in tier
// 2's counters, which nothing has touched yet.
constexpr int CS_ITEMS = 8;
template <int THREADS>
__device__ __forceinline__ void chunk_prefix(const unsigned int* ccount, int nchunks, unsigned int* pre,
                                             unsigned int* t2cnt)
{
    constexpr int WARPS = THREADS / 32;
    __shared__ unsigned int s_w[WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < QUEUE_PARTS) t2cnt[threadIdx.x * COUNTER_STRIDE] = 0;
    unsigned int before = 0;
    for (int base = 0; base < nchunks; base += THREADS * CS_ITEMS) {
        const int b0 = base + threadIdx.x * CS_ITEMS;
        unsigned int c[CS_ITEMS], run = 0;
#pragma unroll
        for (int k = 0; k < CS_ITEMS; k++) {
            c[k] = b0 + k < nchunks ? __ldcg(ccount + b0 + k) : 0u;
            run += c[k];
        }
        unsigned int x = run;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_w[warp] = x;
        __syncthreads();
        if (warp == 0) {
            unsigned int z = lane < WARPS ? s_w[lane] : 0u;
            for (int o = 1; o < WARPS; o <<= 1) {
                const unsigned int y = __shfl_up_sync(0xffffffffu, z, o);
                if (lane >= o) z += y;
            }
            if (lane < WARPS) s_w[lane] = z;
        }
        __syncthreads();
        unsigned int at = before + (warp ? s_w[warp - 1] : 0u) + x - run;
#pragma unroll
        for (int k = 0; k < CS_ITEMS; k++) {
            if (b0 + k < nchunks) pre[b0 + k] = at;
            at += c[k];
        }
        before += s_w[WARPS - 1];
        __syncthreads();  // s_w is rewritten
    }
    if (threadIdx.x == 0) pre[nchunks] = before;
}

// Pass 1 over a batch: a persistent grid takes chunks in order from an atomic
// counter (polygons of very different sizes balance themselves; the next
// chunk's number is on its way while a chunk is worked on), copies the chunk's
// view and polygon summary to shared memory and runs the tile loop on it.  A
// chunk's points in leaves are queued from the chunk's own first place,
// counted in shared memory: no global atomic (see QUEUE_PARTS).  With `pre` the
// block that ends last makes the prefix sums of those counts (see SCAN_FOLD).
template <bool STATS, int UNROLL, int BLOCKS>
__global__ void __launch_bounds__(TPB, BLOCKS) k_batch_locate(const QueryView* __restrict__ views,
                                                     const BatchChunk* __restrict__ chunks, int nchunks,
                                                     unsigned int* next_chunk, const double2* __restrict__ ll,
                                                     uint8_t* __restrict__ out, uint32_t* __restrict__ queue,
                                                     uint32_t* __restrict__ leafq, unsigned int* ccount,
                                                     unsigned int* pre, unsigned int* t2cnt, unsigned int* ended,
                                                     unsigned long long* ctr, int poll_limit)
{
    __shared__ __align__(16) uint32_t s_sum[SUMMARY_WORDS_MAX];  // receives the bulk copies
    __shared__ __align__(16) uint32_t s_view[sizeof(QueryView) / 4];
    __shared__ uint32_t s_mixed[TPB / 32][32 * (B_DESCENTS + UNROLL)];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_chunk, s_late, s_last;
    __shared__ unsigned int s_queued;
    static_assert(sizeof(QueryView) % 4 == 0 && sizeof(QueryView) / 4 <= TPB, "a word of the view per thread");
    if (threadIdx.x == 0) {
        s_late = 0;
        mbar_init(&s_bar);
        s_chunk = (int)atomicAdd(next_chunk, 1u);
        s_queued = 0;
    }
    uint32_t phase = 0;
    bool late = false;  // the same in every thread: read from s_late after a barrier
    int inside = 0;
    __syncthreads();
    for (;;) {
        const int ci = s_chunk;
        if (ci >= nchunks) break;
        const BatchChunk c = chunks[ci];
        if (threadIdx.x < sizeof(QueryView) / 4) s_view[threadIdx.x] = __ldg((const uint32_t*)(views + c.view) + threadIdx.x);
        __syncthreads();
        const QueryView& Q = *(const QueryView*)s_view;
        unsigned int next = 0;
        if (threadIdx.x == 0) {
            if (!late) bulk_stage(s_sum, Q.summary, summary_bytes(Q.swords), &s_bar);
            next = atomicAdd(next_chunk, 1u);
        }
        if (!late) {
            if (!mbar_wait(&s_bar, phase, poll_limit)) s_late = 1;  // any thread's timeout switches the block
            phase ^= 1u;
            __syncthreads();
            late = s_late != 0;
        }
        uint32_t* mixed = s_mixed[threadIdx.x >> 5];
        // after a wait that ran out the block reads the summaries from global
        // memory and never touches s_sum, which the pending copy still targets
        if (!late)
            locate_chunk<STATS, UNROLL>(Q, s_sum, ll + c.start, c.count, out + c.start, (uint32_t)c.start, queue, leafq,
                                        &s_queued, mixed, inside);
        else
            locate_chunk<STATS, UNROLL>(Q, Q.summary, ll + c.start, c.count, out + c.start, (uint32_t)c.start, queue,
                                        leafq, &s_queued, mixed, inside);
        __syncthreads();
        if (threadIdx.x == 0) {
            ccount[ci] = s_queued;
            s_queued = 0;
            s_chunk = (int)next;
        }
        __syncthreads();
    }
    if (late) {
        if (threadIdx.x == 0) atomicAdd(&g_tma_timeouts, 1u);
        mbar_wait(&s_bar, phase ^ 1u);  // the copy in flight ends before the block does (bounded)
    }
    if (pre) {
        if (threadIdx.x == 0) {
            __threadfence();  // this block's counts (thread 0 wrote them) come before its end
            s_last = atomicAdd(ended, 1u) == gridDim.x - 1;
            __threadfence();
        }
        __syncthreads();
        if (s_last) chunk_prefix<TPB>(ccount, nchunks, pre, t2cnt);
    }
    allow_dependents();
    if (STATS && ctr) count_inside(inside, ctr + 3);
}

// The same by a launch of its own, and the tier 2 counters.
constexpr int CS_TPB = 1024;
__global__ void __launch_bounds__(CS_TPB) k_chunk_scan(const unsigned int* __restrict__ ccount, int nchunks,
                                                      unsigned int* __restrict__ pre, unsigned int* __restrict__ t2cnt)
{
    wait_for_predecessor();
    chunk_prefix<CS_TPB>(ccount, nchunks, pre, t2cnt);
    allow_dependents();
}

// --------------------------------------------- the tiers as launches of their own --

// A queue in parts: place p * cap + k holds entry k of part p, counted on
// cnt[p * COUNTER_STRIDE] (which keeps counting past cap).
struct PartQueue {
    unsigned int* cnt = nullptr;
    int parts = 1;
    unsigned int cap = 0;
};

struct Tiers {
    // pass 1's queue: points in leaves and their leaf words, in parts (one
    // polygon), or from each chunk's first place (batches: chunks, pre)
    const uint32_t* q1;
    const uint32_t* l1;
    PartQueue p1;
    const BatchChunk* chunks = nullptr;
    const unsigned int* pre = nullptr;
    int nchunks = 0;
    // that queue in window or leaf order, used when *sorted == 1
    const uint32_t* spts = nullptr;
    const uint32_t* sleaf = nullptr;
    const unsigned int* sorted = nullptr;
    int sstride = 1;  // words from one ordered entry to the next (2: leaf order's interleaved pairs)
    // tier 2's queue behind tier 1: points, leaf words, masks of undecided records
    uint32_t* q2 = nullptr;
    uint32_t* l2 = nullptr;
    uint32_t* m2 = nullptr;
    PartQueue p2;
    unsigned int* over = nullptr;  // raised when a part of it is full
};

// The entries of a part queue in one sequence, part after part, for a warp:
// lanes hold the parts' prefix sums.
struct PartEntries {
    unsigned int pa, pb, total, cap;  // entries before part `lane` and part `lane + 32`

    __device__ __forceinline__ void begin(const PartQueue& P)
    {
        static_assert(QUEUE_PARTS <= 64, "two parts per lane");
        const int lane = threadIdx.x & 31;
        cap = P.cap;
        const unsigned int a = lane < P.parts ? min(P.cnt[lane * COUNTER_STRIDE], cap) : 0u;
        const unsigned int b = lane + 32 < P.parts ? min(P.cnt[(lane + 32) * COUNTER_STRIDE], cap) : 0u;
        unsigned int x = a, y = b;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int u = __shfl_up_sync(0xffffffffu, x, o), v = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) {
                x += u;
                y += v;
            }
        }
        const unsigned int ta = __shfl_sync(0xffffffffu, x, 31);
        pa = x - a;
        pb = ta + y - b;
        total = ta + __shfl_sync(0xffffffffu, y, 31);
    }
    __device__ __forceinline__ unsigned int before(int p) const  // p the same in every lane
    {
        const unsigned int x = __shfl_sync(0xffffffffu, p < 32 ? pa : pb, p & 31);
        return p < 64 ? x : total;
    }
    // the place of entry t = t0 + lane (t0 < total); every lane calls
    __device__ __forceinline__ unsigned int place(unsigned int t0) const
    {
        const unsigned int t = t0 + (threadIdx.x & 31);
        int p = __popc(__ballot_sync(0xffffffffu, pa <= t0)) + __popc(__ballot_sync(0xffffffffu, pb <= t0)) - 1;
        unsigned int lo = before(p), hi = before(p + 1), at = 0;
        for (;;) {
            if (t >= lo) at = (unsigned int)p * cap + (t - lo);
            if (hi >= total || !__any_sync(0xffffffffu, t >= hi)) return at;
            p++;
            lo = hi;
            hi = before(p + 1);
        }
    }
};

// Where a queued point's index view comes from: one polygon...
struct OneView {
    QueryView Q;
    struct Source {
        PartEntries E;
        bool ordered;
    };
    __device__ __forceinline__ const QueryView& of(uint32_t) const { return Q; }
    __device__ __forceinline__ const QueryView& view(int) const { return Q; }
    __device__ __forceinline__ unsigned int begin(const Tiers& T, Source& S) const
    {
        S.ordered = T.sorted && *(const volatile unsigned int*)T.sorted == 1u;
        S.E.begin(T.p1);
        return S.E.total;
    }
    // entry t0 + lane of pass 1's queue: point and leaf word; every lane calls
    __device__ __forceinline__ void fetch(const Tiers& T, const Source& S, unsigned int t0, uint32_t& i, uint32_t& w,
                                          int&) const
    {
        const unsigned int t = t0 + (threadIdx.x & 31);
        const unsigned int at = S.ordered ? t * T.sstride : S.E.place(t0);
        if (t >= S.E.total) return;
        i = S.ordered ? T.spts[at] : T.q1[at];
        w = S.ordered ? T.sleaf[at] : T.l1[at];
    }
};

// The last p with pre[p] <= t, p in [0, n).
__device__ __forceinline__ int last_before(const unsigned int* __restrict__ pre, int n, unsigned int t)
{
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(pre + mid) <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}

// ...or its chunk's.
struct ChunkViews {
    const QueryView* views;
    const BatchChunk* chunks;
    int nchunks;
    struct Source {
        unsigned int total;
    };
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
    __device__ __forceinline__ const QueryView& view(int v) const { return views[v]; }
    __device__ __forceinline__ unsigned int begin(const Tiers& T, Source& S) const
    {
        S.total = T.pre[nchunks];
        return S.total;
    }
    __device__ __forceinline__ void fetch(const Tiers& T, const Source& S, unsigned int t0, uint32_t& i, uint32_t& w,
                                          int& v) const
    {
        const unsigned int t = t0 + (threadIdx.x & 31);
        if (t >= S.total) return;
        const int c = last_before(T.pre, nchunks, t);
        const unsigned int at = (unsigned int)__ldg(&chunks[c].start) + (t - __ldg(T.pre + c));
        v = __ldg(&chunks[c].view);
        i = T.q1[at];
        w = T.l1[at];
    }
};

// A warp's deferred points to tier 2's queue, one atomic on its part's
// counter; a point that finds the part full is marked, and the tier 2 launch
// finishes it from pass 1's queue (pass 1 wrote LABEL_PENDING for every queued
// point, so a mark is never something else's).
constexpr uint8_t LABEL_OVER = 0xFE;
__device__ __forceinline__ void push_deferred(bool defer, uint32_t i, uint32_t w, uint32_t mask, const Tiers& T,
                                              uint8_t* out)
{
    const unsigned int bal = __ballot_sync(0xffffffffu, defer);
    if (!bal) return;
    const int lane = threadIdx.x & 31;
    const unsigned int part = blockIdx.x % (unsigned int)T.p2.parts;
    unsigned int pos = 0;
    if (lane == 0) pos = atomicAdd(T.p2.cnt + part * COUNTER_STRIDE, (unsigned int)__popc(bal));
    pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(bal & ((1u << lane) - 1u));
    if (!defer) return;
    if (pos < T.p2.cap) {
        const unsigned int at = part * T.p2.cap + pos;
        T.q2[at] = i;
        T.l2[at] = w;
        T.m2[at] = mask;
    } else {
        out[i] = LABEL_OVER;
        *T.over = 1u;
    }
}

// Tier 1 over the pass-1 queue, perhaps ordered.  A warp takes 32 entries at a
// time, the next 32 entries' points and leaf words loaded ahead, and meets no
// other warp (the block's rounds used to end in three barriers around one
// atomic; with the counter in parts a warp's own atomic costs nothing).  Four
// blocks per SM: 64 registers, no spills, 251 us for the 9.1M points in leaves
// of 2e7 near-edge points (five blocks, 48 registers: 315).  Half of the issue
// slots and three quarters of the L1's tag lookups are taken (a lane loads its
// own 64-byte leaf).  Copying the leaves to shared memory by the warp together
// took 231 here but 36 us where a batch's tier 1 takes 30.
constexpr int T1_BLOCKS = 4;
template <class VS>
__global__ void __launch_bounds__(TPB, T1_BLOCKS) k_leaf_t1(const __grid_constant__ VS vs,
                                                         const double2* __restrict__ ll, uint8_t* __restrict__ out,
                                                         const __grid_constant__ Tiers T, unsigned long long* ctr)
{
    wait_for_predecessor();
    typename VS::Source S;
    const unsigned int m = vs.begin(T, S);
    QueryCounts c;
    const unsigned int step = gridDim.x * blockDim.x, lane = threadIdx.x & 31;
    unsigned int t0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
    uint32_t ni = 0, nw = 0;
    int nv = 0;
    if (t0 < m) vs.fetch(T, S, t0, ni, nw, nv);
    for (; t0 < m; t0 += step) {
        const uint32_t i = ni, known = nw;
        const QueryView& Q = vs.view(nv);
        const bool mine = t0 + lane < m;
        bool defer = false;
        uint32_t w = 0, mask = 0;
        PointCtx P{0.0, 0.0};
        LeafLoad L;
        double2 p = make_double2(0.0, 0.0);
        const bool in_leaf = (known & KIND_MASK) == KIND_LEAF;
        if (mine) {
            p = ll[i];
            if (in_leaf) L = load_leaf<false>(Q.leaves + (known & INDEX_MASK));
        }
        if (t0 + step < m) vs.fetch(T, S, t0 + step, ni, nw, nv);
        if (mine) {
            w = point_leaf(Q, p, P, known);
            uint8_t lab = (uint8_t)(w & 3u);
            if ((w & KIND_MASK) != KIND_PURE) {
                c.boundary++;
                if (!in_leaf) L = load_leaf<false>(Q.leaves + (w & INDEX_MASK));
                lab = leaf_label_fp32<false>(Q.recs + L.off, L, P, mask);
            }
            defer = lab == LABEL_DEFER;
            if (defer) {
                c.fp64++;
            } else {
                out[i] = lab;
                c.inside += lab == CELL_IN;
            }
        }
        push_deferred(defer, i, w, mask, T, out);
    }
    allow_dependents();
    if (ctr) count_stats(ctr, c);
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
// 256-byte aligned; leaf records are 64 bytes, edge records 16) and their
// sizes are multiples of 16 bytes.  2e7 points, half of them near the
// 1.1M-edge polygon's edges: 946 us a query, 896 with k_leaf_t1 on the same
// leaf-ordered queue, whose per-warp gathers leaf order already makes one
// request per warp and leaf; the staging adds a block barrier and a wait per
// tile and copies every leaf of the tile's range.  It is therefore an option
// (pass-2 order 3).
constexpr int T1S_LEAVES = 256;  // 16 KB of leaf records per tile
constexpr int T1S_RECS = 1024;   // 16 KB of edge records per tile
constexpr int T1S_BLOCKS = 5;

__global__ void __launch_bounds__(TPB, T1S_BLOCKS) k_leaf_t1s(const __grid_constant__ QueryView Q, const double2* __restrict__ ll,
                                                            uint8_t* __restrict__ out,
                                                            const __grid_constant__ Tiers T,
                                                            unsigned long long* ctr, int polls)
{
    __shared__ __align__(16) LeafRec s_leaf[T1S_LEAVES];
    __shared__ __align__(16) float4 s_rec[T1S_RECS];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ uint32_t s_l0, s_r0, s_nr;  // first staged leaf, first staged record, records staged
    __shared__ int s_nl;                   // leaves staged for the tile (0: none)
    __shared__ int s_broken;               // a wait ran out: no more staging
    if (threadIdx.x == 0) {
        mbar_init(&s_bar);
        s_broken = 0;
    }
    __syncthreads();
    wait_for_predecessor();
    PartEntries E;
    E.begin(T.p1);
    const unsigned int m = E.total;
    const bool sorted = *(const volatile unsigned int*)T.sorted == 1u;
    const uint32_t* src = sorted ? T.spts : T.q1;
    const uint32_t* src_leaf = sorted ? T.sleaf : T.l1;
    const unsigned int st = (unsigned int)T.sstride;  // (sorted: entries are at t * st)
    QueryCounts c;
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
        PointCtx P{0.0, 0.0};
        unsigned int at = t * st;
        if (!sorted && (t & ~31u) < m) at = E.place(t & ~31u);
        if (t < m) {
            i = src[at];
            w = point_leaf(Q, ll[i], P, src_leaf[at]);
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
            uint8_t lab = (uint8_t)(w & 3u);
            if ((w & KIND_MASK) != KIND_PURE) {
                c.boundary++;
                const uint32_t li = (w & INDEX_MASK) - s_l0;  // wraps above nl below the first leaf
                bool done = false;
                if (staged && li < (uint32_t)nl) {
                    const LeafLoad L = load_leaf<true>(s_leaf + li);
                    const uint32_t ro = L.off - s_r0;
                    if (ro <= s_nr && (uint32_t)L.cnt() <= s_nr - ro) {
                        lab = leaf_label_fp32<true>(s_rec + ro, L, P, mask);
                        done = true;
                    }
                }
                if (!done) {
                    const LeafLoad L = load_leaf<false>(Q.leaves + (w & INDEX_MASK));
                    lab = leaf_label_fp32<false>(Q.recs + L.off, L, P, mask);
                }
            }
            defer = lab == LABEL_DEFER;
            if (defer) {
                c.fp64++;
            } else {
                out[i] = lab;
                c.inside += lab == CELL_IN;
            }
        }
        if (threadIdx.x == 0 && sorted && b0 + bstep < m) tile_bounds();  // the next tile's, ahead of its start
        push_deferred(defer, i, w, mask, T, out);
        __syncthreads();  // the staged slices are rewritten next round
    }
    allow_dependents();
    if (threadIdx.x == 0 && s_broken) {
        atomicAdd(&g_tma_timeouts, 1u);
        mbar_wait(&s_bar, phase ^ 1u);  // the copy whose wait ran out
    }
    if (ctr) count_stats(ctr, c);
}

// Tier 2's shape: blocks of 128 threads; the warps hide the chain entry ->
// point and aux line -> edge ends.  (us, blocks per SM 5 / 6 / 7 / 8, 2e7
// points, half of them near the 1.1M-edge polygon's edges: all points of an
// FP64-filter query 606 / 571 / 532 / 518, tier 1's deferred points 260 / 240
// / 227 / 239.  A lane loading its own line: 614 and 233 at their best.)
constexpr int T2_TPB = 128;
constexpr int T2_ALL_BLOCKS = 8, T2_BLOCKS = 7;

// Tier 2, then the complete test for what it leaves, over the queue of
// deferred points; ALL: FP64-filter queries, over pass 1's queue.  The next
// entry is loaded ahead, as in tier 1.
template <class VS, bool ALL>
__global__ void __launch_bounds__(T2_TPB, ALL ? T2_ALL_BLOCKS : T2_BLOCKS) k_leaf_t2(const __grid_constant__ VS vs,
                                                              const double2* __restrict__ ll,
                                                              uint8_t* __restrict__ out,
                                                              const __grid_constant__ Tiers T,
                                                              unsigned long long* ctr)
{
    __shared__ __align__(16) uint4 s_lines[T2_TPB / 32][8 * 32];
    uint4* s_aux = s_lines[threadIdx.x >> 5];
    wait_for_predecessor();
    typename VS::Source S;
    PartEntries E;
    unsigned int m;
    if (ALL) {
        m = vs.begin(T, S);
    } else {
        E.begin(T.p2);
        m = E.total;
    }
    QueryCounts c;
    const unsigned int step = gridDim.x * blockDim.x, lane = threadIdx.x & 31;
    unsigned int t0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
    uint32_t ni = 0, nw = 0, nm = MASK_ALL;
    int nv = 0;
    auto fetch = [&](unsigned int at0) {
        if (ALL) {
            vs.fetch(T, S, at0, ni, nw, nv);
        } else {
            const unsigned int at = E.place(at0);
            if (at0 + lane < m) {
                ni = T.q2[at];
                nw = T.l2[at];
                nm = T.m2[at];
            }
        }
    };
    if (t0 < m) fetch(t0);
    for (; t0 < m; t0 += step) {
        const uint32_t i = ni, known = nw, mask = nm;
        const int v = nv;
        const bool mine = t0 + lane < m;
        double2 p = make_double2(0.0, 0.0);
        if (mine) p = ll[i];
        const QueryView& Q = ALL ? vs.view(v) : vs.of(mine ? i : 0);
        copy_aux(s_aux, mine && (known & KIND_MASK) == KIND_LEAF ? Q.aux + (known & INDEX_MASK) : nullptr);
        if (t0 + step < m) fetch(t0 + step);
        PointCtx P{0.0, 0.0};
        uint32_t w = KIND_PURE;
        double q[3];
        if (mine) {
            w = point_leaf(Q, p, P, known);
            gahhg_canon_vertex_xyz(P.lon, P.lat, q);
            if (known == LEAF_UNKNOWN && (w & KIND_MASK) == KIND_LEAF)
                for (int k = 0; k < 8; k++) s_aux[aux_slot(lane, k)] = __ldg((const uint4*)(Q.aux + (w & INDEX_MASK)) + k);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        if (mine) {
            uint8_t lab = (uint8_t)(w & 3u);
            if ((w & KIND_MASK) != KIND_PURE) {
                if (ALL) c.boundary++;
                lab = leaf_label_fp64<true>(Q, w & INDEX_MASK, s_aux, q, mask);
                if (lab == LABEL_DEFER) {
                    c.exact++;
                    lab = leaf_label_exact(&Q, w & INDEX_MASK, P.lon, P.lat);
                }
            }
            out[i] = lab;
            c.inside += lab == CELL_IN;
        }
        __syncwarp();  // the lines are rewritten in the next round
    }
    if (!ALL && *(const volatile unsigned int*)T.over) {
        // points that found their part of tier 2's queue full
        const unsigned int n = vs.begin(T, S);
        for (t0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); t0 < n; t0 += step) {
            vs.fetch(T, S, t0, ni, nw, nv);
            if (t0 + lane >= n || out[ni] != LABEL_OVER) continue;
            const QueryView& Q = vs.view(nv);
            PointCtx P;
            const uint32_t w = point_leaf(Q, ll[ni], P, nw);
            c.exact++;
            const uint8_t lab = leaf_label_exact(&Q, w & INDEX_MASK, P.lon, P.lat);
            out[ni] = lab;
            c.inside += lab == CELL_IN;
        }
    }
    allow_dependents();
    if (ctr) count_stats(ctr, c);
}

// ------------------------------------- pass-2 queue in leaf-window order --
//
// Pass 1 queues points in input order, so on inputs without spatial order
// (C2's near-edge points) the tiers' gathers of leaf and edge records sweep
// the whole index, which is larger than L2 (198 MB on the C1 polygon): over
// half of the records come from DRAM.  Leaves are numbered
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
// PART_BYTES of leaf and edge records; queues below PART_MIN_QUEUE entries
// keep pass-1 order (both kernels return at once and the tiers read the pass-1
// queue).  2e7 points, half of them near the 1.1M-edge polygon's edges, FP32
// filter: 822 us where pass-1 order takes 666, leaf order (below) 896.
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

__global__ void __launch_bounds__(P_TPB) k_part_count(const uint32_t* __restrict__ l1, PartQueue Q, PartScratch S)
{
    __shared__ unsigned int s_cnt[PART_MAX];
    wait_for_predecessor();
    PartEntries E;
    E.begin(Q);
    const unsigned int m = E.total, lane = threadIdx.x & 31;
    if (m < PART_MIN_QUEUE) {
        allow_dependents();
        return;
    }
    for (int k = threadIdx.x; k < S.np; k += P_TPB) s_cnt[k] = 0;
    __syncthreads();
    for (unsigned int t0 = blockIdx.x * P_TPB + (threadIdx.x & ~31u); t0 < m; t0 += gridDim.x * P_TPB) {
        const unsigned int at = E.place(t0);
        if (t0 + lane < m) smem_rank(s_cnt, part_of(l1[at], S.np, S.scale));
        __syncwarp();
    }
    __syncthreads();
    allow_dependents();
    for (int k = threadIdx.x; k < S.np; k += P_TPB)
        if (s_cnt[k]) atomicAdd(S.total + k, s_cnt[k]);
}

__global__ void __launch_bounds__(P_TPB) k_part_scatter(const uint32_t* __restrict__ queue,
                                                        const uint32_t* __restrict__ l1, PartQueue Q, PartScratch S)
{
    __shared__ unsigned int s_start[PART_MAX], s_cnt[PART_MAX], s_base[PART_MAX];
    wait_for_predecessor();
    PartEntries E;
    E.begin(Q);
    const unsigned int m = E.total;
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
            const unsigned int t = base + k * P_TPB + threadIdx.x, t0 = t & ~31u;
            const unsigned int at = t0 < m ? E.place(t0) : 0u;
            q[k] = t < m ? queue[at] : 0u;
            w[k] = t < m ? l1[at] : 0u;
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
};

__device__ __forceinline__ int leaf_bucket(uint32_t w, int nb)
{
    return (w & KIND_MASK) == KIND_LEAF ? (int)min(w & INDEX_MASK, (uint32_t)(nb - 1)) : nb - 1;
}

__global__ void __launch_bounds__(LS_TPB) k_ls_count(const uint32_t* __restrict__ l1, PartQueue Q, LeafSortScratch S)
{
    wait_for_predecessor();
    PartEntries E;
    E.begin(Q);
    const unsigned int m = E.total;
    if (m >= PART_MIN_QUEUE)
        for (unsigned int t0 = blockIdx.x * LS_TPB + (threadIdx.x & ~31u); t0 < m; t0 += gridDim.x * LS_TPB) {
            const unsigned int at = E.place(t0), t = t0 + (threadIdx.x & 31);
            if (t < m) S.rank[t] = atomicAdd(S.cnt + leaf_bucket(l1[at], S.nb), 1u);
        }
    allow_dependents();
}

__device__ __forceinline__ bool long_queue(const PartQueue& Q)
{
    PartEntries E;
    E.begin(Q);
    return E.total >= PART_MIN_QUEUE;
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

__global__ void __launch_bounds__(LS_TPB) k_ls_tile_sums(PartQueue Q, LeafSortScratch S)
{
    __shared__ unsigned int s_w[LS_TPB / 32];
    wait_for_predecessor();
    if (long_queue(Q)) {
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

__global__ void __launch_bounds__(LS_TPB) k_ls_scan(PartQueue Q, LeafSortScratch S)
{
    __shared__ unsigned int s_w[LS_TPB / 32];
    __shared__ unsigned int s_wx[LS_TPB / 32];
    wait_for_predecessor();
    if (long_queue(Q)) {
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
                                                       const uint32_t* __restrict__ l1, PartQueue Q, LeafSortScratch S)
{
    wait_for_predecessor();
    PartEntries E;
    E.begin(Q);
    const unsigned int m = E.total;
    if (m >= PART_MIN_QUEUE) {
        for (unsigned int t0 = blockIdx.x * LS_TPB + (threadIdx.x & ~31u); t0 < m; t0 += gridDim.x * LS_TPB) {
            const unsigned int from = E.place(t0), t = t0 + (threadIdx.x & 31);
            if (t < m) {
                const uint32_t w = l1[from];
                const unsigned int at = S.start[leaf_bucket(w, S.nb)] + S.rank[t];
                if (at < m) {  // counts and entries agree; never write past the queue
                    S.sent[at] = make_uint2(queue[from], w);
                }
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

// Tier 2's queue for `points` points: half of them (near-edge points defer 41 %
// of those in leaves), in equal parts with room for the blocks of tier 1
// being unequal; what finds its part full the tier 2 launch finishes.
PartQueue tier2_parts(long long points, unsigned int* cnt)
{
    return PartQueue{cnt, QUEUE_PARTS, (unsigned int)(points / 2 / QUEUE_PARTS + 1024)};
}

// A tier's blocks: what the chip holds, or a thread for each of `points`.
int tier_grid(int resident, long long points, int tpb)
{
    return (int)std::min<long long>(resident, std::max(1LL, (points + tpb - 1) / tpb));
}

template <class VS>
void tier2_launch(const VS& vs, const double2* ll, uint8_t* out, const Tiers& T, int precision, long long points,
                  unsigned long long* ctr, int sms, cudaStream_t s)
{
    if (precision == GAHHG_QUERY_FP64_FILTER)
        launch_dependent_tpb(k_leaf_t2<VS, true>, tier_grid(sms * T2_ALL_BLOCKS, points, T2_TPB), T2_TPB, s, vs, ll, out,
                             T, ctr);
    else
        launch_dependent_tpb(k_leaf_t2<VS, false>, tier_grid(sms * T2_BLOCKS, points, T2_TPB), T2_TPB, s, vs, ll, out, T,
                             ctr);
}

}  // namespace

// ------------------------------------------------------------------ host --

static const QueryView& make_view(const Grid* g) { return g->lattice->views[0]; }

// Windows of about PART_BYTES of the records the tiers gather per leaf, three
// doubles of a leaf's aux line counted (the whole line: more windows, 855 us
// where 825 were taken by 2e7 points near the 1.1M-edge polygon).
void set_leaf_windows(QueryView& Q, long long nleaves, long long nrecs)
{
    const long long tier_bytes = nrecs * (long long)(sizeof(float4) + sizeof(uint32_t)) +
                                 nleaves * (long long)(sizeof(LeafRec) + 3 * sizeof(double));
    Q.nparts = (int)std::min<long long>(PART_MAX, std::max<long long>(1, (tier_bytes + PART_BYTES - 1) / PART_BYTES));
    if (nleaves < 2 * PART_MAX) Q.nparts = 1;
    Q.part_scale = Q.nparts > 1 ? (float)((double)Q.nparts / (double)nleaves) : 0.0f;
}

// Points per pass.
constexpr long long QUERY_CHUNK = 1LL << 27;
// Queries of at most this many points run as one launch with every tier
// inline (k_query).  us a call, one launch | passes of their own (FP32 filter;
// uniform points, and half of them near an edge in random order):
//              1.1M-edge polygon      100,000 edges          1,100 edges
//   points     uniform     near      uniform     near      uniform     near
//     32,000    6 | 16    10 | 23     6 | 16    10 | 23     6 | 15     9 | 22
//    131,072    8 | 20    16 | 27     8 | 18    17 | 27     8 | 16    27 | 35
//    524,288   10 | 18    35 | 41    10 | 18    32 | 36    12 | 20    43 | 47
//    786,432   10 | 18    49 | 52    11 | 18    41 | 44    14 | 21    58 | 53
//  1,048,576   12 | 20    61 | 59    12 | 19    51 | 51    16 | 21    64 | 66
//  2,097,152   18 | 22   102 | 96    18 | 21    85 | 83    21 | 25   103 | 105
// The line is where the near-edge points take the same either way; uniform
// ones gain by one launch up to there and beyond.
constexpr long long INLINE_MAX = 1LL << 20;
// ... and of at most this many with a point per lane and the summary read in
// place: less than a block per SM, so the query's time is one point's latency
// (staging the summary first: 2 us more).
constexpr long long TINY_MAX = 1LL << 15;

namespace {

int sm_count(int device)
{
    static std::atomic<int> cache[64];
    int sms = (device >= 0 && device < 64) ? cache[device].load(std::memory_order_relaxed) : 0;
    if (!sms) {
        sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (device >= 0 && device < 64) cache[device].store(sms, std::memory_order_relaxed);
    }
    return sms;
}

template <bool FP32, int U, bool STAGE>
void launch_query(const QueryView& Q, const double2* ll, int n, uint8_t* out, unsigned long long* ctr, int sms,
                  cudaStream_t s)
{
    constexpr int POINTS = TPB * U;
    const int grid = (int)std::min<long long>(((long long)n + POINTS - 1) / POINTS, sms * (U == 1 ? 2LL : 4LL));
    const int polls = (int)knob(GAHHG_KNOB_STAGING_POLL_LIMIT);
    auto kern = ctr ? k_query<FP32, true, U, STAGE> : k_query<FP32, false, U, STAGE>;
    kern<<<grid, TPB, STAGE ? summary_bytes(Q.swords) : 0, s>>>(ll, n, out, Q, ctr, polls);
}

// Every tier in one launch, no scratch.
void query_inline(const QueryView& Q, const double2* ll, int n, uint8_t* out, int precision, unsigned long long* ctr,
                  int sms, cudaStream_t s)
{
    if (precision == GAHHG_QUERY_FP64_FILTER) {
        if (n <= TINY_MAX) launch_query<false, 1, false>(Q, ll, n, out, ctr, sms, s);
        else launch_query<false, 2, true>(Q, ll, n, out, ctr, sms, s);
    } else {
        if (n <= TINY_MAX) launch_query<true, 1, false>(Q, ll, n, out, ctr, sms, s);
        else launch_query<true, 2, true>(Q, ll, n, out, ctr, sms, s);
    }
}

}  // namespace

gahhg_status lattice_query(Grid* g, const double* d_lonlat, size_t n, uint8_t* d_labels, int precision,
                           cudaStream_t s, uint64_t* d_counters)
{
    if (n == 0) return GAHHG_OK;
    const QueryView& Q = make_view(g);
    const int sms = sm_count(g->device);
    unsigned long long* ctr = (unsigned long long*)d_counters;
    const bool fp64 = precision == GAHHG_QUERY_FP64_FILTER;
    const long long chunk = std::min<long long>((long long)n, QUERY_CHUNK);
    const long long order = knob(GAHHG_KNOB_GROUPED_PASS2);
    const bool windows = order == 1 && Q.nparts > 1 && chunk >= PART_MIN_QUEUE;
    const bool leaves = (order == 2 || order == 3) && chunk >= PART_MIN_QUEUE && g->lattice->nleaves > 0 &&
                        g->lattice->nleaves < (1LL << 30);
    const bool ordered = windows || leaves;
    if (!ordered && (long long)n <= INLINE_MAX) {
        query_inline(Q, (const double2*)d_lonlat, (int)n, d_labels, precision, ctr, sms, s);
        GAHHG_CUDA_TRY(cudaGetLastError());
        return GAHHG_OK;
    }
    const long long ptiles = (chunk + TPB * LOC_UNROLL - 1) / (TPB * LOC_UNROLL);
    const int lgrid = (int)std::min<long long>(ptiles, sms * 8LL);
    const int parts = std::min(QUEUE_PARTS, lgrid);
    // room for the points of a part's blocks (the last chunk's grid is never larger)
    const long long part_cap =
        (long long)((lgrid + parts - 1) / parts) * ((ptiles + lgrid - 1) / lgrid) * (TPB * LOC_UNROLL);
    if (part_cap * parts > 0xFFFFFFFFll) {
        set_error("query queue of %lld places", part_cap * parts);
        return GAHHG_ERR_CAPACITY;
    }
    const size_t qcap = (size_t)part_cap * parts;
    // Words: [control: overflow flag at 0, order flag at 1, entries per window at +64, windows'
    // cursors at +128, queue counts from CTL_QUEUE, tier 2's from CTL_TIER2]
    // [queue of points in leaves: points, leaf words][FP32 filter: tier 2's
    // queue: points, leaf words, masks][with an order: the ordered queue][leaf order: entries
    // per leaf: nb][leaf starts: nb + 1][tile sums][ranks].
    constexpr size_t CTL_QUEUE = 192, CTL_TIER2 = CTL_QUEUE + QUEUE_PARTS * COUNTER_STRIDE,
                     CTL_WORDS = CTL_TIER2 + QUEUE_PARTS * COUNTER_STRIDE;
    const PartQueue q2parts = tier2_parts(chunk, nullptr);
    const size_t cap2 = fp64 ? 0 : (size_t)q2parts.parts * q2parts.cap;
    const int nb = leaves ? (int)g->lattice->nleaves + 1 : 0;
    const int tiles = (nb + LS_TILE - 1) / LS_TILE;
    size_t words = CTL_WORDS;
    auto take = [&words](size_t k) {
        const size_t at = words;
        words += (k + 1) & ~(size_t)1;  // even: pairs are 8-byte aligned
        return at;
    };
    const size_t q2 = take(cap2), l2 = take(cap2), m2 = take(cap2);
    const size_t q1 = take(qcap), l1 = take(qcap);
    const size_t so = take(ordered ? 2 * (size_t)chunk : 0);
    const size_t lc = take(nb), ls = take(leaves ? nb + 1 : 0), lt = take(tiles), lr = take(leaves ? chunk : 0);
    uint32_t* mem = nullptr;
    GAHHG_TRY(pool_alloc((void**)&mem, sizeof(uint32_t) * words, g->device, s));
    gahhg_status st = GAHHG_OK;
    for (long long off = 0; off < (long long)n && st == GAHHG_OK; off += chunk) {
        const int m = (int)std::min<long long>(chunk, (long long)n - off);
        const double2* ll = (const double2*)d_lonlat + off;
        uint8_t* out = d_labels + off;
        unsigned int* ctl = mem;
        unsigned int* qc = ctl + CTL_QUEUE;
        if (cudaMemsetAsync(ctl, 0, sizeof(unsigned int) * CTL_WORDS, s) != cudaSuccess ||
            (leaves && cudaMemsetAsync(mem + lc, 0, sizeof(unsigned int) * nb, s) != cudaSuccess)) {
            set_error("query scratch: %s", cudaGetErrorString(cudaGetLastError()));
            st = GAHHG_ERR_CUDA;
            break;
        }
        Tiers T;
        T.q2 = mem + q2;
        T.l2 = mem + l2;
        T.m2 = mem + m2;
        T.p2 = q2parts;
        T.p2.cnt = ctl + CTL_TIER2;
        T.over = ctl;
        // the points in leaves, queued with their leaf words
        uint32_t *queue = mem + q1, *leafq = mem + l1;
        T.q1 = queue;
        T.l1 = leafq;
        T.p1 = PartQueue{qc, parts, (unsigned int)part_cap};
        const long long mtiles = ((long long)m + TPB * LOC_UNROLL - 1) / (TPB * LOC_UNROLL);
        const int polls = (int)knob(GAHHG_KNOB_STAGING_POLL_LIMIT);
        auto kl = ctr ? k_locate<true> : k_locate<false>;
        kl<<<(int)std::min<long long>(mtiles, lgrid), TPB, summary_bytes(Q.swords), s>>>(
            ll, m, out, Q, queue, leafq, qc, parts, (unsigned int)part_cap, ctr, polls);
        if (ordered) {
            // ... put in window or leaf order
            T.sorted = ctl + 1;
            if (windows) {
                PartScratch W;
                W.done = ctl + 1;
                W.total = ctl + 64;
                W.cursor = ctl + 128;
                W.spts = mem + so;
                W.sleaf = W.spts + chunk;
                W.np = Q.nparts;
                W.scale = Q.part_scale;
                launch_dependent_tpb(k_part_count, sms * 4, P_TPB, s, T.l1, T.p1, W);
                launch_dependent_tpb(k_part_scatter, sms * 4, P_TPB, s, T.q1, T.l1, T.p1, W);
                T.spts = W.spts;
                T.sleaf = W.sleaf;
            } else {
                LeafSortScratch LS;
                LS.done = ctl + 1;
                LS.sent = (uint2*)(mem + so);
                LS.cnt = mem + lc;
                LS.start = mem + ls;
                LS.tsum = mem + lt;
                LS.rank = mem + lr;
                LS.nb = nb;
                LS.tiles = tiles;
                launch_dependent_tpb(k_ls_count, sms * 8, LS_TPB, s, T.l1, T.p1, LS);
                launch_dependent_tpb(k_ls_tile_sums, std::min(tiles, sms * 8), LS_TPB, s, T.p1, LS);
                launch_dependent_tpb(k_ls_scan, std::min(tiles, sms * 8), LS_TPB, s, T.p1, LS);
                launch_dependent_tpb(k_ls_scatter, sms * 8, LS_TPB, s, T.q1, T.l1, T.p1, LS);
                T.spts = (const uint32_t*)LS.sent;
                T.sleaf = T.spts + 1;
                T.sstride = 2;
            }
        }
        if (!fp64 && leaves && order == 3)
            launch_dependent(k_leaf_t1s, sms * T1S_BLOCKS, s, Q, ll, out, T, ctr, polls);
        else if (!fp64)
            launch_dependent(k_leaf_t1<OneView>, sms * T1_BLOCKS, s, OneView{Q}, ll, out, T, ctr);
        tier2_launch(OneView{Q}, ll, out, T, precision, m, ctr, sms, s);
        if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) {
            set_error("query launch: %s", cudaGetErrorString(e));
            st = GAHHG_ERR_CUDA;
        }
    }
    cudaFreeAsync(mem, s);
    return st;
}

// ------------------------------------------------- allocation-free query --
//
// The query with every tier inline takes no scratch at all, so callers that
// must not allocate (see gahhg_query_device_noalloc in include/gahhg.h) get
// it at any size up to the entry point's limit.

constexpr long long NOALLOC_MAX_POINTS = 1LL << 21;  // 2,097,152 points per call

long long lattice_noalloc_max_points() { return NOALLOC_MAX_POINTS; }

gahhg_status lattice_query_noalloc(Grid* g, const double* d_lonlat, size_t n, uint8_t* d_labels, int precision,
                                   cudaStream_t s)
{
    if ((long long)n > NOALLOC_MAX_POINTS) {
        set_error("gahhg_query_device_noalloc: %zu points exceed the fixed maximum of %lld per call", n,
                  NOALLOC_MAX_POINTS);
        return GAHHG_ERR_CAPACITY;
    }
    GAHHG_TRY(check_points_aligned(d_lonlat));
    if (n == 0) return GAHHG_OK;
    query_inline(make_view(g), (const double2*)d_lonlat, (int)n, d_labels, precision, nullptr, sm_count(g->device), s);
    GAHHG_CUDA_TRY(cudaGetLastError());
    return GAHHG_OK;
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

// Points of a chunk of a segment whose summary has `swords` words: what the
// caller asked for, but 16 points per word at least as long as that makes
// chunks of 4,096 points or less, and 2 per word in any case, so that staging
// the summary costs at most two bytes per point, from L2.  (16 per word for
// every summary made chunks of 65,536 points, fewer than the blocks of the grid:
// the SMs stood idle 43 % of the pass, 150 us where 2 per word take 85; 1 and 4
// per word 87 and 91.  2 per word for small summaries too made chunks of 256
// points where a caller asks for that: 16.4M points in 16 polygons of 20 edges
// 387 us, 152 with 16.)
static long long chunk_step(int chunk_points, int swords)
{
    return std::max<long long>(chunk_points, std::max(2LL * swords, std::min(16LL * swords, 4096LL)));
}

// Chunks of a segment's step of points, segment after segment.
void batch_write_chunks(const long long* offsets, int nseg, int chunk_points, const int* swords, const int* seg_view,
                        void* out, int* nchunks)
{
    BatchChunk* v = (BatchChunk*)out;
    int n = 0;
    for (int p = 0; p < nseg; p++) {
        const long long step = chunk_step(chunk_points, swords ? swords[p] : 0);
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
                                uint32_t* queue, uint32_t* leafq, unsigned int* ccount, unsigned int* pre,
                                unsigned int* t2cnt, unsigned int* ended, unsigned long long* ctr, int polls)
{
    if constexpr (I < BATCH_NSHAPES) {
        if (shape != I) {
            batch_locate_launch<I + 1>(shape, grid, s, views, chunks, nchunks, next_chunk, ll, out, queue, leafq,
                                       ccount, pre, t2cnt, ended, ctr, polls);
            return;
        }
        constexpr int U = BATCH_SHAPES[I].unroll, B = BATCH_SHAPES[I].blocks;
        if (ctr)
            k_batch_locate<true, U, B><<<grid, TPB, 0, s>>>(views, chunks, nchunks, next_chunk, ll, out, queue, leafq,
                                                            ccount, pre, t2cnt, ended, ctr, polls);
        else
            k_batch_locate<false, U, B><<<grid, TPB, 0, s>>>(views, chunks, nchunks, next_chunk, ll, out, queue,
                                                             leafq, ccount, pre, t2cnt, ended, ctr, polls);
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

// [tier 2's counters][points in leaves: points, leaf words][tier 2's queue:
// points, leaf words, masks][queue counts of the chunks, their prefix sums]
size_t batch_queue_words(long long queue_cap, long long nchunks)
{
    const PartQueue p2 = tier2_parts(queue_cap, nullptr);
    return (size_t)QUEUE_PARTS * COUNTER_STRIDE + 2 * (size_t)queue_cap + 3 * (size_t)p2.parts * p2.cap +
           2 * (size_t)nchunks + 1;
}

// At most this many chunk counts are scanned by the last block of pass 1, one
// tile of its threads; more by a launch of their own with four times the
// threads.  (us of a replay, last block | launch: 100 chunks 14.4 | 15.9, 512
// 18.4 | 18.4, 2,000 28.3 | 28.2, 8,000 52.7 | 50.8.  With the launch alone, the
// tiers at full grids and tier 2's counters cleared by a memset, batches of a
// few hundred points took 16-18 us where they take 12-16.)
constexpr int SCAN_FOLD = TPB * CS_ITEMS;

// counters: [1] next chunk, [2] overflow flag, [3] blocks that ended.  The
// queue holds batch_queue_words(queue_cap, nchunks) words; the chunks hold
// `points` points, queue_cap at most.  Everything is enqueued on `s` (no
// allocation, no host synchronisation), so it can be captured in a graph.
gahhg_status batch_query_launch(const void* d_views, const void* d_chunks, int nchunks, const double* d_lonlat,
                                uint8_t* d_labels, int precision, uint32_t* queue, long long queue_cap,
                                long long points, unsigned int* counters, uint64_t* d_stats, cudaStream_t s, int device,
                                bool zero_counters, int shape)
{
    if (nchunks == 0) return GAHHG_OK;
    const int sms = sm_count(device);
    const QueryView* views = (const QueryView*)d_views;
    const BatchChunk* chunks = (const BatchChunk*)d_chunks;
    unsigned long long* ctr = (unsigned long long*)d_stats;
    if (zero_counters) GAHHG_CUDA_TRY(cudaMemsetAsync(counters, 0, 5 * sizeof(unsigned int), s));
    const bool fp64 = precision == GAHHG_QUERY_FP64_FILTER;
    Tiers T;
    T.p2 = tier2_parts(queue_cap, queue);
    const size_t cap2 = (size_t)T.p2.parts * T.p2.cap;
    uint32_t* q1 = queue + QUEUE_PARTS * COUNTER_STRIDE;
    T.q1 = q1;
    T.over = counters + 2;
    T.l1 = q1 + queue_cap;
    T.q2 = q1 + 2 * queue_cap;
    T.l2 = T.q2 + cap2;
    T.m2 = T.l2 + cap2;
    unsigned int* ccount = T.m2 + cap2;
    T.pre = ccount + nchunks;
    const int polls = (int)knob(GAHHG_KNOB_STAGING_POLL_LIMIT);
    if (shape < 0 || shape >= BATCH_NSHAPES) shape = 0;
    const int grid = std::min(nchunks, sms * BATCH_SHAPES[shape].blocks);  // persistent: every block resident
    const double2* ll = (const double2*)d_lonlat;
    unsigned int* pre = ccount + nchunks;
    const bool fold = nchunks <= SCAN_FOLD;
    batch_locate_launch<0>(shape, grid, s, views, chunks, nchunks, counters + 1, ll, d_labels, q1, q1 + queue_cap, ccount,
                           fold ? pre : nullptr, T.p2.cnt, counters + 3, ctr, polls);
    if (!fold) launch_dependent_tpb(k_chunk_scan, 1, CS_TPB, s, (const unsigned int*)ccount, nchunks, pre, T.p2.cnt);
    const ChunkViews vs{views, chunks, nchunks};
    if (!fp64)
        launch_dependent(k_leaf_t1<ChunkViews>, tier_grid(sms * T1_BLOCKS, points, TPB), s, vs, ll, d_labels, T, ctr);
    tier2_launch(vs, ll, d_labels, T, precision, points, ctr, sms, s);
    GAHHG_CUDA_TRY(cudaGetLastError());
    return GAHHG_OK;
}

}  // namespace gahhg
