// query_ref.cu - point queries with the reference's semantics (FP64).
//
// kernel_PISP (source/GPISPAHHG.cu:1422-1504): locate the point among the 42
// level-0 cells, descend through center and border subcells, and in a leaf
// with edges count crossings of arc(cell center, p) with each edge
// (device_isEEInter :351-378, epsilon rules included).
//
// Same arithmetic, less of it per point and in parallel:
//   * a table over longitude/latitude holds, per box, the cell every point of
//     the box comes to in the descent, or the label when that cell is a leaf
//     without edges: the descent is run once per box, and a plane test counts
//     only when it is certain for the whole box (the margin is the box's
//     radius), so a point that starts from its box's entry takes the same
//     path and the label is unchanged bit for bit.  Boxes that do not end in
//     a label are divided 4 x 4 again;
//   * the other points take eight lanes each: a level of the descent tests
//     the seven cells that may follow in one step (the first that holds the
//     point in the reference's order is taken), against border normals stored
//     at a fixed stride per cell, so a level costs two dependent loads where a
//     thread went through up to seven cells and six borders of each in turn;
//   * per (leaf, edge) the edge's normal and the sign class of its product
//     with the leaf's center are computed once, with the operations the
//     reference repeats per point, in list order, so a crossing test reads 32
//     consecutive bytes and most tests end after one product.
// Input is lon/lat (16 B/point), converted on the device with the canonical
// conversion (FakeLL2XYZ semantics, gahhg_canon.h) where a point's XYZ is
// needed; output is one byte per point.
#include <algorithm>

#include "gahhg_canon.h"
#include "gahhg_internal.h"

namespace gahhg {

namespace {

constexpr int CELL_BORDERS = 6;  // most borders of a cell
// A cell's border normals; cells with fewer borders repeat the first, which
// changes no "all borders" test.
struct __align__(16) QNormals {
    double n[CELL_BORDERS][3];
};
// What may follow a cell in the descent, in the reference's order: its center
// subcell, then its borders' subcells (-1: none; next[0] == -1: a leaf).
struct __align__(32) QNext {
    int next[8];
};
struct __align__(16) QCell {
    int rnum, rstart, type, pad;
};
struct QEdge {
    D3 p0, p1;
};
// A leaf's edge: the great circle's normal, the edge, and the class of
// normal . center (1: below -epsilon, 2: above epsilon, 0: between).
struct __align__(32) QRef {
    double n[3];
    int edge;
    int cls;
};

// The table's entries: a cell to start the descent from, ROOT (level 0),
// FINAL | label, or (512 x 256 boxes alone) FINER | a block of 4 x 4 entries.
constexpr uint32_t ENTRY_FINAL = 0x80000000u;
constexpr uint32_t ENTRY_FINER = 0x40000000u;
constexpr uint32_t ENTRY_ROOT = 0x3FFFFFFFu;
constexpr uint32_t ENTRY_INDEX = 0x3FFFFFFFu;

// 512 x 256 boxes of 0.7 degrees (512 KB), made through 32 x 16 and 128 x 64
// ones so that the boxes of a level start where the box around them ended,
// and room for 4 x 4 boxes of 0.18 degrees in 16,384 of them (1 MB; boxes
// beyond it keep their cell).
constexpr int TABLE_NX = 512, TABLE_NY = 256, TABLE_FAN = 4;
constexpr int TABLE_FINER = 16384;

struct QueryView {
    const QNormals* N;
    const QNext* X;
    const QCell* C;
    const D3* center;
    const QEdge* E;
    const QRef* R;
    const uint32_t* table;
    const uint32_t* finer;
};

struct QLayout {
    DevArray<QNormals> N;
    DevArray<QNext> X;
    DevArray<QCell> C;
    DevArray<D3> center;
    DevArray<QEdge> E;
    DevArray<QRef> R;
    DevArray<uint32_t> table, finer, coarse, middle;
    DevArray<int> boxes;  // [0] divided boxes, then their indices
};

constexpr int TPB = 256;

__global__ void k_prep_cells(const Cell* C, const Border* B, const D3* V, int nc, QCell* out, QNormals* norm,
                             QNext* next, D3* center)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nc) return;
    const Cell c = C[t];
    QCell q;
    q.rnum = c.rnum;
    q.rstart = c.rstart;
    q.type = c.type;
    q.pad = 0;
    out[t] = q;
    QNormals m;
    QNext x;
    x.next[0] = c.subcell;
    x.next[7] = -1;
    // center as kernel_PISP computes it (source/GPISPAHHG.cu:1481-1485)
    D3 s = d3(0.0, 0.0, 0.0);
    for (int i = 0; i < CELL_BORDERS; i++) {
        const Border b = B[c.bstart + (i < c.bnum ? i : 0)];
        for (int k = 0; k < 3; k++) m.n[i][k] = b.n[k];
        x.next[1 + i] = i < c.bnum ? b.subcell : -1;
        if (i < c.bnum) s = s + V[b.v[0]];
    }
    s = s / (double)c.bnum;
    center[t] = normalize(s);
    norm[t] = m;
    next[t] = x;
}

__global__ void k_prep_edges(const D3* pv, const int* pe, int n, QEdge* out)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    QEdge e;
    e.p0 = pv[pe[2 * t]];
    e.p1 = pv[pe[2 * t + 1]];
    out[t] = e;
}

// Eight lanes per cell: its edges' records (kernel_PISP's edge normal and its
// product with the center, source/GPISPAHHG.cu:351-378, 1481-1485).
__global__ void k_prep_refs(const QCell* C, const QNext* X, const D3* center, int nc, const int* refs, const QEdge* E,
                            QRef* out)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = t >> 3;
    if (c >= nc) return;
    const QCell q = C[c];
    if (X[c].next[0] != -1) return;
    for (int k = t & 7; k < q.rnum; k += 8) {
        const int id = refs[q.rstart + k];
        const QEdge e = E[id];
        const D3 n = normalize(cross(e.p0, e.p1 - e.p0));
        const double r2 = dot(n, center[c]);
        QRef r;
        r.n[0] = n.x;
        r.n[1] = n.y;
        r.n[2] = n.z;
        r.edge = id;
        r.cls = less_zero(r2) ? 1 : (gre_zero(r2) ? 2 : 0);
        out[q.rstart + k] = r;
    }
}

// The smallest product of p with the cell's border normals... as the tests
// take it: bit 0 every product is at least `in`, bit 1 some product is below
// `out`.  (A product that is not a number fails neither test, as in the
// reference, whose tests are "below -epsilon".)
__device__ __forceinline__ unsigned int cell_sides(D3 p, int cid, const QueryView& q, double in, double out)
{
    const double2* src = (const double2*)q.N[cid].n;
    double v[3 * CELL_BORDERS];
#pragma unroll
    for (int k = 0; k < 3 * CELL_BORDERS / 2; k++) {
        const double2 d = __ldg(src + k);
        v[2 * k] = d.x;
        v[2 * k + 1] = d.y;
    }
    bool below = false, some = false;
#pragma unroll
    for (int i = 0; i < CELL_BORDERS; i++) {
        const double ret = v[3 * i] * p.x + v[3 * i + 1] * p.y + v[3 * i + 2] * p.z;
        below |= ret < in;
        some |= ret < out;
    }
    return (below ? 0u : 1u) | (some ? 2u : 0u);
}

// The search of a point (r = 0) or of a whole box of points within chord r of
// p, by a group of eight lanes: the lane's candidate against the cell tests,
// then the first candidate in order that is not certainly outside.
struct Found {
    int cell;      // that candidate, -1: every candidate is certainly outside
    bool certain;  // it certainly holds all points
};

__device__ __forceinline__ Found first_of(int cand, D3 p, double r, const QueryView& q, unsigned int grp, int gshift)
{
    // (normals are unit to a rounding; 1e-12 covers the products' rounding
    // where a box's points stand for its center)
    const double slack = r > 0.0 ? r + 1e-12 : 0.0;
    const unsigned int sd = cand >= 0 ? cell_sides(p, cand, q, -POSITION_EPSILON + slack, -POSITION_EPSILON - slack) : 2u;
    const unsigned int open = (__ballot_sync(grp, !(sd & 2u)) >> gshift) & 0xFFu;
    const unsigned int sure = (__ballot_sync(grp, (sd & 1u) != 0) >> gshift) & 0xFFu;
    Found f{-1, false};
    if (open) {
        const int l = __ffs(open) - 1;
        f.cell = __shfl_sync(grp, cand, l, 8);
        f.certain = (sure >> l) & 1u;
    }
    return f;
}

constexpr int MAX_DEPTH = 64;

// Descends from `entry` (a cell, or ROOT).  A point ends in a leaf or with
// cell -1 (the reference's descent gives up); a box also where the next cell
// is not certain, with its entry so far.
struct Descent {
    int cell;   // -1: gives up; for a box -2: not past level 0
    bool leaf;
};

__device__ __forceinline__ Descent descend(uint32_t entry, D3 p, double r, const QueryView& q)
{
    const int lane = threadIdx.x & 31, gl = lane & 7, gshift = lane & 24;
    const unsigned int grp = 0xFFu << gshift;
    int cur = (int)entry;
    if (entry == ENTRY_ROOT) {
        Found f{-1, false};
        for (int i0 = 0; i0 < 42 && f.cell < 0; i0 += 8) f = first_of(i0 + gl < 42 ? i0 + gl : -1, p, r, q, grp, gshift);
        if (f.cell < 0) return Descent{-1, false};
        if (r > 0.0 && !f.certain) return Descent{-2, false};
        cur = f.cell;
    }
    for (int depth = 0; depth < MAX_DEPTH; depth++) {
        const int cand = q.X[cur].next[gl];
        if (__shfl_sync(grp, cand, 0, 8) == -1) return Descent{cur, true};
        const Found f = first_of(cand, p, r, q, grp, gshift);
        if (f.cell < 0) return Descent{-1, false};
        if (r > 0.0 && !f.certain) return Descent{cur, false};
        cur = f.cell;
    }
    return Descent{cur, true};
}

// One table level, eight lanes per box: boxes 0 .. nx * ny - 1, or (finer) the
// 4 x 4 boxes of the divided ones.  Each box starts from the entry of the box
// around it.  divide: a box that has no label joins the list of divided boxes.
__global__ void __launch_bounds__(TPB) k_table(QueryView q, int nx, int ny, const uint32_t* up, bool finer,
                                               const int* boxes, uint32_t* out, int* divide)
{
    const int nb = finer ? min(boxes[0], TABLE_FINER) * TABLE_FAN * TABLE_FAN : nx * ny;
    for (int t = (blockIdx.x * TPB + threadIdx.x) >> 3; t < nb; t += gridDim.x * TPB >> 3) {
        int ix, iy;
        uint32_t e = ENTRY_ROOT;
        if (finer) {
            const int b = boxes[1 + t / (TABLE_FAN * TABLE_FAN)], l = t % (TABLE_FAN * TABLE_FAN);
            ix = b % TABLE_NX * TABLE_FAN + l % TABLE_FAN;
            iy = b / TABLE_NX * TABLE_FAN + l / TABLE_FAN;
            e = up[nb + t / (TABLE_FAN * TABLE_FAN)];  // the divided box's own entry, kept behind the blocks
        } else {
            ix = t % nx;
            iy = t / nx;
            if (up) e = up[(iy / TABLE_FAN) * (nx / TABLE_FAN) + ix / TABLE_FAN];
        }
        const double dlon = 360.0 / nx, dlat = 180.0 / ny;
        const double lat = -90.0 + (iy + 0.5) * dlat;
        if (!(e & ENTRY_FINAL)) {
            double xyz[3];
            gahhg_canon_vertex_xyz(-180.0 + (ix + 0.5) * dlon, lat, xyz);
            // radius: along a parallel, then a meridian (the widest parallel of the
            // box), and the locate arithmetic's margin
            const double rad = GAHHG_PI_TRUNC / 180.0;
            const double eq = fmax(fabs(lat) - 0.5 * dlat, 0.0) * rad;
            const double r = 0.5 * dlat * rad + 0.5 * dlon * rad * cos(eq) * (1.0 + 1e-9) + 1e-7;
            const Descent d = descend(e, d3(xyz[0], xyz[1], xyz[2]), r, q);
            if (d.cell == -1) {
                e = ENTRY_FINAL;  // no cell for any of its points: undefined
            } else if (d.cell >= 0) {
                e = (uint32_t)d.cell;
                if (d.leaf && q.C[d.cell].rnum == 0) e = ENTRY_FINAL | (uint32_t)q.C[d.cell].type;
            }
        }
        if ((threadIdx.x & 7) == 0) {
            out[t] = e;
            if (divide && !(e & ENTRY_FINAL)) {
                const int k = atomicAdd(divide, 1);
                if (k < TABLE_FINER) divide[1 + k] = t;
            }
        }
    }
}

// The divided boxes' entries: kept behind the blocks of finer boxes while
// those are made, and replaced by the block's number.
__global__ void k_divide(const int* boxes, uint32_t* table, uint32_t* finer)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = min(boxes[0], TABLE_FINER);
    if (k >= n) return;
    finer[n * TABLE_FAN * TABLE_FAN + k] = table[boxes[1 + k]];
    table[boxes[1 + k]] = ENTRY_FINER | (uint32_t)k;
}

// A block's rounds: the table entries of its points (a label, or a place in a
// queue in shared memory), then the queued points, eight lanes each, through
// the descent and the leaf's edges; so warps are full of points that need the
// step, where a thread per point took the longest descent and the longest
// list of its warp.  The table pass is bound by its reads, the rest by the
// latency of the descent's loads.  Uniform points on the 1,100-edge star
// polygon, us, a thread per point from level 0 -> the table and eight lanes:
// 1e3 points 170 -> 14, 1e5 182 -> 21, 1e6 1165 -> 73 (66 with boxes of 0.09
// degrees, whose table took 336 us to make where this one takes 127).
template <int PER>
__global__ void __launch_bounds__(TPB) k_query_ref(const double2* __restrict__ lonlat, long long n,
                                                   uint8_t* __restrict__ out, QueryView q,
                                                   unsigned long long* inside_count)
{
    constexpr int TILE = TPB * PER;
    __shared__ uint32_t s_point[TILE], s_entry[TILE];
    __shared__ int s_n;
    const int lane = threadIdx.x & 31, gl = lane & 7;
    const unsigned int grp = 0xFFu << (lane & 24);
    int inside = 0;
    constexpr double SX = TABLE_NX / 360.0, SY = TABLE_NY / 180.0;
    for (long long base = (long long)blockIdx.x * TILE; base < n; base += (long long)gridDim.x * TILE) {
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        double2 ll[PER];
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const long long i = base + k * TPB + threadIdx.x;
            ll[k] = i < n ? lonlat[i] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const long long i = base + k * TPB + threadIdx.x;
            uint32_t e = ENTRY_ROOT;
            const double la = ll[k].y + 90.0;
            if (fabs(ll[k].x) <= 180.0 && la >= 0.0 && la <= 180.0) {
                const double u = (ll[k].x + 180.0) * SX, v = la * SY;
                const int ix = min((int)u, TABLE_NX - 1), iy = min((int)v, TABLE_NY - 1);
                e = __ldg(q.table + iy * TABLE_NX + ix);
                if ((e & (ENTRY_FINAL | ENTRY_FINER)) == ENTRY_FINER) {
                    const int fx = min((int)((u - ix) * TABLE_FAN), TABLE_FAN - 1);
                    const int fy = min((int)((v - iy) * TABLE_FAN), TABLE_FAN - 1);
                    e = __ldg(q.finer + (e & ENTRY_INDEX) * (TABLE_FAN * TABLE_FAN) + fy * TABLE_FAN + fx);
                }
            }
            const bool want = i < n && !(e & ENTRY_FINAL);
            if (i < n && !want) {
                out[i] = (uint8_t)(e & 3u);
                inside += (e & 3u) == CELL_IN;
            }
            const unsigned int m = __ballot_sync(0xffffffffu, want);
            int at = 0;
            if (lane == 0 && m) at = atomicAdd(&s_n, __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (want) {
                s_point[at] = (uint32_t)(k * TPB + threadIdx.x);
                s_entry[at] = e;
            }
        }
        __syncthreads();
        const int m = s_n;
        for (int t = threadIdx.x >> 3; t < m; t += TPB / 8) {
            const long long i = base + s_point[t];
            const double2 c2 = lonlat[i];
            // gahhg_canon_query_xyz, the latitude's sine and cosine on even
            // lanes and the longitude's on odd ones
            double sn, cs;
            gahhg_canon_sincos(gahhg_canon_rad((gl & 1) ? c2.x : gahhg_canon_query_lat(c2.y)), &sn, &cs);
            const double sa = __shfl_sync(grp, sn, 0, 8), ca = __shfl_sync(grp, cs, 0, 8);
            const double so = __shfl_sync(grp, sn, 1, 8), co = __shfl_sync(grp, cs, 1, 8);
            const D3 p = d3(ca * so, sa, ca * co);
            const Descent d = descend(s_entry[t], p, 0.0, q);
            uint8_t lab = 0;
            if (d.cell >= 0) {
                const QCell c = q.C[d.cell];
                lab = (uint8_t)c.type;
                if (c.rnum != 0) {
                    const D3 center = q.center[d.cell];
                    const D3 np = normalize(cross(center, p - center));
                    int count = 0;
                    for (int k = gl; k < c.rnum; k += 8) {
                        const QRef r = q.R[c.rstart + k];
                        const double r3 = r.n[0] * p.x + r.n[1] * p.y + r.n[2] * p.z;
                        if ((r.cls == 1 && less_zero(r3)) || (r.cls == 2 && gre_zero(r3))) continue;
                        const QEdge e = q.E[r.edge];
                        const double r0 = dot(np, e.p0), r1 = dot(np, e.p1);
                        if (!((less_zero(r0) && less_zero(r1)) || (gre_zero(r0) && gre_zero(r1)))) count++;
                    }
                    for (int k = 4; k > 0; k >>= 1) count += __shfl_xor_sync(grp, count, k);
                    if (count & 1) lab = (uint8_t)(3 - c.type);
                }
            }
            if (gl == 0) {
                out[i] = lab;
                inside += lab == CELL_IN;
            }
        }
        __syncthreads();
    }
    if (inside_count) {
        __shared__ int s_sum;
        if (threadIdx.x == 0) s_sum = 0;
        __syncthreads();
        for (int d = 16; d > 0; d >>= 1) inside += __shfl_down_sync(0xffffffffu, inside, d);
        if ((threadIdx.x & 31) == 0 && inside) atomicAdd(&s_sum, inside);
        __syncthreads();
        if (threadIdx.x == 0 && s_sum) atomicAdd(inside_count, (unsigned long long)s_sum);
    }
}

}  // namespace

static QueryView query_view(const QLayout* L)
{
    return QueryView{L->N.ptr, L->X.ptr, L->C.ptr, L->center.ptr, L->E.ptr, L->R.ptr, L->table.ptr, L->finer.ptr};
}

gahhg_status grid_prepare_query(Grid* g)
{
    if (g->qlayout) return GAHHG_OK;
    cudaStream_t s = g->stream;
    QLayout* L = new QLayout();
    const Level& last = g->levels[g->gnum - 1];
    const int nc = last.cstart + last.cnum, ne = g->poly->pv_num;
    constexpr int FF = TABLE_FAN * TABLE_FAN;
    constexpr int MX = TABLE_NX / TABLE_FAN, MY = TABLE_NY / TABLE_FAN, CX = MX / TABLE_FAN, CY = MY / TABLE_FAN;
    gahhg_status st;
    if ((st = L->N.alloc(nc, s)) != GAHHG_OK || (st = L->X.alloc(nc, s)) != GAHHG_OK ||
        (st = L->C.alloc(nc, s)) != GAHHG_OK || (st = L->center.alloc(nc, s)) != GAHHG_OK ||
        (st = L->E.alloc(ne, s)) != GAHHG_OK || (st = L->R.alloc(last.rnum, s)) != GAHHG_OK ||
        (st = L->coarse.alloc(CX * CY, s)) != GAHHG_OK || (st = L->middle.alloc(MX * MY, s)) != GAHHG_OK || (st = L->table.alloc(TABLE_NX * TABLE_NY, s)) != GAHHG_OK ||
        (st = L->finer.alloc(TABLE_FINER * (FF + 1), s)) != GAHHG_OK ||
        (st = L->boxes.alloc(TABLE_FINER + 1, s)) != GAHHG_OK) {
        delete L;
        return st;
    }
    GAHHG_CUDA_TRY(cudaMemsetAsync(L->boxes.ptr, 0, sizeof(int), s));
    k_prep_cells<<<(nc + TPB - 1) / TPB, TPB, 0, s>>>(g->C.ptr, g->B.ptr, g->V.ptr, nc, L->C.ptr, L->N.ptr, L->X.ptr,
                                                      L->center.ptr);
    k_prep_edges<<<(ne + TPB - 1) / TPB, TPB, 0, s>>>(g->poly->d_pv, g->poly->d_pe, ne, L->E.ptr);
    k_prep_refs<<<(8 * nc + TPB - 1) / TPB, TPB, 0, s>>>(L->C.ptr, L->X.ptr, L->center.ptr, nc, g->refs.ptr, L->E.ptr,
                                                         L->R.ptr);
    const QueryView q = query_view(L);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
    auto blocks = [sms](long long boxes) { return (int)std::min<long long>((8 * boxes + TPB - 1) / TPB, sms * 16LL); };
    k_table<<<blocks(CX * CY), TPB, 0, s>>>(q, CX, CY, nullptr, false, nullptr, L->coarse.ptr, nullptr);
    k_table<<<blocks(MX * MY), TPB, 0, s>>>(q, MX, MY, L->coarse.ptr, false, nullptr, L->middle.ptr, nullptr);
    k_table<<<blocks(TABLE_NX * TABLE_NY), TPB, 0, s>>>(q, TABLE_NX, TABLE_NY, L->middle.ptr, false, nullptr,
                                                        L->table.ptr, L->boxes.ptr);
    k_divide<<<TABLE_FINER / TPB, TPB, 0, s>>>(L->boxes.ptr, L->table.ptr, L->finer.ptr);
    k_table<<<blocks((long long)TABLE_FINER * FF), TPB, 0, s>>>(q, TABLE_NX * TABLE_FAN, TABLE_NY * TABLE_FAN,
                                                                L->finer.ptr, true, L->boxes.ptr, L->finer.ptr, nullptr);
    GAHHG_CUDA_TRY(cudaGetLastError());
    GAHHG_CUDA_TRY(cudaStreamSynchronize(s));
    g->qlayout = L;
    return GAHHG_OK;
}

void free_query_layout(void* p)
{
    QLayout* L = (QLayout*)p;
    if (!L) return;
    L->N.release();
    L->X.release();
    L->C.release();
    L->center.release();
    L->E.release();
    L->R.release();
    L->table.release();
    L->finer.release();
    L->coarse.release();
    L->middle.release();
    L->boxes.release();
    delete L;
}

size_t query_layout_bytes(const void* p)
{
    const QLayout* L = (const QLayout*)p;
    if (!L) return 0;
    return L->N.cap * sizeof(QNormals) + L->X.cap * sizeof(QNext) + L->C.cap * sizeof(QCell) +
           L->center.cap * sizeof(D3) + L->E.cap * sizeof(QEdge) + L->R.cap * sizeof(QRef) +
           (L->table.cap + L->finer.cap + L->coarse.cap + L->middle.cap + L->boxes.cap) * sizeof(uint32_t);
}

gahhg_status grid_query_ref(Grid* g, const double* d_lonlat, size_t n, uint8_t* d_labels, cudaStream_t s,
                            uint64_t* d_counters)
{
    GAHHG_TRY(grid_prepare_query(g));
    if (n == 0) return GAHHG_OK;
    QLayout* L = (QLayout*)g->qlayout;
    const QueryView q = query_view(L);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
    unsigned long long* ctr = d_counters ? (unsigned long long*)d_counters + 3 : nullptr;
    // rounds of 1,024 points fill the later steps' warps; below a round per
    // resident block the chip is filled by smaller rounds instead
    const long long tiles = ((long long)n + TPB * 4 - 1) / (TPB * 4);
    if (tiles >= sms * 4LL)
        k_query_ref<4><<<(int)std::min<long long>(tiles, sms * 16LL), TPB, 0, s>>>(
            (const double2*)d_lonlat, (long long)n, d_labels, q, ctr);
    else
        k_query_ref<1><<<(int)(((long long)n + TPB - 1) / TPB), TPB, 0, s>>>((const double2*)d_lonlat, (long long)n,
                                                                             d_labels, q, ctr);
    GAHHG_CUDA_TRY(cudaGetLastError());
    return GAHHG_OK;
}

}  // namespace gahhg
