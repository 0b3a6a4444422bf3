// lattice_build.cu - builds the exact-label index (lattice.cuh) of one
// polygon, or of many polygons together.
//
// The index is a lattice over longitude/latitude:
//   * top level: W x H cells of equal angular size over the polygon's domain;
//     a cell's region is its rectangle of (lon, lat) mapped through the
//     canonical conversion;
//   * an edge is listed in a cell when it may meet the cell's geodesic hull
//     (cell_box.cuh; cells too wide for a rectangle use a cap around them);
//   * a cell listing more than K edges is split 4 x 4, down to a depth limit;
//   * every cell center has an exact label: the first center is reached from a
//     point just left of an outer-ring edge through six fixed hub points, row
//     0 and each column are chained by the crossing parity of the paths
//     center -> middle of the border -> neighbouring center, each half against
//     its own cell's edges, and a child takes its parent's label XOR the
//     parity of the arc parent center -> child center against the parent's
//     edges.
//
// Every step runs once for all polygons of the build (concatenated edges and
// nodes, a polygon table for the per-polygon geometry), so launches and host
// round trips scale with levels, not with polygons: two round trips before
// the levels, one per level and one at the end (and one for every 64 edges tried
// where a polygon's first edges give no reference point).  A polygon's index does not
// depend on what it was built with, up to numbering (node words hold child
// indices relative to the polygon's first top node; leaves, records and edge
// ids count over the whole set).
//
// The 1.1M-edge polygon (device work, us per step): child labels by exact
// predicates on every child 4072, cap tests of children 1945, level-0
// neighbour parities 2336, list sorts 1709, leaf records 1048, 21 scans 738,
// level-0 labels 404.  With the lists and the labels' crossings taken in the
// cells' projection planes, children's lists filtered in order and one scan
// per level, the whole build is 1.7 ms of kernels in 2.1 ms where it was 14 in
// 17-19.
#include <cfloat>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <thread>

#include "exact_pred.cuh"
#include "host_copy.h"
#include "lattice.cuh"
#include "local_frame.cuh"

namespace gahhg {

namespace {

constexpr int TPB = 256;
inline int blocks_for(long long n) { return (int)std::max(1LL, (n + TPB - 1) / TPB); }

__host__ __device__ inline double lat_of(const D3& p) { return asin(fmin(1.0, fmax(-1.0, p.y))) / RAD; }
__host__ __device__ inline double lon_of(const D3& p) { return atan2(p.x, p.z) / RAD; }

// Latitude/longitude box (degrees) of arc AB; full_lon when it may cross a pole.
__host__ __device__ inline void arc_box(const D3& A, const D3& B, double& la0, double& la1, double& lo0, double& lo1,
                               bool& full_lon)
{
    double a = lat_of(A), b = lat_of(B);
    la0 = fmin(a, b);
    la1 = fmax(a, b);
    const D3 N = cross(A, B);
    const double nn = sqrt(dot(N, N));
    if (nn > 1e-300) {
        const D3 n = N * (1.0 / nn);
        D3 V = d3(-n.y * n.x, 1.0 - n.y * n.y, -n.y * n.z);  // highest point of the great circle
        const double vv = sqrt(dot(V, V));
        if (vv > 1e-300) {
            V = V * (1.0 / vv);
            for (int sgn = 0; sgn < 2; sgn++) {
                const D3 P = sgn ? -V : V;
                if (dot(cross(N, A), P) >= 0 && dot(cross(B, N), P) >= 0) {
                    const double lp = lat_of(P);
                    la0 = fmin(la0, lp);
                    la1 = fmax(la1, lp);
                }
            }
        }
    }
    full_lon = false;
    double oa = lon_of(A), ob = lon_of(B);
    if (fabs(a) > 89.999 || fabs(b) > 89.999 || la1 > 89.99 || la0 < -89.99) {
        full_lon = true;
        lo0 = -180;
        lo1 = 180;
        return;
    }
    if (oa > ob) {
        double t = oa;
        oa = ob;
        ob = t;
    }
    if (ob - oa <= 180.0) {
        lo0 = oa;
        lo1 = ob;
    } else {
        lo0 = ob;
        lo1 = oa + 360.0;
    }
}

// The edges' FP64 ends side by side (48 B: three aligned 16-byte loads); the
// build's kernels and the query's FP64 tier read edges from here.
__global__ void k_edge_ends(const D3* pv, const int* pe, long long n, double2* ends)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const D3 a = pv[pe[2 * e]], b = pv[pe[2 * e + 1]];
    ends[3 * e + 0] = make_double2(a.x, a.y);
    ends[3 * e + 1] = make_double2(a.z, b.x);
    ends[3 * e + 2] = make_double2(b.y, b.z);
}

__device__ __forceinline__ void load_edge(const double2* __restrict__ ends, long long e, D3& A, D3& B)
{
    const double2 u = __ldg(ends + 3 * e), v = __ldg(ends + 3 * e + 1), w = __ldg(ends + 3 * e + 2);
    A = d3(u.x, u.y, v.x);
    B = d3(v.y, w.x, w.y);
}

__device__ __forceinline__ bool same3(const D3& a, const D3& b) { return a.x == b.x && a.y == b.y && a.z == b.z; }

// base[0..n] ascending: the p with base[p] <= x < base[p + 1] (the last such
// p when ranges are empty)
__device__ __forceinline__ int find_range(const long long* __restrict__ base, int n, long long x)
{
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(base + mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The polygon of an item: the build's only one when there is no array.
__device__ __forceinline__ int poly_of(const int* __restrict__ poly, long long i) { return poly ? poly[i] : 0; }

// A set's edges from its vertices and rings (ring r: vertices rbase[r] to
// rbase[r + 1], walked backwards when dir[r]): the edge's polygon and its ends
// as k_edge_ends stores them.  (The edges' vertex numbers came from the host,
// 8 bytes an edge in a copy per polygon, until they were made here.)
__global__ void k_ring_edges(const D3* __restrict__ pv, const long long* __restrict__ rbase,
                             const uint8_t* __restrict__ dir, int nrings, const long long* __restrict__ ebase, int np,
                             long long ne, int* __restrict__ epoly, double2* __restrict__ ends)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    epoly[e] = find_range(ebase, np, e);
    const int r = find_range(rbase, nrings, e);
    const long long first = rbase[r], last = rbase[r + 1] - 1;
    const bool back = dir[r] != 0;
    const long long va = back ? last - (e - first) : e;
    const long long vb = back ? (va > first ? va - 1 : last) : (va < last ? va + 1 : first);
    const D3 a = pv[va], b = pv[vb];
    ends[3 * e + 0] = make_double2(a.x, a.y);
    ends[3 * e + 1] = make_double2(a.z, b.x);
    ends[3 * e + 2] = make_double2(b.y, b.z);
}

// ----------------------------------------------------------------- domain --
//
// Longitude/latitude domain of a polygon's edges: per edge its latitude range
// and the 0.1-degree longitude bins it touches (edges whose great circle rises
// above their ends by their great-circle box, the others by their ends'
// latitude and longitude, padded by 1e-4 degrees).  Min, max and OR do not
// depend on the order of the edges.
constexpr int DOMAIN_BIN_WORDS = (3600 + 31) / 32;
struct DomainOut {
    unsigned long long latmin, latmax;  // order-preserving keys of the doubles
    unsigned int full;
    unsigned int bins[DOMAIN_BIN_WORDS];
};

__device__ __forceinline__ unsigned long long order_key(double x)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
double from_order_key(unsigned long long k)
{
    const unsigned long long u = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
    double x;
    memcpy(&x, &u, sizeof x);
    return x;
}

// Each block takes a contiguous range of edges and accumulates in shared
// memory, flushing to the polygon's result when the polygon changes: a block
// writes a polygon once, not once per warp.
__global__ void __launch_bounds__(TPB) k_domain_scan(const double2* __restrict__ ends, long long ne,
                                                     const int* __restrict__ epoly, long long per_block,
                                                     DomainOut* out)
{
    __shared__ unsigned int s_bins[DOMAIN_BIN_WORDS];
    __shared__ unsigned long long s_min, s_max;
    __shared__ unsigned int s_full;
    const long long b0 = (long long)blockIdx.x * per_block, b1 = min(b0 + per_block, ne);
    for (long long r0 = b0; r0 < b1;) {
        // the run of this polygon's edges within the block's range
        const int p = poly_of(epoly, r0);
        __syncthreads();
        for (int k = threadIdx.x; k < DOMAIN_BIN_WORDS; k += TPB) s_bins[k] = 0;
        if (threadIdx.x == 0) {
            s_min = ~0ull;
            s_max = 0ull;
            s_full = 0;
        }
        __syncthreads();
        double lmin = 90.0, lmax = -90.0;
        bool full = false;
        long long r1 = r0;  // end of the run, the same in every thread
        bool more = true;
        while (more && r1 < b1) {
            const long long e = r1 + threadIdx.x;
            const bool mine = e < b1 && poly_of(epoly, e) == p;
            if (mine) {
                D3 a, b;
                load_edge(ends, e, a, b);
                if (!same3(a, b)) {
                    double la0, la1, lo0, lo1;
                    bool fl = false;
                    const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
                    const double sy = fmax(fabs(a.y), fabs(b.y));
                    // its great circle passes the higher end by c^2 / 8 tan(lat)
                    if ((dx * dx + dy * dy + dz * dz) * sy > 8e-6 * sqrt(fmax(1.0 - sy * sy, 0.0))) {
                        arc_box(a, b, la0, la1, lo0, lo1, fl);
                    } else {
                        // ... by less than 1e-6 rad: its ends and 1e-4 deg
                        const double ta = lat_of(a), tb = lat_of(b);
                        double oa = lon_of(a), ob = lon_of(b);
                        la0 = fmin(ta, tb) - 1e-4;
                        la1 = fmax(ta, tb) + 1e-4;
                        if (oa > ob) {
                            const double t = oa;
                            oa = ob;
                            ob = t;
                        }
                        if (ob - oa <= 180.0) {
                            lo0 = oa;
                            lo1 = ob;
                        } else {
                            lo0 = ob;
                            lo1 = oa + 360.0;
                        }
                        if (fabs(ta) > 89.9 || fabs(tb) > 89.9) fl = true;
                    }
                    lmin = fmin(lmin, la0);
                    lmax = fmax(lmax, la1);
                    if (fl) {
                        full = true;
                    } else {
                        const int k0 = (int)floor((lo0 + 180.0) * 10.0) - 1, k1 = (int)floor((lo1 + 180.0) * 10.0) + 1;
                        for (int k = k0; k <= k1 && k <= k0 + 3600; k++) {
                            const int bit = ((k % 3600) + 3600) % 3600;
                            const unsigned int w = 1u << (bit & 31);
                            if (!(*(volatile unsigned int*)&s_bins[bit >> 5] & w)) atomicOr(&s_bins[bit >> 5], w);
                        }
                    }
                }
            }
            // edges are in polygon order, so the lanes that are mine come first
            const int n = __syncthreads_count(mine);
            r1 += n;
            more = n == TPB;
        }
        for (int d = 16; d > 0; d >>= 1) {
            lmin = fmin(lmin, __shfl_down_sync(0xffffffffu, lmin, d));
            lmax = fmax(lmax, __shfl_down_sync(0xffffffffu, lmax, d));
        }
        full = __any_sync(0xffffffffu, full);
        if ((threadIdx.x & 31) == 0) {
            if (lmin <= lmax) {
                atomicMin(&s_min, order_key(lmin));
                atomicMax(&s_max, order_key(lmax));
            }
            if (full) s_full = 1;
        }
        __syncthreads();
        for (int k = threadIdx.x; k < DOMAIN_BIN_WORDS; k += TPB)
            if (s_bins[k]) atomicOr(&out[p].bins[k], s_bins[k]);
        if (threadIdx.x == 0) {
            atomicMin(&out[p].latmin, s_min);
            atomicMax(&out[p].latmax, s_max);
            if (s_full) atomicOr(&out[p].full, 1u);
        }
        r0 = r1;
    }
}

// ------------------------------------------------ the first center's label --

__constant__ double c_hubs[6][3] = {
    {1.0, 0.000731, 0.000419},  {-1.0, 0.000627, -0.000883}, {0.000577, 1.0, 0.000941},
    {-0.000351, -1.0, 0.000713}, {0.000809, -0.000467, 1.0}, {-0.000689, 0.000523, -1.0},
};

__device__ int nearest_hub(const double* q)
{
    int best = 0;
    double bd = -1e300;
    for (int k = 0; k < 6; k++) {
        const double d = c_hubs[k][0] * q[0] + c_hubs[k][1] * q[1] + c_hubs[k][2] * q[2];
        if (d > bd) {
            bd = d;
            best = k;
        }
    }
    return best;
}

// A point xi just left of edge AB and its mirror image xo (the exact oracle
// takes the same steps: offset 1e-3 * chord along the edge normal); false
// when the edge gives none.
__device__ bool reference_points(const D3& a, const D3& b, double* xi, double* xo)
{
    const double A[3] = {a.x, a.y, a.z}, B[3] = {b.x, b.y, b.z};
    const double m[3] = {A[0] + B[0], A[1] + B[1], A[2] + B[2]};
    const double nm = sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
    const double N[3] = {A[1] * B[2] - A[2] * B[1], A[2] * B[0] - A[0] * B[2], A[0] * B[1] - A[1] * B[0]};
    const double nn = sqrt(N[0] * N[0] + N[1] * N[1] + N[2] * N[2]);
    if (exact::same(A, B) || !(nm > 1e-3) || !(nn > 0)) return false;
    const double d[3] = {A[0] - B[0], A[1] - B[1], A[2] - B[2]};
    const double t = 1e-3 * sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    for (int k = 0; k < 3; k++) {
        xi[k] = m[k] / nm + t * (N[k] / nn);
        xo[k] = m[k] / nm - t * (N[k] / nn);
    }
    return exact::orient(A, B, xi) > 0 && exact::orient(A, B, xo) < 0;
}

// The arcs whose crossings decide a polygon's first center: arc 0 from xo to
// xi (must cross exactly edge `edge`), then the path xi -> hubs -> center
// (through hubs whenever an arc would exceed about 84 degrees).
constexpr int ORIGIN_PTS = 6;  // xo, xi, up to three hubs, the center
struct OriginArcs {
    double pt[ORIGIN_PTS][3];
    int np;    // points in use (0: the edge gives no reference point)
    int edge;  // the edge crossed by arc 0, within the polygon
};
struct OriginHits {
    int par[ORIGIN_PTS - 1];
    int cnt0, last0;  // crossings of arc 0
    int on0;          // an edge end coincides with an end of arc 0
    int coincident;   // ... with another point of the path
};
__device__ __forceinline__ OriginHits no_hits()
{
    OriginHits h;
    for (int k = 0; k < ORIGIN_PTS - 1; k++) h.par[k] = 0;
    h.cnt0 = 0;
    h.last0 = -1;
    h.on0 = 0;
    h.coincident = 0;
    return h;
}
// Arc 0 crosses its own edge and no other, and meets no vertex.
__device__ __forceinline__ bool arc0_serves(const OriginArcs& a, const OriginHits& h)
{
    return a.np > 0 && !h.on0 && h.par[0] == 1 && h.cnt0 == 1 && h.last0 == a.edge;
}

__device__ int origin_path(const double* xin, const double* center, double (*pt)[3])
{
    int np = 0;
    for (int k = 0; k < 3; k++) pt[np][k] = xin[k];
    np++;
    const double ud = (xin[0] * center[0] + xin[1] * center[1] + xin[2] * center[2]) /
                      sqrt((xin[0] * xin[0] + xin[1] * xin[1] + xin[2] * xin[2]) *
                           (center[0] * center[0] + center[1] * center[1] + center[2] * center[2]));
    if (ud < 0.1) {
        const int ha = nearest_hub(xin), hb = nearest_hub(center);
        for (int k = 0; k < 3; k++) pt[np][k] = c_hubs[ha][k];
        np++;
        if ((ha ^ 1) == hb) {  // opposite hubs: go round
            for (int k = 0; k < 3; k++) pt[np][k] = c_hubs[(ha + 2) % 6][k];
            np++;
        }
        if (hb != ha) {
            for (int k = 0; k < 3; k++) pt[np][k] = c_hubs[hb][k];
            np++;
        }
    }
    for (int k = 0; k < 3; k++) pt[np][k] = center[k];
    return np + 1;
}

// Polygons 0 .. np of the arrays: the arcs from outer edge `edge` of each.
__global__ void k_origin_setup(const double2* __restrict__ ends, const PolyGeo* __restrict__ pg,
                               const long long* __restrict__ ebase, int np, int edge, OriginArcs* arcs,
                               OriginHits* hits)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    OriginArcs a;
    a.np = 0;
    a.edge = edge;
    D3 A, B;
    load_edge(ends, ebase[p] + edge, A, B);
    double xi[3], xo[3];
    if (reference_points(A, B, xi, xo)) {
        const NodeCap c00 = node_cap(pg[p].g, 0, 0, 0);
        for (int k = 0; k < 3; k++) a.pt[0][k] = xo[k];
        a.np = 1 + origin_path(xi, c00.R, a.pt + 1);
    }
    arcs[p] = a;
    hits[p] = no_hits();
}

// Edges [e0, e1) against their polygons' arcs (one pass over the edges; the
// arcs of one polygon are the same for a whole warp, mostly).
__global__ void __launch_bounds__(TPB) k_origin_cross(const double2* __restrict__ ends, long long e0, long long e1,
                                                      const int* __restrict__ epoly,
                                                      const long long* __restrict__ ebase,
                                                      const OriginArcs* __restrict__ arcs, OriginHits* hits)
{
    const long long e = e0 + (long long)blockIdx.x * TPB + threadIdx.x;
    if (e >= e1) return;
    const int p = poly_of(epoly, e);
    const OriginArcs& a = arcs[p];
    const int np = a.np;
    if (np == 0) return;
    D3 a3, b3;
    load_edge(ends, e, a3, b3);
    const double A[3] = {a3.x, a3.y, a3.z}, B[3] = {b3.x, b3.y, b3.z};
    if (exact::same(A, B)) return;
    for (int k = 0; k + 1 < np; k++) {
        const double P[3] = {a.pt[k][0], a.pt[k][1], a.pt[k][2]};
        const double Q[3] = {a.pt[k + 1][0], a.pt[k + 1][1], a.pt[k + 1][2]};
        if (exact::same(A, P) || exact::same(B, P) || exact::same(A, Q) || exact::same(B, Q)) {
            if (k == 0) hits[p].on0 = 1;
            else hits[p].coincident = 1;
            continue;
        }
        if (!exact::crossing(P, Q, A, B)) continue;
        atomicXor(&hits[p].par[k], 1);
        if (k == 0) {
            atomicAdd(&hits[p].cnt0, 1);
            atomicMax(&hits[p].last0, (int)(e - ebase[p]));
        }
    }
}

// origin[p] = the label of polygon p's first level-0 center from the
// crossings found, -1 when a hub or the center coincides with a vertex,
// ORIGIN_OPEN (counted in `open`) when the edge gave no reference point.
constexpr int ORIGIN_OPEN = -2;
__global__ void k_origin(const OriginArcs* __restrict__ arcs, const OriginHits* __restrict__ hits, int np, int* origin,
                         int* open)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const OriginHits& h = hits[p];
    if (!arc0_serves(arcs[p], h)) {
        origin[p] = ORIGIN_OPEN;
        atomicAdd(open, 1);
        return;
    }
    int par = 0;
    for (int k = 1; k + 1 < arcs[p].np; k++) par ^= h.par[k];
    origin[p] = h.coincident ? -1 : par ? CELL_OUT : CELL_IN;
}

// A polygon whose first edge gives no reference point (of no length, or with
// other edges closer than a thousandth of its own length) takes the first
// outer edge that does.  ORIGIN_CANDS edges are tried at a time, by a pass of
// the whole grid over the polygon's edges: a comb of 160,000 edges, none of
// which serves before the last one, was held up 29 s when one block tried one
// edge after the other, 4.2 s by a grid and a round trip for each.
constexpr int ORIGIN_CANDS = 64;
__global__ void __launch_bounds__(ORIGIN_CANDS) k_origin_cands(const double2* __restrict__ ends, long long e0, int first,
                                                              int nouter, OriginArcs* cands, OriginHits* hits)
{
    const int k = threadIdx.x;
    OriginArcs a;
    a.np = 0;
    a.edge = first + k;
    if (a.edge < nouter) {
        D3 A, B;
        load_edge(ends, e0 + a.edge, A, B);
        if (reference_points(A, B, a.pt[1], a.pt[0])) a.np = 2;
    }
    cands[k] = a;
    hits[k] = no_hits();
}

__global__ void __launch_bounds__(TPB) k_origin_try(const double2* __restrict__ ends, long long e0, long long e1,
                                                    const OriginArcs* __restrict__ cands, OriginHits* hits)
{
    __shared__ double s_pt[ORIGIN_CANDS][2][3];
    __shared__ int s_np[ORIGIN_CANDS];
    for (int t = threadIdx.x; t < ORIGIN_CANDS; t += TPB) {
        s_np[t] = cands[t].np;
        for (int j = 0; j < 6; j++) s_pt[t][j / 3][j % 3] = cands[t].np ? cands[t].pt[j / 3][j % 3] : 0.0;
    }
    __syncthreads();
    const long long e = e0 + (long long)blockIdx.x * TPB + threadIdx.x;
    if (e >= e1) return;
    D3 a3, b3;
    load_edge(ends, e, a3, b3);
    const double A[3] = {a3.x, a3.y, a3.z}, B[3] = {b3.x, b3.y, b3.z};
    if (exact::same(A, B)) return;
    for (int k = 0; k < ORIGIN_CANDS; k++) {
        if (!s_np[k]) continue;
        const double *P = s_pt[k][0], *Q = s_pt[k][1];
        if (exact::same(A, P) || exact::same(B, P) || exact::same(A, Q) || exact::same(B, Q)) {
            hits[k].on0 = 1;
        } else if (exact::crossing(P, Q, A, B)) {
            atomicXor(&hits[k].par[0], 1);
            atomicAdd(&hits[k].cnt0, 1);
            atomicMax(&hits[k].last0, (int)(e - e0));
        }
    }
}

// *pick = the first candidate's edge that serves, -1 when none does.
__global__ void __launch_bounds__(ORIGIN_CANDS) k_origin_pick(const OriginArcs* __restrict__ cands,
                                                             const OriginHits* __restrict__ hits, int* pick)
{
    __shared__ int s_first;
    if (threadIdx.x == 0) s_first = INT_MAX;
    __syncthreads();
    if (arc0_serves(cands[threadIdx.x], hits[threadIdx.x])) atomicMin(&s_first, cands[threadIdx.x].edge);
    __syncthreads();
    if (threadIdx.x == 0) *pick = s_first == INT_MAX ? -1 : s_first;
}

// ------------------------------------------------- level 0: edges -> cells --

// A level-0 row: canonical sine and cosine of its center latitude, its cells'
// rectangle [-x1, x1] x [y0, y1] (x1 < 0: they use caps), the plane
// coordinate of the middle of the upper and lower border (qu, qd), and the
// radius of a cap that covers the cell (edges too long to project, and cells
// without a rectangle).  A row's cells differ only in longitude, so these are
// computed once per row, not per (edge, cell) test.
struct RowRec {
    double sa, ca, x1, y0, y1, qu, qd, r;
};

__global__ void k_l0_tables(const PolyGeo* __restrict__ pg, const long long* __restrict__ rbase,
                            const long long* __restrict__ cbase, int np, RowRec* rows, double2* cols)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nr = rbase[np], nc = cbase[np];
    if (t < nr) {
        const int p = find_range(rbase, np, t);
        const Geo& g = pg[p].g;
        const int iy = (int)(t - rbase[p]);
        RowRec r;
        gahhg_canon_sincos(gahhg_canon_rad(g.lat0 + ((double)iy + 0.5) * g.dlat0), &r.sa, &r.ca);
        double hl, hp;
        if (level_boxes(g, 0, hl, hp)) {
            const cellbox::Box b = cellbox::own_box(r.sa, r.ca, hl, hp);
            r.x1 = b.x1;
            r.y0 = b.y0;
            r.y1 = b.y1;
            r.r = b.x1 + fmax(-b.y0, b.y1);
        } else {
            r.x1 = -1.0;
            r.y0 = r.y1 = 0.0;
            r.r = node_cap(g, 0, 0, iy).r;
        }
        double sb, cb;
        gahhg_canon_sincos(gahhg_canon_rad(g.lat0 + (double)(iy + 1) * g.dlat0), &sb, &cb);
        r.qu = (r.ca * sb - r.sa * cb) / (r.ca * cb + r.sa * sb);
        gahhg_canon_sincos(gahhg_canon_rad(g.lat0 + (double)iy * g.dlat0), &sb, &cb);
        r.qd = (r.ca * sb - r.sa * cb) / (r.ca * cb + r.sa * sb);
        rows[t] = r;
    } else if (t < nr + nc) {
        const long long u = t - nr;
        const int p = find_range(cbase, np, u);
        const Geo& g = pg[p].g;
        double so, co;
        gahhg_canon_sincos(gahhg_canon_rad(g.lon0 + ((double)(u - cbase[p]) + 0.5) * g.dlon0), &so, &co);
        cols[u] = make_double2(so, co);
    }
}

// What an edge adds to a level-0 cell: bit 31 it is listed there; bits 0..3
// its crossing parity with the half arcs center -> middle of the upper,
// lower, left and right border (left and right on row 0 alone, where the
// columns' chains start); bit 4 a crossing is not certain in the plane.  The
// path between two neighbouring centers goes through the border's middle, so
// its parity is the XOR of two half arcs, each in the hull of one cell and so
// against that cell's list alone, found in the pass that tests the pair
// anyway: the separate pass over merged lists with exact predicates took 2336
// us on the 1.1M-edge polygon.  (In a column that path is the arc between the
// centers; in a row it has a corner, see l0_exact_parity.)
constexpr uint32_t L0_HIT = 0x80000000u;
constexpr uint32_t L0_UP = 1u, L0_DOWN = 2u, L0_LEFT = 4u, L0_RIGHT = 8u, L0_UNSURE = 16u;

__device__ __forceinline__ uint32_t l0_pair(const Geo& g, const RowRec& r, double2 col, int iy, int ix, const D3& A,
                                            const D3& B)
{
    const cellbox::Frame f{r.sa, r.ca, col.x, col.y};
    double ax, ay, bx, by;
    if (r.x1 >= 0.0 && cellbox::project(f, A, ax, ay) && cellbox::project(f, B, bx, by)) {
        if (!cellbox::meets(ax, ay, bx, by, cellbox::Box{-r.x1, r.x1, r.y0, r.y1})) return 0;
        uint32_t s = L0_HIT;
        const int u = cellbox::crosses_from_center(ax, ay, bx, by, 0.0, r.qu);
        const int d = cellbox::crosses_from_center(ax, ay, bx, by, 0.0, r.qd);
        s |= (u > 0 ? L0_UP : 0u) | (d > 0 ? L0_DOWN : 0u) | (u < 0 || d < 0 ? L0_UNSURE : 0u);
        if (iy == 0) {
            const double latc = g.lat0 + 0.5 * g.dlat0;
            for (int side = 0; side < 2; side++) {
                double m[3], qx, qy;
                gahhg_canon_vertex_xyz(g.lon0 + (double)(ix + side) * g.dlon0, latc, m);
                int c = -1;
                if (cellbox::project(f, d3(m[0], m[1], m[2]), qx, qy))
                    c = cellbox::crosses_from_center(ax, ay, bx, by, qx, qy);
                s |= (c > 0 ? (side ? L0_RIGHT : L0_LEFT) : 0u) | (c < 0 ? L0_UNSURE : 0u);
            }
        }
        return s;
    }
    const D3 R = cellbox::center_of(f);
    const double Rv[3] = {R.x, R.y, R.z};
    return edge_hits_cap(A, B, Rv, r.r) ? (L0_HIT | L0_UNSURE) : 0u;
}

// Level-0 candidates of one edge: rows [iy0, iy0 + nrows) by up to two
// column ranges [c0, c0 + n0) and [c1, c1 + n1) (the inflated longitude
// interval may wrap past 360 degrees relative to the domain's west edge).
struct EdgeBox {
    int iy0, nrows, c0, n0, c1, n1;
};

// Edges with at most SMALL_CELLS candidates are tested by their own thread,
// the hits in a 32-bit mask; a longer edge's candidates are split into work
// items of one row by at most L0_CHUNK columns, so no thread tests more
// cells: an edge near a pole (all columns) or a very long edge has a box of
// up to millions of cells, and one thread per edge would hold its block for
// tens of milliseconds.
constexpr int SMALL_CELLS = 32;
constexpr int L0_CHUNK = 64;
// Work items whose hit masks the count pass keeps for the fill pass (8 bytes
// each; beyond this the fill pass tests again).
constexpr unsigned long long L0_MASK_ITEMS = 1ull << 26;

__device__ inline int l0_chunks(int n) { return (n + L0_CHUNK - 1) / L0_CHUNK; }

// Candidate box of edge AB in the level-0 grid g.
__device__ void edge_box(const Geo& g, const D3& A, const D3& B, EdgeBox& bx)
{
    const int W = g.W, H = g.H;
    double la0, la1, lo0, lo1;
    bool full;
    arc_box(A, B, la0, la1, lo0, lo1, full);
    // How far (degrees) the box reaches beyond the edge's own ranges: the
    // hull of a cell stays in the cell's longitudes and passes its parallels
    // by at most |sin cos| (sec hl - 1) <= 0.26 hl^2; 1e-5 degrees cover the
    // locate margin and the rounding of the arc sine near a pole.  Cells that
    // use caps: the cap's radius.
    double hl, hp, rdeg, wide;
    if (level_boxes(g, 0, hl, hp)) {
        rdeg = 0.26 * hl * hl / RAD + 1e-5;
        wide = 1e-5;
    } else {
        const double rmax = (CAP_FACTOR * (0.5 * g.dlat0 + 0.5 * g.dlon0 * g.cap_cos) * RAD) * (1.0 + 1e-6) + LOC_MARGIN;
        rdeg = wide = rmax / RAD + 1e-9;
    }
    la0 -= rdeg;
    la1 += rdeg;
    int iy0 = (int)floor((la0 - g.lat0) / g.dlat0), iy1 = (int)floor((la1 - g.lat0) / g.dlat0);
    iy0 = max(iy0, 0);
    iy1 = min(iy1, H - 1);
    const double maxlat = fmax(fabs(la0), fabs(la1));
    long long r0a = 0, r0b = W - 1, r1a = 1, r1b = 0;
    bool all_cols = full || maxlat >= 89.0;
    if (!all_cols) {
        const double c = cos(maxlat * RAD);
        const double wdeg = wide / c;
        const double len = (lo1 - lo0) + 2 * wdeg;
        if (len >= 360.0) {
            all_cols = true;
        } else {
            double a = lo0 - wdeg - g.lon0;
            a -= 360.0 * floor(a / 360.0);  // [0, 360)
            r0a = (long long)floor(a / g.dlon0);
            r0b = (long long)floor((a + len) / g.dlon0);
            if (a + len >= 360.0) {
                r1a = 0;
                r1b = (long long)floor((a + len - 360.0) / g.dlon0);
            }
        }
    }
    if (all_cols) {
        r0a = 0;
        r0b = W - 1;
        r1a = 1;
        r1b = 0;
    }
    r0a = max(r0a, 0LL);
    r0b = min(r0b, (long long)W - 1);
    r1b = min(r1b, (long long)W - 1);
    bx.iy0 = iy0;
    bx.nrows = max(0, iy1 - iy0 + 1);
    bx.c0 = (int)r0a;
    bx.n0 = (int)max(0LL, r0b - r0a + 1);
    bx.c1 = (int)r1a;
    bx.n1 = (int)max(0LL, r1b - r1a + 1);
}

struct L0View {
    const double2* ends;
    long long ne;
    const int* epoly;
    const PolyGeo* pg;
    const RowRec* rows;
    const double2* cols;
};

// Work items of the long edges and list entries of all, in all polygons.
struct L0Totals {
    unsigned long long items, pairs;
};

// Per edge: its candidate box; a short edge's tests, counts and hit mask; a
// long edge's number of work items.
__global__ void __launch_bounds__(TPB) k_l0_edges(L0View v, EdgeBox* box, int* items, uint32_t* emask, int* cnt,
                                                  uint32_t* state, L0Totals* totals)
{
    const long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    unsigned long long nit = 0, npr = 0;
    if (t < v.ne) {
        EdgeBox b{0, 0, 0, 0, 0, 0};
        D3 A, B;
        load_edge(v.ends, t, A, B);
        uint32_t m = 0;
        if (!same3(A, B)) {
            const PolyGeo& P = v.pg[poly_of(v.epoly, t)];
            edge_box(P.g, A, B, b);
            const int w = b.n0 + b.n1;
            if ((long long)b.nrows * w <= SMALL_CELLS) {
                for (int r = 0; r < b.nrows; r++) {
                    const int iy = b.iy0 + r;
                    const RowRec row = v.rows[P.row0 + iy];
                    for (int c = 0; c < w; c++) {
                        const int ix = c < b.n0 ? b.c0 + c : b.c1 + (c - b.n0);
                        const uint32_t h = l0_pair(P.g, row, __ldg(v.cols + P.col0 + ix), iy, ix, A, B);
                        if (!h) continue;
                        m |= 1u << (r * w + c);
                        const long long node = P.top + (long long)iy * P.g.W + ix;
                        atomicAdd(&cnt[node], 1);
                        const uint32_t par = h & 15u;
                        if (par) atomicXor(&state[node], par);
                        if (h & L0_UNSURE) atomicOr(&state[node], L0_UNSURE);
                        npr++;
                    }
                }
            } else {
                nit = (unsigned long long)b.nrows * (l0_chunks(b.n0) + l0_chunks(b.n1));
            }
        }
        box[t] = b;
        emask[t] = m;
        items[t] = (int)min(nit, (unsigned long long)INT_MAX);
    }
    for (int o = 16; o > 0; o >>= 1) {
        nit += __shfl_down_sync(0xffffffffu, nit, o);
        npr += __shfl_down_sync(0xffffffffu, npr, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (nit) atomicAdd(&totals->items, nit);
        if (npr) atomicAdd(&totals->pairs, npr);
    }
}

// The long edges' pairs over their work items.  PASS 0 tests an item's cells
// and counts per cell, keeping the item's hits in mask[it] when mask is
// given; PASS 1 fills the lists from those masks (or tests again).
template <int PASS>
__global__ void __launch_bounds__(TPB) k_l0_items(L0View v, const EdgeBox* __restrict__ box,
                                                  const int* __restrict__ item_off, int total, int* cnt,
                                                  uint32_t* state, const int* off, int* cursor, int* list,
                                                  unsigned long long* mask, L0Totals* totals)
{
    static_assert(L0_CHUNK <= 64, "a 64-bit hit mask per item");
    unsigned long long npr = 0;
    for (long long i = (long long)blockIdx.x * TPB + threadIdx.x; i < total; i += gridDim.x * TPB) {
        const int it = (int)i;
        unsigned long long m = 0;
        if (PASS == 1 && mask) {
            m = mask[it];
            if (!m) continue;
        }
        long long lo = 0, hi = v.ne;  // the last edge whose first item is <= it
        while (hi - lo > 1) {
            const long long mid = (lo + hi) >> 1;
            if (item_off[mid] <= it) lo = mid;
            else hi = mid;
        }
        const long long t = lo;
        const EdgeBox b = box[t];
        const PolyGeo& P = v.pg[poly_of(v.epoly, t)];
        const int W = P.g.W, H = P.g.H;
        const int k0 = l0_chunks(b.n0), kk = k0 + l0_chunks(b.n1);
        const int local = it - item_off[t];
        const int iy = kk ? b.iy0 + local / kk : -1;
        const int ch = kk ? local % kk : 0;
        int xa, xb;
        if (ch < k0) {
            xa = b.c0 + ch * L0_CHUNK;
            xb = min(b.c0 + b.n0, xa + L0_CHUNK);
        } else {
            xa = b.c1 + (ch - k0) * L0_CHUNK;
            xb = min(b.c1 + b.n1, xa + L0_CHUNK);
        }
        if (iy < 0 || iy >= H || xa < 0 || xb > W) {
            if (PASS == 0 && mask) mask[it] = 0;
            continue;
        }
        const long long row = P.top + (long long)iy * W;
        if (PASS == 0 || !mask) {
            D3 A, B;
            load_edge(v.ends, t, A, B);
            const RowRec rr = v.rows[P.row0 + iy];
            for (int ix = xa; ix < xb; ix++) {
                const uint32_t h = l0_pair(P.g, rr, __ldg(v.cols + P.col0 + ix), iy, ix, A, B);
                if (!h) continue;
                m |= 1ull << (ix - xa);
                if (PASS == 0) {
                    if (h & 15u) atomicXor(&state[row + ix], h & 15u);
                    if (h & L0_UNSURE) atomicOr(&state[row + ix], L0_UNSURE);
                }
            }
        }
        if (PASS == 0) {
            if (mask) mask[it] = m;
            npr += __popcll(m);
            for (unsigned long long r = m; r; r &= r - 1) atomicAdd(&cnt[row + xa + __ffsll((long long)r) - 1], 1);
        } else {
            for (unsigned long long r = m; r; r &= r - 1) {
                const long long node = row + xa + __ffsll((long long)r) - 1;
                list[off[node] + atomicAdd(&cursor[node], 1)] = (int)t;
            }
        }
    }
    if (PASS == 0) {
        for (int o = 16; o > 0; o >>= 1) npr += __shfl_down_sync(0xffffffffu, npr, o);
        if ((threadIdx.x & 31) == 0 && npr) atomicAdd(&totals->pairs, npr);
    }
}

// The short edges' list entries, from their hit masks.
__global__ void __launch_bounds__(TPB) k_l0_fill(L0View v, const EdgeBox* __restrict__ box,
                                                 const uint32_t* __restrict__ emask, const int* __restrict__ off,
                                                 int* cursor, int* list)
{
    const long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= v.ne) return;
    uint32_t m = emask[t];
    if (!m) return;
    const EdgeBox b = box[t];
    const PolyGeo& P = v.pg[poly_of(v.epoly, t)];
    const int w = b.n0 + b.n1;
    while (m) {
        const int k = __ffs(m) - 1;
        m &= m - 1u;
        const int r = k / w, c = k % w;
        const int ix = c < b.n0 ? b.c0 + c : b.c1 + (c - b.n0);
        const long long node = P.top + (long long)(b.iy0 + r) * P.g.W + ix;
        list[off[node] + atomicAdd(&cursor[node], 1)] = (int)t;
    }
}

// The level-0 lists are filled with atomics, so their order is arbitrary;
// sorting makes the index deterministic.  Short lists are sorted by their own
// thread, middling ones by a warp (each entry's rank by counting the smaller
// ones: entries are distinct), long ones by a whole block, so no thread
// spends O(n^2) steps on one list.  (Deeper lists are filtered from their
// parent's in order.)
constexpr int SORT_THREAD = 8;
constexpr int SORT_WARP = 512;
constexpr int SORT_SMEM = 12256;  // ints staged in shared memory (48 KB with the block's counter)
constexpr int SORT_TPB = 512;

__global__ void k_sort_lists(const int* cnt, const int* off, int nn, int* list, int* mid_ids, int* nmid)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nn) return;
    const int n = cnt[p];
    if (n <= 1) return;
    if (n > SORT_THREAD) {
        mid_ids[atomicAdd(nmid, 1)] = p;
        return;
    }
    int* L = list + off[p];
    for (int i = 1; i < n; i++) {
        int x = L[i], j = i - 1;
        while (j >= 0 && L[j] > x) {
            L[j + 1] = L[j];
            j--;
        }
        L[j + 1] = x;
    }
}

// A warp per middling list (taken from a counter); longer ones are handed on
// in place.
__global__ void __launch_bounds__(TPB) k_sort_mid(const int* cnt, const int* off, int* list, const int* mid_ids,
                                                  const int* nmid, int* next, int* long_ids, int* nlong)
{
    __shared__ int sm[TPB / 32][SORT_WARP];
    const int lane = threadIdx.x & 31;
    int* s = sm[threadIdx.x >> 5];
    const int m = *nmid;
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(next, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= m) break;
        const int p = mid_ids[i];
        const int n = cnt[p];
        if (n > SORT_WARP) {
            if (lane == 0) long_ids[atomicAdd(nlong, 1)] = p;
            continue;
        }
        int* L = list + off[p];
        for (int k = lane; k < n; k += 32) s[k] = L[k];
        __syncwarp();
        for (int k = lane; k < n; k += 32) {
            const int x = s[k];
            int r = 0;
            for (int j = 0; j < n; j++) r += s[j] < x;
            L[r] = x;
        }
        __syncwarp();
    }
}

// Block-wide bitonic sort, ascending, of a[0..n) in the form where every
// comparator puts the minimum at the lower index (the first step of each
// merge compares mirrored positions).  Positions >= n act as +infinity, so
// comparators that reach them are skipped and no padding is stored.
__device__ void block_bitonic_sort(int* a, int n)
{
    int lg = 1;
    while ((1 << lg) < n) lg++;
    const int half = 1 << (lg - 1);  // comparators per step
    for (int lk = 1; lk <= lg; lk++) {
        const int k = 1 << lk;
        for (int lj = lk - 1; lj >= 0; lj--) {
            const int j = 1 << lj;
            for (int t = threadIdx.x; t < half; t += blockDim.x) {
                int i, q;
                if (lj == lk - 1) {  // mirrored compare across the two sorted halves
                    const int base = (t >> lj) << lk, pp = t & (j - 1);
                    i = base + pp;
                    q = base + k - 1 - pp;
                } else {
                    i = ((t >> lj) << (lj + 1)) + (t & (j - 1));
                    q = i + j;
                }
                if (q < n) {
                    const int x = a[i], y = a[q];
                    if (x > y) {
                        a[i] = y;
                        a[q] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// One list per block iteration (a persistent grid takes them from a counter):
// in shared memory up to SORT_SMEM entries, in place in global memory beyond.
__global__ void __launch_bounds__(SORT_TPB) k_sort_long(const int* cnt, const int* off, int* list,
                                                        const int* long_ids, const int* nlong, int* next)
{
    __shared__ int sm[SORT_SMEM];
    __shared__ int s_i;
    const int m = *nlong;
    for (;;) {
        if (threadIdx.x == 0) s_i = atomicAdd(next, 1);
        __syncthreads();
        const int i = s_i;
        if (i >= m) break;
        const int p = long_ids[i];
        const int n = cnt[p];
        int* L = list + off[p];
        if (n <= SORT_SMEM) {
            for (int k = threadIdx.x; k < n; k += blockDim.x) sm[k] = L[k];
            __syncthreads();
            block_bitonic_sort(sm, n);
            for (int k = threadIdx.x; k < n; k += blockDim.x) L[k] = sm[k];
        } else {
            block_bitonic_sort(L, n);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------ exact label tests --

// true when R coincides with an end of an edge of the list
__device__ bool center_on_vertex(const double* R, const double2* ends, const int* list, int cnt)
{
    for (int k = 0; k < cnt; k++) {
        D3 a, b;
        load_edge(ends, list[k], a, b);
        if ((a.x == R[0] && a.y == R[1] && a.z == R[2]) || (b.x == R[0] && b.y == R[1] && b.z == R[2])) return true;
    }
    return false;
}

// Moves R off a polygon vertex it coincides with (exact comparison).
__device__ void nudge_center(const Geo& g, int lvl, NodeCap& c, const double2* ends, const int* list, int cnt)
{
    const double sc = level_scale(lvl);
    for (int tries = 0; tries < 8; tries++) {
        if (!center_on_vertex(c.R, ends, list, cnt)) return;
        c.lonc += g.dlon0 / sc * (1.0 / 1024.0);
        c.latc += g.dlat0 / sc * (1.0 / 2048.0);
        gahhg_canon_vertex_xyz(c.lonc, c.latc, c.R);
    }
}

// parity of edges (from up to two sorted lists, union) crossing arc P->Q
__device__ int arc_parity_lists(const double2* ends, const double* P, const double* Q, const int* L1, int n1,
                                const int* L2, int n2, int* bad)
{
    int par = 0, i = 0, j = 0;
    while (i < n1 || j < n2) {
        int e;
        if (j >= n2 || (i < n1 && L1[i] < L2[j])) {
            e = L1[i++];
        } else if (i >= n1 || L2[j] < L1[i]) {
            e = L2[j++];
        } else {
            e = L1[i];
            i++;
            j++;
        }
        D3 a, b;
        load_edge(ends, e, a, b);
        const double A[3] = {a.x, a.y, a.z}, B[3] = {b.x, b.y, b.z};
        if (exact::same(A, B)) continue;
        if (exact::same(A, P) || exact::same(B, P) || exact::same(A, Q) || exact::same(B, Q)) {
            atomicAdd(bad, 1);
            continue;
        }
        par ^= exact::crossing(P, Q, A, B) ? 1 : 0;
    }
    return par;
}

// Exact parity between two level-0 centers (each moved off a vertex where it
// coincides with one) along a path that stays in their cells' hulls, where the
// cells' lists hold every edge.  Upwards that is the arc itself: it leaves the
// lower cell through the border between them.  Sideways it need not be: the
// arc between two centers of row 0 rises above their parallel by hl^2 / 2 sin
// cos, which in cells 64 times wider than high is above both cells.  The path
// goes through the middle of the border between them instead, each half
// against its own cell's list (as the plane's half arcs do); a middle that is
// a vertex moves along the border.
__device__ __noinline__ int l0_exact_parity(const double2* ends, const Geo& g, int i, int j, const int* La, int na,
                                            int i2, int j2, const int* Lb, int nb, int* bad)
{
    NodeCap a = node_cap(g, 0, i, j), b = node_cap(g, 0, i2, j2);
    nudge_center(g, 0, a, ends, La, na);
    nudge_center(g, 0, b, ends, Lb, nb);
    if (i == i2) return arc_parity_lists(ends, a.R, b.R, La, na, Lb, nb, bad);
    const double lon = g.lon0 + (double)i2 * g.dlon0;
    double lat = g.lat0 + ((double)j + 0.5) * g.dlat0, M[3];
    gahhg_canon_vertex_xyz(lon, lat, M);
    for (int tries = 0; tries < 8; tries++) {
        if (!center_on_vertex(M, ends, La, na) && !center_on_vertex(M, ends, Lb, nb)) break;
        lat += g.dlat0 * (1.0 / 2048.0);
        gahhg_canon_vertex_xyz(lon, lat, M);
    }
    return arc_parity_lists(ends, a.R, M, La, na, nullptr, 0, bad) ^
           arc_parity_lists(ends, M, b.R, Lb, nb, nullptr, 0, bad);
}

// Level-0 neighbour parities: per polygon its W (H - 1) vertical pairs, then
// its W - 1 horizontal pairs of row 0, from pb[p] in `par`: two half arcs of
// the pair pass, or the exact test where a crossing was not certain.
__global__ void k_l0_parity(const double2* __restrict__ ends, const PolyGeo* __restrict__ pg,
                            const long long* __restrict__ pb, int np, const int* __restrict__ cnt,
                            const int* __restrict__ off, const int* __restrict__ list,
                            const uint32_t* __restrict__ state, uint8_t* par, int* bad)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= pb[np]) return;
    const int p = np > 1 ? find_range(pb, np, t) : 0;
    const PolyGeo& P = pg[p];
    const int W = P.g.W, H = P.g.H;
    const long long u = t - pb[p];
    const long long nv = (long long)W * (H - 1);
    const bool vert = u < nv;
    const int j = vert ? (int)(u / W) : 0, i = vert ? (int)(u - (long long)j * W) : (int)(u - nv);
    const long long a0 = P.top + (long long)j * W + i, b0 = vert ? a0 + W : a0 + 1;
    const uint32_t sa = state[a0], sb = state[b0];
    int r;
    if (!((sa | sb) & L0_UNSURE))
        r = vert ? ((sa & L0_UP) != 0) ^ ((sb & L0_DOWN) != 0) : ((sa & L0_RIGHT) != 0) ^ ((sb & L0_LEFT) != 0);
    else
        r = l0_exact_parity(ends, P.g, i, j, list + off[a0], cnt[a0], vert ? i : i + 1, vert ? j + 1 : 0,
                            list + off[b0], cnt[b0], bad);
    par[t] = (uint8_t)r;
}

// Labels of the level-0 centers: row 0 by prefix XOR of the horizontal
// parities, columns by the vertical ones.  A block takes 32 columns of one
// polygon (gb: first 32-column group of each); its 32 warps take a share of
// the rows each, first their XOR, then (from the shares before) the labels:
// reads of 32 consecutive bytes, where a thread per column walked all rows
// in turn (404 us on the 5954 x 1410 grid of the 1.1M-edge polygon).
__global__ void __launch_bounds__(1024) k_l0_labels(const PolyGeo* __restrict__ pg, const long long* __restrict__ gb,
                                                    const long long* __restrict__ pb, int np,
                                                    const uint8_t* __restrict__ par, const int* __restrict__ origin,
                                                    uint8_t* label)
{
    __shared__ uint8_t s_x[32][33];
    __shared__ int s_row0;
    const int p = np > 1 ? find_range(gb, np, blockIdx.x) : 0;
    const PolyGeo& P = pg[p];
    const int W = P.g.W, H = P.g.H;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i0 = (int)(blockIdx.x - gb[p]) * 32, i = i0 + lane;
    const uint8_t* vpar = par + pb[p];
    const uint8_t* hpar = vpar + (long long)W * (H - 1);
    if (threadIdx.x == 0) s_row0 = 0;
    __syncthreads();
    int h = 0;
    for (int k = threadIdx.x; k < i0; k += 1024) h ^= hpar[k];
    h = __reduce_xor_sync(0xffffffffu, h);
    if (lane == 0 && h) atomicXor(&s_row0, 1);
    // this warp's rows of vertical pairs
    const int per = (H - 1 + 31) / 32, j0 = min(w * per, H - 1), j1 = min(j0 + per, H - 1);
    int x = 0;
    if (i < W)
        for (int j = j0; j < j1; j++) x ^= vpar[(long long)j * W + i];
    s_x[w][lane] = (uint8_t)x;
    __syncthreads();
    if (i >= W) return;
    int f = s_row0;
    for (int k = i0; k < i; k++) f ^= hpar[k];
    for (int k = 0; k < w; k++) f ^= s_x[k][lane];
    const int l0 = origin[p];  // 1 or 2
    uint8_t* col = label + P.top + i;
    if (w == 0) col[0] = (uint8_t)(f ? 3 - l0 : l0);
    for (int j = j0; j < j1; j++) {
        f ^= vpar[(long long)j * W + i];
        col[(long long)(j + 1) * W] = (uint8_t)(f ? 3 - l0 : l0);
    }
}

// Label of the region outside each polygon's domain: parity of the arc from
// a border cell's center to the center of the virtual cell just beyond the
// border, against that cell's edges (oxy[p] = (ix, iy, ox, oy) from the host,
// ox == INT_MIN: no such region).
__global__ void k_outside_label(const double2* __restrict__ ends, const PolyGeo* __restrict__ pg, int np,
                                const int4* __restrict__ oxy, const int* cnt, const int* off, const int* list,
                                const uint8_t* label, uint8_t* out, int* bad)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const int4 o = oxy[p];
    if (o.z == INT_MIN) {
        out[p] = CELL_UNDEFINED;
        return;
    }
    const PolyGeo& P = pg[p];
    const long long v = P.top + (long long)o.y * P.g.W + o.x;
    NodeCap a = node_cap(P.g, 0, o.x, o.y);
    nudge_center(P.g, 0, a, ends, list + off[v], cnt[v]);
    const NodeCap b = node_cap(P.g, 0, o.z, o.w);
    const int par = arc_parity_lists(ends, a.R, b.R, list + off[v], cnt[v], nullptr, 0, bad);
    out[p] = (uint8_t)(par ? 3 - label[v] : label[v]);
}

// Level-0 nodes' polygons.
__global__ void k_l0_polys(const long long* __restrict__ tops, int np, int nn, int* npoly)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < nn) npoly[v] = find_range(tops, np, v);
}

// ------------------------------------------------------------- level scan --
//
// One pass over a level's edge counts gives every prefix the level needs:
// list starts, and for non-empty nodes the index among refined nodes or among
// leaves and the leaf's first record (decoupled look-back as in scan.cu: a
// tile's status holds its sums, then its prefix; two 64-bit words per tile,
// word 0 = list entries and leaves, word 1 = leaf records and refined nodes,
// each with a 2-bit state; a warp per word looks back 32 tiles at a time).
// The values' fields hold 16 entries for each of the level above, which has
// 2^28 at most (PAIR_BUDGET), and any level's nodes; level 0's entries, which
// may be more, are counted in 64 bits where they are found (L0Totals).
// Waits are bounded; one that runs out sums the late tile's counts itself
// (DeviceErrors::scan_lookback_timeout counts it).
constexpr int LS_TPB = 256;
constexpr int LS_ITEMS = 8;
constexpr int LS_TILE = LS_TPB * LS_ITEMS;
constexpr int LS_LO = 33;  // bits of a word's low value (entries, records); the state is in the top two bits
static_assert(4 * PAIR_BUDGET < 1LL << LS_LO, "16 entries for each of PAIR_BUDGET / 4");
static_assert(INDEX_MASK / 4 < 1u << (62 - LS_LO) && NODE_BUDGET < 1LL << (62 - LS_LO), "a level's leaves");

struct LevelSums {
    long long pairs, recs;
    int leaves, refined;
};

struct LevelScan {
    const int* cnt;
    int nn;
    const int* npoly;
    const PolyGeo* pg;
    int kmax;  // a bound above every polygon's K stops the refinement: INT_MAX
    int* off;
    int* idx;
    int* rec;
    unsigned long long* status;  // 2 words per tile, zero before the pass
    unsigned int* next;          // tile counter, zero before the pass
    LevelSums* sums;
    DeviceErrors* err;
    long long spin_limit;
};

// The two words' contribution of a node with c edges.
__device__ __forceinline__ void ls_value(int c, int K, unsigned long long& w0, unsigned long long& w1)
{
    const bool refined = c > K, leaf = c > 0 && !refined;
    w0 = (unsigned long long)(unsigned)c + (leaf ? 1ull << LS_LO : 0ull);
    w1 = (leaf ? (unsigned long long)(unsigned)c : 0ull) + (refined ? 1ull << LS_LO : 0ull);
}

__device__ __forceinline__ int ls_k(const LevelScan& S, int p)
{
    return S.kmax == INT_MAX ? INT_MAX : S.pg[poly_of(S.npoly, p)].K;
}

__global__ void __launch_bounds__(LS_TPB) k_level_scan(LevelScan S)
{
    __shared__ int s_tile;
    __shared__ unsigned long long s_w[2][LS_TPB / 32], s_prefix[2], s_total[2];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_tile = (int)atomicAdd(S.next, 1u);
    __syncthreads();
    const int tile = s_tile;
    const int base = tile * LS_TILE + t * LS_ITEMS;
    int c[LS_ITEMS], K[LS_ITEMS];
    unsigned long long sum0 = 0, sum1 = 0;
#pragma unroll
    for (int k = 0; k < LS_ITEMS; k++) {
        const int p = base + k;
        c[k] = p < S.nn ? S.cnt[p] : 0;
        K[k] = c[k] > 0 ? ls_k(S, p) : INT_MAX;
        unsigned long long a, b;
        ls_value(c[k], K[k], a, b);
        sum0 += a;
        sum1 += b;
    }
    unsigned long long i0 = sum0, i1 = sum1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long y0 = __shfl_up_sync(0xffffffffu, i0, d), y1 = __shfl_up_sync(0xffffffffu, i1, d);
        if (lane >= d) {
            i0 += y0;
            i1 += y1;
        }
    }
    if (lane == 31) {
        s_w[0][warp] = i0;
        s_w[1][warp] = i1;
    }
    __syncthreads();
    if (warp < 2) {  // warp w: word w's offsets over the block's warps, then its look-back
        const unsigned long long v = lane < LS_TPB / 32 ? s_w[warp][lane] : 0ull;
        unsigned long long x = v;
#pragma unroll
        for (int d = 1; d < LS_TPB / 32; d <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane < LS_TPB / 32) s_w[warp][lane] = x - v;
        const unsigned long long agg = __shfl_sync(0xffffffffu, x, LS_TPB / 32 - 1);
        constexpr unsigned long long AGG = 1ull << 62, PRE = 2ull << 62, VAL = AGG - 1;
        unsigned long long excl = 0;
        unsigned long long* st = S.status + warp;
        if (tile > 0) {
            if (lane == 0) atomicExch(&st[2 * (size_t)tile], AGG | agg);
            int j = tile - 1;
            long long spins = 0;
            while (j >= 0) {
                const int mine = j - lane;
                const unsigned long long w = mine >= 0 ? *(volatile unsigned long long*)&st[2 * (size_t)mine] : PRE;
                const unsigned int pre = __ballot_sync(0xffffffffu, (w >> 62) == 2);
                const int stop = pre ? __ffs(pre) - 1 : 31;  // lanes 0..stop count
                const unsigned int late = __ballot_sync(0xffffffffu, (w >> 62) == 0 && lane <= stop);
                if (late) {
                    if (++spins <= S.spin_limit) {
                        if (spins > 64) __nanosleep(64);
                        continue;
                    }
                    // the nearest tile that is late: the sums up to it, then its own from its counts
                    const int first = __ffs(late) - 1;
                    unsigned long long a = lane < first ? (w & VAL) : 0ull;
                    const int lt = j - first;
                    for (int k = lane; k < LS_TILE; k += 32) {
                        const int p = lt * LS_TILE + k;
                        const int cc = p < S.nn ? S.cnt[p] : 0;
                        unsigned long long v0, v1;
                        ls_value(cc, cc > 0 ? ls_k(S, p) : INT_MAX, v0, v1);
                        a += warp ? v1 : v0;
                    }
                    for (int d = 16; d > 0; d >>= 1) a += __shfl_xor_sync(0xffffffffu, a, d);
                    excl += a;
                    if (lane == 0) atomicAdd(&S.err->scan_lookback_timeout, 1);
                    spins = 0;
                    j = lt - 1;
                    continue;
                }
                unsigned long long a = lane <= stop && mine >= 0 ? (w & VAL) : 0ull;
                for (int d = 16; d > 0; d >>= 1) a += __shfl_xor_sync(0xffffffffu, a, d);
                excl += a;
                if (pre) break;
                j -= 32;
            }
        }
        if (lane == 0) {
            atomicExch(&st[2 * (size_t)tile], PRE | (excl + agg));
            s_prefix[warp] = excl;
            s_total[warp] = excl + agg;
        }
    }
    __syncthreads();
    constexpr unsigned long long LO = (1ull << LS_LO) - 1;
    if (t == 0 && (long long)(tile + 1) * LS_TILE >= S.nn) {
        S.sums->pairs = (long long)(s_total[0] & LO);
        S.sums->leaves = (int)(s_total[0] >> LS_LO);
        S.sums->recs = (long long)(s_total[1] & LO);
        S.sums->refined = (int)(s_total[1] >> LS_LO);
    }
    unsigned long long r0 = s_prefix[0] + s_w[0][warp] + i0 - sum0, r1 = s_prefix[1] + s_w[1][warp] + i1 - sum1;
#pragma unroll
    for (int k = 0; k < LS_ITEMS; k++) {
        if (c[k] > 0) {  // empty nodes need no place
            const int p = base + k;
            const bool refined = c[k] > K[k];
            S.off[p] = (int)(r0 & LO);
            S.idx[p] = (int)((refined ? r1 : r0) >> LS_LO);
            if (!refined) S.rec[p] = (int)(r1 & LO);
        }
        unsigned long long a, b;
        ls_value(c[k], K[k], a, b);
        r0 += a;
        r1 += b;
    }
}

// --------------------------------------------------------------- one level --

// A level of the build, as its kernels take it.  Level-0 coordinates follow
// from the node's index.
struct LevelView {
    int nn;
    const int* cnt;
    const int* off;
    const int* idx;   // refined nodes: index among them; leaves: index among the level's leaves
    const int* rec;   // leaves: first record within the level
    const int* list;
    const uint2* ixy;
    const int* npoly;
    const uint8_t* label;
    int kmax;
    int lvl;
};

__device__ __forceinline__ void node_xy(const LevelView& v, const PolyGeo& P, int p, long long& ix, long long& iy)
{
    if (v.ixy) {
        const uint2 c = v.ixy[p];
        ix = c.x;
        iy = c.y;
    } else {
        const int u = (int)(p - P.top);
        iy = u / P.g.W;
        ix = u - (int)iy * P.g.W;
    }
}

// Node words of a level, and its refined nodes and leaves as lists.
__global__ void k_encode(LevelView v, const PolyGeo* __restrict__ pg, int child_start, int leaf_base, uint32_t* words,
                         int* rnode, int* lnode)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= v.nn) return;
    const int c = v.cnt[p];
    uint32_t w;
    if (c == 0) {
        w = KIND_PURE | v.label[p];
    } else {
        const PolyGeo& P = pg[poly_of(v.npoly, p)];
        const int i = v.idx[p];
        if (v.kmax != INT_MAX && c > P.K) {
            rnode[i] = p;
            w = KIND_INNER | (uint32_t)(child_start + FAN * FAN * (long long)i - P.top);
        } else {
            lnode[i] = p;
            w = KIND_LEAF | (uint32_t)(leaf_base + i);
        }
    }
    words[p] = w;
}

// A child as the pair pass takes it, in its parent's projection plane: the
// rectangle around the cell and the center.
struct ChildLane {
    cellbox::Frame f;  // the parent's
    bool boxes;        // false: the level uses caps
    cellbox::Box box;
    double qx, qy;
    uint2 ixy;
};

constexpr int KIDS = FAN * FAN;
constexpr int CORNERS = (FAN + 1) * (FAN + 1);

// Child l of node p, by the 16 lanes of half a warp together: the children's
// rows and columns share their sines and cosines and their corners, so a lane
// takes one center's row or column, one border's, and two of the 25 corners,
// which `s_pt` passes on.
__device__ __forceinline__ ChildLane child_lane(const LevelView& v, const PolyGeo& P, int p, int l, double2* s_pt)
{
    constexpr unsigned int ALL = 0xffffffffu;
    const Geo& g = P.g;
    long long ix, iy;
    node_xy(v, P, p, ix, iy);
    const int cx = l & (FAN - 1), cy = l / FAN;
    ChildLane c;
    c.ixy = make_uint2((unsigned)(ix * FAN + cx), (unsigned)(iy * FAN + cy));
    const double sc = level_scale(v.lvl), sc1 = level_scale(v.lvl + 1);
    // lanes 0, 1: the parent's latitude and longitude; 2..5 columns, 6..9 rows
    double deg = g.lat0 + ((double)iy + 0.5) * (g.dlat0 / sc);
    if (l == 1) deg = g.lon0 + ((double)ix + 0.5) * (g.dlon0 / sc);
    if (l >= 2) deg = g.lon0 + ((double)(ix * FAN + (l - 2)) + 0.5) * (g.dlon0 / sc1);
    if (l >= 2 + FAN) deg = g.lat0 + ((double)(iy * FAN + min(l - 2 - FAN, FAN - 1)) + 0.5) * (g.dlat0 / sc1);
    double sn, cs;
    gahhg_canon_sincos(gahhg_canon_rad(deg), &sn, &cs);
    c.f.sa = __shfl_sync(ALL, sn, 0, KIDS);
    c.f.ca = __shfl_sync(ALL, cs, 0, KIDS);
    c.f.so = __shfl_sync(ALL, sn, 1, KIDS);
    c.f.co = __shfl_sync(ALL, cs, 1, KIDS);
    const double so = __shfl_sync(ALL, sn, 2 + cx, KIDS), co = __shfl_sync(ALL, cs, 2 + cx, KIDS);
    const double sa = __shfl_sync(ALL, sn, 2 + FAN + cy, KIDS), ca = __shfl_sync(ALL, cs, 2 + FAN + cy, KIDS);
    c.qx = c.qy = 0.0;
    double hl, hp;
    c.boxes = level_boxes(g, v.lvl, hl, hp);
    if (c.boxes) cellbox::project(c.f, d3(ca * so, sa, ca * co), c.qx, c.qy);
    // lanes 0..4: the rows' borders, 5..9: the columns', at half the angle
    sincos(l <= FAN ? (l - 2) * 0.5 * hp : (min(l - 1 - FAN, FAN) - 2) * 0.25 * hl, &sn, &cs);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int j = min(l + KIDS * k, CORNERS - 1), row = j / (FAN + 1), col = j - row * (FAN + 1);
        const double sp = __shfl_sync(ALL, sn, row, KIDS), cp = __shfl_sync(ALL, cs, row, KIDS);
        const double h = __shfl_sync(ALL, sn, FAN + 1 + col, KIDS), ch = __shfl_sync(ALL, cs, FAN + 1 + col, KIDS);
        double2 q;
        cellbox::corner_at(c.f.sa, c.f.ca, 2.0 * h * ch, h, sp, cp, q.x, q.y);
        s_pt[j] = q;
    }
    __syncwarp();
    const double2* t = s_pt + cy * (FAN + 1) + cx;
    const double2 q0 = t[0], q1 = t[1], q2 = t[FAN + 1], q3 = t[FAN + 2];
    c.box = cellbox::corners_box(q0.x, q0.y, q1.x, q1.y, q2.x, q2.y, q3.x, q3.y);
    __syncwarp();  // s_pt may be rewritten
    return c;
}

// The pair pass: every edge of a refined node against its 16 children, in the
// list and across the arc between the centers.  Half a warp takes a node, a
// lane a child: the lanes project 16 edges at a time into shared memory, then
// each tests its child against them one after the other.  A ballot gives an
// edge's hits (for the fill), and a child's count and crossing parity stay in
// its lane.  The tests' FP64 instructions bound the pass (two thirds of the
// issue slots), so what an edge's tests share is made once (Segment).  A warp
// per node and a lane per edge left two thirds of the lanes idle (refined
// nodes of the 1.1M-edge polygon have about ten edges) and took 16 ballots a
// step besides: 655 us for its four levels, and 187 for a pass before that
// wrote the children's rectangles, which the lanes make here: 506 for both
// (six blocks per SM; four 631, eight 513, ten 558).
//
// Nodes with more than PAIR_LONG edges are handed to k_child_pairs_long, where
// a block takes each, so that no warp works on one node for long.
constexpr int PAIR_LONG = 256;
constexpr int PAIR_TPB = 128;

struct PairArgs {
    const double2* ends;
    const PolyGeo* pg;
    const int* rnode;
    int nref;
    uint2* cixy;
    int* cpoly;  // null for one polygon
    uint16_t* hit;
    int* ccnt;
    uint8_t* cpar;  // bit 0: parity of the center arc, bit 1: not certain
    int* longs;     // refined nodes with long lists
    int* nlong;
};

// Edges first, first + 1, ... (16 of them), first + step, ... of a list of n
// at `start`, by the half warp whose lanes hold the children `c`.  Both halves
// of a warp step together.
__device__ __forceinline__ void pair_steps(const PairArgs& a, const LevelView& v, const ChildLane& c, const Geo& g,
                                           cellbox::Segment* s_edge, int start, int n, int first, int step, int& count,
                                           unsigned int& par, unsigned int& uns)
{
    constexpr unsigned int ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, l = lane & (KIDS - 1);
    for (int k0 = first; __any_sync(ALL, k0 < n); k0 += step) {
        const int m = max(0, min(KIDS, n - k0));
        bool ok = false;
        if (l < m) {
            D3 A, B;
            load_edge(a.ends, v.list[start + k0 + l], A, B);
            double ax, ay, bx, by;
            ok = c.boxes && cellbox::project(c.f, A, ax, ay) && cellbox::project(c.f, B, bx, by);
            if (ok) s_edge[l] = cellbox::segment(ax, ay, bx, by);
        }
        const unsigned int planar = __ballot_sync(ALL, ok) >> (lane & KIDS);
        __syncwarp();
        const int most = __reduce_max_sync(ALL, m);
        unsigned int mine = 0;
        for (int k = 0; k < most; k++) {
            bool hit = false;
            if (k < m) {
                if ((planar >> k) & 1u) {
                    const cellbox::Segment e = s_edge[k];
                    hit = cellbox::meets(e, c.box);
                    const int x = cellbox::crosses_from_center(e, c.qx, c.qy);
                    par ^= x > 0;
                    uns |= x < 0;
                } else {
                    // cells too wide for a rectangle, or an edge too long to
                    // project: caps around the children, exact labels
                    D3 A, B;
                    load_edge(a.ends, v.list[start + k0 + k], A, B);
                    const NodeCap cap = node_cap(g, v.lvl + 1, (long long)c.ixy.x, (long long)c.ixy.y);
                    hit = edge_hits_cap(A, B, cap.R, cap.r);
                    uns = 1;
                }
            }
            const unsigned int hits = (__ballot_sync(ALL, hit) >> (lane & KIDS)) & 0xffffu;
            count += hit;
            if (l == k) mine = hits;
        }
        if (l < m) a.hit[start + k0 + l] = (uint16_t)mine;
        __syncwarp();  // s_edge is rewritten
    }
}

__global__ void __launch_bounds__(PAIR_TPB, 6) k_child_pairs(PairArgs a, LevelView v)
{
    __shared__ cellbox::Segment s_edge[PAIR_TPB];
    __shared__ double2 s_pt[PAIR_TPB / KIDS][CORNERS];
    const int l = threadIdx.x & (KIDS - 1);
    const long long t = (long long)blockIdx.x * PAIR_TPB + threadIdx.x;
    const bool node = t < (long long)KIDS * a.nref;
    const int r = node ? (int)(t / KIDS) : a.nref - 1;  // (halves beyond the last node repeat it, without edges)
    const int p = a.rnode[r];
    const int poly = poly_of(v.npoly, p);
    const PolyGeo& P = a.pg[poly];
    const ChildLane c = child_lane(v, P, p, l, s_pt[threadIdx.x / KIDS]);
    const int len = v.cnt[p];
    const bool here = node && len <= PAIR_LONG;
    int count = 0;
    unsigned int par = 0, uns = 0;
    pair_steps(a, v, c, P.g, s_edge + (threadIdx.x & ~(KIDS - 1)), v.off[p], here ? len : 0, 0, KIDS, count, par, uns);
    if (!node) return;
    a.cixy[t] = c.ixy;
    if (a.cpoly) a.cpoly[t] = poly;
    if (here) {
        a.ccnt[t] = count;
        a.cpar[t] = (uint8_t)(par | uns << 1);
    } else if (l == 0) {
        a.longs[atomicAdd(a.nlong, 1)] = r;
    }
}

__global__ void __launch_bounds__(TPB) k_child_pairs_long(PairArgs a, LevelView v)
{
    __shared__ cellbox::Segment s_edge[TPB];
    __shared__ double2 s_pt[TPB / KIDS][CORNERS];
    __shared__ int s_cnt[KIDS];
    __shared__ unsigned int s_par[KIDS];
    const int l = threadIdx.x & (KIDS - 1), half = threadIdx.x / KIDS;
    const int m = *a.nlong;
    for (int i = blockIdx.x; i < m; i += gridDim.x) {
        const int r = a.longs[i], p = a.rnode[r];
        __syncthreads();
        if (threadIdx.x < KIDS) s_cnt[threadIdx.x] = s_par[threadIdx.x] = 0;
        __syncthreads();
        const PolyGeo& P = a.pg[poly_of(v.npoly, p)];
        const ChildLane c = child_lane(v, P, p, l, s_pt[threadIdx.x / KIDS]);
        int count = 0;
        unsigned int par = 0, uns = 0;
        pair_steps(a, v, c, P.g, s_edge + half * KIDS, v.off[p], v.cnt[p], half * KIDS, TPB, count, par, uns);
        if (count) atomicAdd(&s_cnt[l], count);
        if (par) atomicXor(&s_par[l], 1u);
        if (uns) atomicOr(&s_par[l], 2u);
        __syncthreads();
        if (threadIdx.x < KIDS) {
            const size_t o = KIDS * (size_t)r + threadIdx.x;
            a.ccnt[o] = s_cnt[threadIdx.x];
            a.cpar[o] = (uint8_t)s_par[threadIdx.x];
        }
    }
}

// The children's lists from the hits, in the parent's order (a warp per
// refined node, ballots give each entry its place), and the labels whose
// parity is certain.
__global__ void __launch_bounds__(TPB) k_child_fill(LevelView v, const int* __restrict__ rnode, int nref,
                                                    const uint16_t* __restrict__ hit, const int* __restrict__ ccnt,
                                                    const int* __restrict__ coff, const uint8_t* __restrict__ cpar,
                                                    int* clist, uint8_t* clabel)
{
    const int lane = threadIdx.x & 31;
    const int r = blockIdx.x * (TPB / 32) + (threadIdx.x >> 5);
    if (r >= nref) return;
    const int p = rnode[r];
    const int n = v.cnt[p], start = v.off[p];
    int at = 0;  // lane l < 16: the next place in child l's list
    if (lane < FAN * FAN) {
        const size_t c = FAN * FAN * (size_t)r + lane;
        at = ccnt[c] > 0 ? coff[c] : 0;
        const int l = v.label[p];
        clabel[c] = (uint8_t)((cpar[c] & 1u) ? 3 - l : l);
    }
    const unsigned int below = (1u << lane) - 1u;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        const unsigned int m = k < n ? hit[start + k] : 0u;
        const int e = m ? v.list[start + k] : 0;
#pragma unroll
        for (int l = 0; l < FAN * FAN; l++) {
            const unsigned int b = __ballot_sync(0xffffffffu, (m >> l) & 1u);
            const int place = __shfl_sync(0xffffffffu, at, l);
            if ((m >> l) & 1u) clist[place + __popc(b & below)] = e;
            if (lane == l) at += __popc(b);
        }
    }
}

// Children whose center arc's parity was not certain: exact predicates, with
// centers moved off a vertex they coincide with.
__global__ void __launch_bounds__(TPB) k_child_exact(const double2* __restrict__ ends, LevelView v,
                                                     const PolyGeo* __restrict__ pg, const int* __restrict__ rnode,
                                                     int nchild, const uint2* __restrict__ cixy,
                                                     const int* __restrict__ ccnt, const int* __restrict__ coff,
                                                     const int* __restrict__ clist, const uint8_t* __restrict__ cpar,
                                                     uint8_t* clabel, int* bad)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nchild || !(cpar[c] & 2u)) return;
    const int p = rnode[c >> 4];
    const PolyGeo& P = pg[poly_of(v.npoly, p)];
    long long ix, iy;
    node_xy(v, P, p, ix, iy);
    NodeCap a = node_cap(P.g, v.lvl, ix, iy);
    nudge_center(P.g, v.lvl, a, ends, v.list + v.off[p], v.cnt[p]);
    NodeCap b = node_cap(P.g, v.lvl + 1, cixy[c].x, cixy[c].y);
    if (ccnt[c] > 0) nudge_center(P.g, v.lvl + 1, b, ends, clist + coff[c], ccnt[c]);
    const int par = arc_parity_lists(ends, a.R, b.R, v.list + v.off[p], v.cnt[p], nullptr, 0, bad);
    clabel[c] = (uint8_t)(par ? 3 - v.label[p] : v.label[p]);
}

// ----------------------------------------------------------- leaf records --

// A thread per leaf of a level.
__global__ void __launch_bounds__(TPB) k_leaf_records(const double2* __restrict__ ends, LevelView v,
                                                      const PolyGeo* __restrict__ pg, const int* __restrict__ lnode,
                                                      int nleaf, int leaf_base, long long rec_base, LeafRec* leaves,
                                                      float4* recs, uint32_t* eids, LeafAux* aux, int* bad)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nleaf) return;
    const int p = lnode[i];
    const PolyGeo& P = pg[poly_of(v.npoly, p)];
    long long ix, iy;
    node_xy(v, P, p, ix, iy);
    const int n = v.cnt[p];
    const int* list = v.list + v.off[p];
    const double sc = level_scale(v.lvl);
    NodeCap c;
    c.r = 0.0;
    c.lonc = P.g.lon0 + ((double)ix + 0.5) * (P.g.dlon0 / sc);
    c.latc = P.g.lat0 + ((double)iy + 0.5) * (P.g.dlat0 / sc);
    gahhg_canon_vertex_xyz(c.lonc, c.latc, c.R);
    nudge_center(P.g, v.lvl, c, ends, list, n);
    LeafRec L;
    L.lon = c.lonc;
    L.lat = c.latc;
    const long long ro = rec_base + v.rec[p];
    L.off = (uint32_t)ro;
    L.cnt = (uint16_t)min(n, 65535);
    L.label = v.label[p];
    L.pad = 0;
    {
        double sb, cb;
        gahhg_canon_sincos(gahhg_canon_rad(L.lat), &sb, &cb);
        L.sb = (float)sb;
        L.cb = (float)cb;
    }
    if (n > 65535) atomicAdd(bad + 1, 1);
    local_frame::Basis fb;
    local_frame::basis_at(c.lonc, c.latc, fb);
    LeafAux X;
    for (int k = 0; k < 3; k++) X.R[k] = c.R[k];
    for (int k = 0; k < LEAF_INLINE; k++) {
        L.rec[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = 0; j < 6; j++) X.ends[k][j] = 0.0;
    }
    X.off = L.off;
    X.cnt = L.cnt;
    X.label = L.label;
    X.signs = 0;
    for (int k = 0; k < n; k++) {
        const int e = list[k];
        D3 a, b;
        load_edge(ends, e, a, b);
        const double A[3] = {a.x, a.y, a.z}, B[3] = {b.x, b.y, b.z};
        const int s1 = exact::orient(A, B, c.R);
        if (s1 == 0) atomicAdd(bad, 1);
        float r[4];
        local_frame::edge_record(A, B, fb, s1 < 0, r);
        const float4 rec = make_float4(r[0], r[1], r[2], r[3]);
        const uint32_t word = (uint32_t)e | (s1 > 0 ? 0x80000000u : 0u);
        if (k < LEAF_INLINE) {
            L.rec[k] = rec;
            for (int j = 0; j < 3; j++) {
                X.ends[k][j] = A[j];
                X.ends[k][3 + j] = B[j];
            }
            if (s1 > 0) X.signs |= (uint8_t)(1u << k);
        } else {
            recs[ro + k] = rec;
        }
        eids[ro + k] = word;
    }
    leaves[leaf_base + i] = L;
    aux[leaf_base + i] = X;
}

// Coarse summaries (QueryView): cell c of polygon p (sc[p]: its first cell in
// the set) goes into its summary words from soff[p].  Four lanes share a
// cell's rows.
__global__ void k_summary(const uint32_t* __restrict__ nodes, const PolyGeo* __restrict__ pg,
                          const long long* __restrict__ sc, const int* __restrict__ cshift,
                          const long long* __restrict__ soff, int np, const uint8_t* __restrict__ outside,
                          uint32_t* summary)
{
    const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long t = u >> 2;
    if (t >= sc[np]) return;
    const int p = find_range(sc, np, t);
    const int c = (int)(t - sc[p]);
    const Geo& g = pg[p].g;
    const int W = g.W, H = g.H, cs = cshift[p];
    const int f = 1 << cs;
    const int CW = (W + f - 1) >> cs, CH = (H + f - 1) >> cs;
    int cx = c % (CW + 2) - 1, cy = c / (CW + 2) - 1;
    uint32_t code = 3u;  // bits seen: 1 an out cell, 2 an in cell, 4 a cell with edges
    // the ring: the domain's last cells where it goes round or reaches a pole
    if (g.full_lon) cx = min(max(cx, 0), CW - 1);
    if (g.to_south) cy = max(cy, 0);
    if (g.to_north) cy = min(cy, CH - 1);
    if (cx < 0 || cx >= CW || cy < 0 || cy >= CH) {
        code = outside[p];
    } else {
        const uint32_t* top = nodes + pg[p].top;
        uint32_t seen = 0;
        for (int y = cy * f + (int)(u & 3); y < min((cy + 1) * f, H); y += 4)
            for (int x = cx * f; x < min((cx + 1) * f, W); x++) {
                const uint32_t w = top[(size_t)y * W + x];
                seen |= (w & KIND_MASK) == KIND_PURE ? (w & 3u) : 4u;
            }
        const unsigned int grp = 0xFu << (threadIdx.x & 28);
        seen |= __shfl_xor_sync(grp, seen, 1);
        seen |= __shfl_xor_sync(grp, seen, 2);
        code = seen == 1u || seen == 2u ? seen : 0u;
    }
    if ((u & 3) == 0 && code) atomicOr(&summary[soff[p] + (c >> 4)], code << ((c & 15) * 2));
}

}  // namespace

// The level-0 grid from the domain scan's result (host).
static gahhg_status geo_from_scan(const DomainOut& h, const Polygon* P, long long target, Geo* G)
{
    double latmin = h.latmax == 0ull ? 90.0 : from_order_key(h.latmin);
    double latmax = h.latmax == 0ull ? -90.0 : from_order_key(h.latmax);
    bool full = h.full != 0;
    std::vector<uint8_t> bins(3600);  // 0.1-degree longitude bins touched by some arc
    for (int k = 0; k < 3600; k++) bins[k] = (h.bins[k >> 5] >> (k & 31)) & 1u;
    if (latmin > latmax) {
        set_error("exact index: polygon has no edges of positive length");
        return GAHHG_ERR_ARG;
    }
    // largest circular run of untouched bins = the longitude gap left outside
    int gstart = 0, glen = 0;
    if (!full) {
        int best = 0, bs = 0;
        for (int st = 0; st < 3600; st++) {
            if (bins[st] || bins[(st + 3599) % 3600] == 0) continue;  // runs start after a touched bin
            int len = 0;
            while (len < 3600 && !bins[(st + len) % 3600]) len++;
            if (len > best) {
                best = len;
                bs = st;
            }
        }
        gstart = bs;
        glen = best;
        if (glen == 0) full = true;
    }
    double lon0 = -180.0, lon_span = 360.0;
    if (!full) {
        lon0 = ((gstart + glen) % 3600) * 0.1 - 180.0;
        lon_span = (3600 - glen) * 0.1;
    }
    double lat_span = std::max(latmax - latmin, 1e-6);
    // Cells are `aspect` times wider in longitude than in latitude, so that
    // they are about square on the sphere at the median latitude of the
    // vertices; near a pole square-in-degrees cells are needles that every
    // edge crosses by the dozen.  Below an aspect of 2 cells stay square in
    // degrees.
    double aspect = 1.0;
    {
        // a strided sample of a few thousand vertices is enough for the median
        const int stride = std::max(1, P->pv_num / 4096);
        std::vector<double> alat;
        alat.reserve(P->pv_num / stride + 1);
        for (int v = 0; v < P->pv_num; v += stride) alat.push_back(fabs(P->lonlat[2 * v + 1]));
        if (!alat.empty()) {
            std::nth_element(alat.begin(), alat.begin() + alat.size() / 2, alat.end());
            const double a = 1.0 / std::max(cos(std::min(alat[alat.size() / 2], 89.99) * RAD), 1e-9);
            if (a >= 2.0) aspect = std::min(a, 64.0);
        }
    }
    // cell height (degrees) for about `target` cells, with the padding included
    double cell = sqrt(std::max(lon_span, 1e-6) * lat_span / ((double)std::max(target, 1LL) * aspect));
    bool full_lon = full, north = false, south = false;
    for (int it = 0; it < 3; it++) {
        const double pad = cell * 1.5;
        double la = latmin - pad, lb = latmax + pad;
        north = lb >= 89.0;
        south = la <= -89.0;
        bool fl = full || north || south;
        double lspan = 360.0, l0 = -180.0;
        if (!fl) {
            const double maxabs = std::min(89.0, std::max(fabs(la), fabs(lb)));
            const double padlon = std::max(pad / cos(maxabs * RAD), pad * aspect);
            lspan = lon_span + 2.0 * padlon;
            l0 = lon0 - padlon;
            if (lspan >= 359.0) fl = true;
        }
        if (fl) {
            lspan = 360.0;
            l0 = -180.0;
            if (!north && !south) {
                if (latmin + latmax >= 0.0)
                    north = true;
                else
                    south = true;
            }
        }
        if (north) lb = 90.0;
        if (south) la = -90.0;
        la = std::max(la, -90.0);
        lb = std::min(lb, 90.0);
        full_lon = fl;
        G->lon0 = l0;
        G->lat0 = la;
        lon_span = fl ? 360.0 : lon_span;
        const double ncell = sqrt(lspan * (lb - la) / ((double)std::max(target, 1LL) * aspect));
        if (it < 2 && fabs(ncell - cell) > 1e-3 * cell) {
            cell = ncell;
            if (!fl) lon0 = lon0;  // unchanged: padding recomputed from the unpadded span
            continue;
        }
        long long W = std::max(1LL, (long long)ceil(lspan / (cell * aspect)));
        long long H = std::max(1LL, (long long)ceil((lb - la) / cell));
        W = std::min(W, 16384LL);
        H = std::min(H, 16384LL);
        if ((long long)W * H >= (long long)INDEX_MASK / 4) {
            set_error("exact index: top level too large");
            return GAHHG_ERR_CAPACITY;
        }
        G->W = (int)W;
        G->H = (int)H;
        G->dlon0 = lspan / (double)W;
        G->dlat0 = (lb - la) / (double)H;
        G->full_lon = full_lon;
        G->to_north = north;
        G->to_south = south;
        // cos(latitude) at the domain's equator-ward edge, rounded up
        const double la_eq = (la <= 0.0 && lb >= 0.0) ? 0.0 : std::min(fabs(la), fabs(lb));
        G->cap_cos = std::min(1.0, cos(la_eq * RAD) * (1.0 + 1e-9) + 1e-12);
        break;
    }
    return GAHHG_OK;
}


void LatticeSet::release()
{
    nodes.release();
    leaves.release();
    recs.release();
    eids.release();
    ends.release();
    aux.release();
    summary.release();
}

long long LatticeSet::bytes() const
{
    return nnodes * (long long)sizeof(uint32_t) + nleaves * (long long)(sizeof(LeafRec) + sizeof(LeafAux)) +
           nrecs * (long long)(sizeof(float4) + sizeof(uint32_t)) + nedges * 3 * (long long)sizeof(double2);
}

long long LatticeSet::device_bytes() const
{
    return (long long)(nodes.cap * sizeof(uint32_t) +
                       leaves.cap * sizeof(LeafRec) + recs.cap * sizeof(float4) + eids.cap * sizeof(uint32_t) +
                       ends.cap * sizeof(double2) + aux.cap * sizeof(LeafAux) + summary.cap * sizeof(uint32_t));
}

namespace {

// A level's arrays on the device.
struct LevelBuf {
    int nn = 0;      // nodes at this level
    int gstart = 0;  // global index of the first node
    LevelSums sums{};
    int kmax = 0;
    DevArray<int> cnt, off, idx, rec, list, poly, rnode, lnode;
    DevArray<uint2> ixy;
    DevArray<uint8_t> label, cpar;
    DevArray<uint32_t> words;
    DevArray<uint16_t> hit;  // per list entry: the children that list it
    size_t bytes() const
    {
        return sizeof(int) * (cnt.cap + off.cap + idx.cap + rec.cap + list.cap + poly.cap + rnode.cap + lnode.cap +
                              words.cap) +
               sizeof(uint2) * ixy.cap + label.cap + cpar.cap + sizeof(uint16_t) * hit.cap;
    }
};

// host array -> device array on s (the device array is allocated here)
template <class T>
gahhg_status upload(DevArray<T>& d, const std::vector<T>& h, cudaStream_t s)
{
    GAHHG_TRY(d.alloc(h.size(), s));
    if (!h.empty()) GAHHG_CUDA_TRY(cudaMemcpyAsync(d.ptr, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, s));
    return GAHHG_OK;
}

template <class T>
gahhg_status alloc_zero(DevArray<T>& d, size_t n, cudaStream_t s)
{
    GAHHG_TRY(d.alloc(n, s));
    GAHHG_CUDA_TRY(cudaMemsetAsync(d.ptr, 0, sizeof(T) * std::max<size_t>(n, 1), s));
    return GAHHG_OK;
}

// The whole build's small device words, cleared at its start.
struct BuildWords {
    struct {
        L0Totals l0;
        LevelSums level;
        int open;  // polygons without the label of their first center
    } sums;
    int pick;
    int bad[2];      // [0] coincidences, [1] leaves of more than 65,535 edges
    int sort[4];     // middling lists, next, long lists, next
    DeviceErrors err;
};

struct Builder {
    cudaStream_t s = nullptr;
    int sms = 148;
    int np = 0;
    LatticeSet* L = nullptr;
    DevArray<int> epoly;
    DevArray<PolyGeo> d_pg;
    DevArray<BuildWords> words;
    BuildWords* w = nullptr;
    std::vector<PolyGeo> pg;
    std::vector<LevelBuf> lv;
    std::string prefix;  // of error messages

    // GAHHG_DEBUG: wall time of each phase (synchronising) on stderr
    bool dbg = false;
    double tph = 0.0;
    void phase(const char* name)
    {
        if (!dbg) return;
        cudaStreamSynchronize(s);
        const double t = now_seconds();
        fprintf(stderr, "lattice phase %-12s %9.3f ms\n", name, (t - tph) * 1e3);
        tph = t;
    }

    const int* polys_of_nodes(const LevelBuf& b) const { return np > 1 ? b.poly.ptr : nullptr; }
    LevelView view(int lvl) const
    {
        const LevelBuf& b = lv[lvl];
        return LevelView{b.nn,      b.cnt.ptr, b.off.ptr, b.idx.ptr, b.rec.ptr, b.list.ptr, lvl ? b.ixy.ptr : nullptr,
                         polys_of_nodes(b), b.label.ptr, b.kmax, lvl};
    }

    // The level's prefixes and totals; `stop`: every non-empty node is a leaf.
    gahhg_status scan_once(int lvl, bool stop)
    {
        LevelBuf& b = lv[lvl];
        b.kmax = stop ? INT_MAX : 0;
        const int tiles = (b.nn + LS_TILE - 1) / LS_TILE;
        DevArray<unsigned long long> status;
        GAHHG_TRY(alloc_zero(status, 2 * (size_t)tiles + 1, s));
        GAHHG_TRY(b.off.alloc(b.nn, s));
        GAHHG_TRY(b.idx.alloc(b.nn, s));
        GAHHG_TRY(b.rec.alloc(b.nn, s));
        const LevelScan S{b.cnt.ptr, b.nn, polys_of_nodes(b), d_pg.ptr, b.kmax, b.off.ptr, b.idx.ptr, b.rec.ptr,
                          status.ptr, (unsigned int*)(status.ptr + 2 * (size_t)tiles), &w->sums.level, &w->err,
                          knob(GAHHG_KNOB_SCAN_SPIN_LIMIT)};
        k_level_scan<<<tiles, LS_TPB, 0, s>>>(S);
        decltype(w->sums) h;
        GAHHG_CUDA_TRY(cudaMemcpyAsync(&h, &w->sums, sizeof h, cudaMemcpyDeviceToHost, s));
        GAHHG_CUDA_TRY(cudaStreamSynchronize(s));
        b.sums = h.level;
        if (lvl == 0) b.sums.pairs = (long long)h.l0.pairs;
        return GAHHG_OK;
    }
    // A level's entries have 32-bit places, and below the top the budget.
    bool too_long(int lvl) const { return lv[lvl].sums.pairs > (lvl ? PAIR_BUDGET : (long long)INT_MAX); }

    // ... under the budgets (`nodes`: in all, this level's included).  Bounded
    // refinement: a polygon whose edges fill an area densely (not a curve)
    // would need cells below the edge spacing everywhere.  Past the budget the
    // remaining cells stay leaves with more edges: the labels are the same,
    // the crossing loops longer.  (The budgets hold for the whole set.)
    gahhg_status scan(int lvl, long long nodes)
    {
        GAHHG_TRY(scan_once(lvl, lvl >= MAX_LEVEL));
        const LevelSums& c = lv[lvl].sums;
        if (!too_long(lvl) && c.refined > 0 &&
            (nodes + (long long)c.refined * FAN * FAN > NODE_BUDGET || 4 * c.pairs > PAIR_BUDGET))
            return scan_once(lvl, true);
        return GAHHG_OK;
    }

    gahhg_status retry_origins(const std::vector<long long>& ebase, const long long* d_ebase,
                               const std::vector<int>& nouter, OriginArcs* arcs, OriginHits* hits, int* origin);
    gahhg_status set_edges(Polygon* const* polys, const std::vector<long long>& ebase, const long long* d_ebase,
                           long long ne, int device);
    gahhg_status run(Grid* g, Polygon* const* polys, int count, const int* top_cells, const int* leaf_edges,
                     const D3* d_pv, const int* d_pe);
};

// The edges of a set whose vertices are on the host: one copy for all
// polygons, gathered by the copy team into its page-locked slots or, small
// sets, into one array.  (Two copies from pageable memory for each of 82
// polygons of 1.1M edges in all took 4.6 ms of a build of 6.6; without them 3.8
// there.)
gahhg_status Builder::set_edges(Polygon* const* polys, const std::vector<long long>& ebase, const long long* d_ebase,
                                long long ne, int device)
{
    std::vector<HostStage::Part> parts;
    std::vector<long long> rbase(1, 0);
    std::vector<uint8_t> dir;
    for (int p = 0; p < np; p++) {
        const Polygon* P = polys[p];
        if (P->pv_num == 0) continue;
        parts.push_back(HostStage::Part{P->pv.data(), sizeof(D3) * (size_t)P->pv_num});
        for (int r = 0; r + 1 < (int)P->ring_start.size(); r++) {
            const int a = P->ring_start[r];
            if (P->ring_start[r + 1] == a) continue;
            rbase.push_back(ebase[p] + P->ring_start[r + 1]);
            dir.push_back(P->pe[2 * (size_t)a] != a);
        }
    }
    DevArray<D3> pv;
    DevArray<long long> d_rbase;
    DevArray<uint8_t> d_dir;
    GAHHG_TRY(pv.alloc(ne, s));
    GAHHG_TRY(epoly.alloc(ne, s));
    GAHHG_TRY(upload(d_rbase, rbase, s));
    GAHHG_TRY(upload(d_dir, dir, s));
    const size_t bytes = sizeof(D3) * (size_t)ne;
    std::vector<uint8_t> all;
    if (HostStage* stage = HostStage::acquire(device, polys[0]->pv.data(), bytes, true)) {
        const cudaError_t e = stage->to_device(pv.ptr, parts, s);
        HostStage::release(stage);
        GAHHG_CUDA_TRY(e);
    } else if (bytes < HostStage::MIN_BYTES) {
        all.resize(bytes);
        uint8_t* to = all.data();
        for (const HostStage::Part& q : parts) {
            memcpy(to, q.host, q.bytes);
            to += q.bytes;
        }
        GAHHG_CUDA_TRY(cudaMemcpyAsync(pv.ptr, all.data(), bytes, cudaMemcpyHostToDevice, s));
    } else {
        uint8_t* to = (uint8_t*)pv.ptr;
        for (const HostStage::Part& q : parts) {
            GAHHG_CUDA_TRY(cudaMemcpyAsync(to, q.host, q.bytes, cudaMemcpyHostToDevice, s));
            to += q.bytes;
        }
    }
    k_ring_edges<<<blocks_for(ne), TPB, 0, s>>>(pv.ptr, d_rbase.ptr, d_dir.ptr, (int)dir.size(), d_ebase, np, ne,
                                                epoly.ptr, L->ends.ptr);
    GAHHG_CUDA_TRY(cudaGetLastError());
    return GAHHG_OK;
}

// The first centers' labels of the polygons left open by k_origin: 0 where no
// outer edge gives a reference point.
gahhg_status Builder::retry_origins(const std::vector<long long>& ebase, const long long* d_ebase,
                                    const std::vector<int>& nouter, OriginArcs* arcs, OriginHits* hits, int* origin)
{
    std::vector<int> h(np);
    GAHHG_CUDA_TRY(cudaMemcpyAsync(h.data(), origin, sizeof(int) * np, cudaMemcpyDeviceToHost, s));
    GAHHG_CUDA_TRY(cudaStreamSynchronize(s));
    DevArray<OriginArcs> cands;
    DevArray<OriginHits> chits;
    GAHHG_TRY(cands.alloc(ORIGIN_CANDS, s));
    GAHHG_TRY(chits.alloc(ORIGIN_CANDS, s));
    const double2* ends = L->ends.ptr;
    for (int p = 0; p < np; p++) {
        if (h[p] != ORIGIN_OPEN) continue;
        const long long e0 = ebase[p], e1 = ebase[p + 1];
        int pick = -1;
        for (int first = 0; first < nouter[p] && pick < 0; first += ORIGIN_CANDS) {
            k_origin_cands<<<1, ORIGIN_CANDS, 0, s>>>(ends, e0, first, nouter[p], cands.ptr, chits.ptr);
            k_origin_try<<<blocks_for(e1 - e0), TPB, 0, s>>>(ends, e0, e1, cands.ptr, chits.ptr);
            k_origin_pick<<<1, ORIGIN_CANDS, 0, s>>>(cands.ptr, chits.ptr, &w->pick);
            GAHHG_CUDA_TRY(cudaMemcpyAsync(&pick, &w->pick, sizeof pick, cudaMemcpyDeviceToHost, s));
            GAHHG_CUDA_TRY(cudaStreamSynchronize(s));
        }
        if (pick < 0) {
            GAHHG_CUDA_TRY(cudaMemsetAsync(origin + p, 0, sizeof(int), s));
            continue;
        }
        k_origin_setup<<<1, TPB, 0, s>>>(ends, d_pg.ptr + p, d_ebase + p, 1, pick, arcs + p, hits + p);
        k_origin_cross<<<blocks_for(e1 - e0), TPB, 0, s>>>(ends, e0, e1, np > 1 ? epoly.ptr : nullptr, d_ebase, arcs,
                                                           hits);
        k_origin<<<1, TPB, 0, s>>>(arcs + p, hits + p, 1, origin + p, &w->sums.open);
        GAHHG_CUDA_TRY(cudaGetLastError());
    }
    return GAHHG_OK;
}

gahhg_status Builder::run(Grid* g, Polygon* const* polys, int count, const int* top_cells, const int* leaf_edges,
                          const D3* d_pv, const int* d_pe)
{
    s = g->stream;
    np = count;
    dbg = getenv("GAHHG_DEBUG") != nullptr;
    tph = now_seconds();
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
    GAHHG_TRY(alloc_zero(words, 1, s));
    w = words.ptr;

    // ---- edges and vertices (a polygon has as many edges as vertices)
    std::vector<long long> ebase(np + 1, 0);
    std::vector<int> nouter(np);
    for (int p = 0; p < np; p++) {
        const Polygon* P = polys[p];
        ebase[p + 1] = ebase[p] + P->pv_num;
        nouter[p] = P->ring_start.size() > 1 ? P->ring_start[1] : P->pv_num;
    }
    const long long ne = ebase[np];
    if (ne >= INT_MAX / 2) {
        set_error("%s%lld edges exceed the limit of one build", prefix.c_str(), ne);
        return GAHHG_ERR_CAPACITY;
    }
    L->count = np;
    L->nedges = ne;
    DevArray<long long> d_ebase;
    GAHHG_TRY(upload(d_ebase, ebase, s));
    GAHHG_TRY(L->ends.alloc(3 * (size_t)ne, s));
    const double2* ends = L->ends.ptr;
    if (d_pv) {
        if (ne > 0) k_edge_ends<<<blocks_for(ne), TPB, 0, s>>>(d_pv, d_pe, ne, L->ends.ptr);
    } else if (ne > 0) {
        GAHHG_TRY(set_edges(polys, ebase, d_ebase.ptr, ne, g->device));
    }
    const int* ep = np > 1 ? epoly.ptr : nullptr;
    phase("edges");

    // ---- domains (one scan for every polygon, one round trip)
    pg.resize(np);
    std::vector<long long> tops(np + 1, 0), rbase(np + 1, 0), cbase(np + 1, 0);
    {
        std::vector<DomainOut> h(np);
        for (auto& d : h) {
            memset(&d, 0, sizeof d);
            d.latmin = ~0ull;
        }
        DevArray<DomainOut> d;
        GAHHG_TRY(upload(d, h, s));
        const long long per = std::max<long long>(TPB, ((ne + sms * 8LL - 1) / (sms * 8LL) + TPB - 1) / TPB * TPB);
        if (ne > 0) k_domain_scan<<<(int)((ne + per - 1) / per), TPB, 0, s>>>(ends, ne, ep, per, d.ptr);
        GAHHG_CUDA_TRY(cudaMemcpyAsync(h.data(), d.ptr, sizeof(DomainOut) * np, cudaMemcpyDeviceToHost, s));
        GAHHG_CUDA_TRY(cudaStreamSynchronize(s));
        // the level-0 grids on host threads (a polygon's takes tens of microseconds)
        std::vector<gahhg_status> st(np, GAHHG_OK);
        std::vector<std::string> msg(np);
        auto geo_range = [&](int p0, int p1) {
            for (int p = p0; p < p1; p++) {
                const long long n = polys[p]->pv_num;
                const long long target = top_cells && top_cells[p] > 0
                                             ? (long long)top_cells[p]
                                             : std::min<long long>(std::max<long long>(8LL * n, 1024), 8LL << 20);
                st[p] = geo_from_scan(h[p], polys[p], target, &pg[p].g);
                if (st[p] != GAHHG_OK) msg[p] = last_error();
            }
        };
        const int nt = std::max(1, std::min({np / 16, 16, (int)std::max(1u, std::thread::hardware_concurrency())}));
        if (nt == 1) {
            geo_range(0, np);
        } else {
            std::vector<std::thread> th;
            for (int t = 0; t < nt; t++)
                th.emplace_back(geo_range, (int)((long long)np * t / nt), (int)((long long)np * (t + 1) / nt));
            for (auto& t : th) t.join();
        }
        for (int p = 0; p < np; p++) {
            if (st[p] != GAHHG_OK) {
                if (prefix.empty()) set_error("%s", msg[p].c_str());
                else set_error("polygon %d: %s", p, msg[p].c_str());
                return st[p];
            }
            pg[p].K = leaf_edges && leaf_edges[p] > 0 ? leaf_edges[p] : DEFAULT_LEAF_EDGES;
            pg[p].top = tops[p];
            pg[p].row0 = (int)rbase[p];
            pg[p].col0 = (int)cbase[p];
            tops[p + 1] = tops[p] + (long long)pg[p].g.W * pg[p].g.H;
            rbase[p + 1] = rbase[p] + pg[p].g.H;
            cbase[p + 1] = cbase[p] + pg[p].g.W;
        }
    }
    const long long n0 = tops[np];
    if (n0 >= NODE_BUDGET && np > 1) {
        set_error("%s%lld level-0 cells exceed the node budget", prefix.c_str(), n0);
        return GAHHG_ERR_CAPACITY;
    }
    GAHHG_TRY(upload(d_pg, pg, s));
    DevArray<RowRec> rows;
    DevArray<double2> cols;
    {
        DevArray<long long> d_rbase, d_cbase;
        GAHHG_TRY(upload(d_rbase, rbase, s));
        GAHHG_TRY(upload(d_cbase, cbase, s));
        GAHHG_TRY(rows.alloc(rbase[np], s));
        GAHHG_TRY(cols.alloc(cbase[np], s));
        k_l0_tables<<<blocks_for(rbase[np] + cbase[np]), TPB, 0, s>>>(d_pg.ptr, d_rbase.ptr, d_cbase.ptr, np, rows.ptr,
                                                                     cols.ptr);
    }
    phase("domain");

    // ---- exact label of every polygon's first level-0 center
    DevArray<int> origin;
    DevArray<OriginArcs> arcs;
    DevArray<OriginHits> ohits;
    GAHHG_TRY(origin.alloc(np, s));
    GAHHG_TRY(arcs.alloc(np, s));
    GAHHG_TRY(ohits.alloc(np, s));
    k_origin_setup<<<blocks_for(np), TPB, 0, s>>>(ends, d_pg.ptr, d_ebase.ptr, np, 0, arcs.ptr, ohits.ptr);
    k_origin_cross<<<blocks_for(ne), TPB, 0, s>>>(ends, 0, ne, ep, d_ebase.ptr, arcs.ptr, ohits.ptr);
    k_origin<<<blocks_for(np), TPB, 0, s>>>(arcs.ptr, ohits.ptr, np, origin.ptr, &w->sums.open);
    phase("origin");

    // ---- level 0: candidate boxes, pair tests, counts
    lv.reserve(MAX_LEVEL + 2);
    lv.emplace_back();
    {
        LevelBuf& l0 = lv[0];
        l0.nn = (int)n0;
        l0.gstart = 0;
        GAHHG_TRY(alloc_zero(l0.cnt, l0.nn, s));
        if (np > 1) {
            DevArray<long long> d_tops;
            GAHHG_TRY(upload(d_tops, tops, s));
            GAHHG_TRY(l0.poly.alloc(l0.nn, s));
            k_l0_polys<<<blocks_for(l0.nn), TPB, 0, s>>>(d_tops.ptr, np, l0.nn, l0.poly.ptr);
        }
    }
    const L0View v0{ends, ne, ep, d_pg.ptr, rows.ptr, cols.ptr};
    DevArray<uint32_t> state, emask;
    DevArray<EdgeBox> boxes;
    DevArray<int> items, item_off;
    DevArray<unsigned long long> hits;
    GAHHG_TRY(alloc_zero(state, n0, s));
    GAHHG_TRY(emask.alloc(ne, s));
    GAHHG_TRY(boxes.alloc(ne, s));
    GAHHG_TRY(items.alloc(ne, s));
    k_l0_edges<<<blocks_for(ne), TPB, 0, s>>>(v0, boxes.ptr, items.ptr, emask.ptr, lv[0].cnt.ptr, state.ptr, &w->sums.l0);
    decltype(w->sums) first;
    GAHHG_CUDA_TRY(cudaMemcpyAsync(&first, &w->sums, sizeof first, cudaMemcpyDeviceToHost, s));
    GAHHG_CUDA_TRY(cudaStreamSynchronize(s));
    const L0Totals tot = first.l0;
    if (first.open) GAHHG_TRY(retry_origins(ebase, d_ebase.ptr, nouter, arcs.ptr, ohits.ptr, origin.ptr));
    if (tot.items > (unsigned long long)INT_MAX) {
        set_error("%s%llu level-0 candidate work items exceed 2^31 (fewer top cells are needed)", prefix.c_str(),
                  tot.items);
        return GAHHG_ERR_CAPACITY;
    }
    if (tot.items) {
        GAHHG_TRY(item_off.alloc(ne, s));
        GAHHG_TRY(scan_state_reserve(&g->scan_state, ne, s));
        GAHHG_TRY(scan_exclusive(items.ptr, item_off.ptr, (int)ne, (int*)&w->sort[3], g->scan_state, &w->err, s));
        // the count pass's hits per item, so the fill pass does not test again
        if (tot.items <= L0_MASK_ITEMS) GAHHG_TRY(hits.alloc(tot.items, s));
        k_l0_items<0><<<sms * 8, TPB, 0, s>>>(v0, boxes.ptr, item_off.ptr, (int)tot.items, lv[0].cnt.ptr, state.ptr,
                                              nullptr, nullptr, nullptr, hits.ptr, &w->sums.l0);
    }
    phase("l0 count");
    GAHHG_TRY(scan(0, n0));
    if (too_long(0)) {
        set_error("%s%lld list entries on level 0 exceed 2^31 (fewer top cells are needed)", prefix.c_str(),
                  lv[0].sums.pairs);
        return GAHHG_ERR_CAPACITY;
    }
    {
        LevelBuf& l0 = lv[0];
        DevArray<int> cursor, mid, longs;
        GAHHG_TRY(alloc_zero(cursor, l0.nn, s));
        GAHHG_TRY(l0.list.alloc(l0.sums.pairs, s));
        k_l0_fill<<<blocks_for(ne), TPB, 0, s>>>(v0, boxes.ptr, emask.ptr, l0.off.ptr, cursor.ptr, l0.list.ptr);
        if (tot.items)
            k_l0_items<1><<<sms * 8, TPB, 0, s>>>(v0, boxes.ptr, item_off.ptr, (int)tot.items, l0.cnt.ptr, state.ptr,
                                                  l0.off.ptr, cursor.ptr, l0.list.ptr, hits.ptr, nullptr);
        GAHHG_CUDA_TRY(cudaMemsetAsync(w->sort, 0, sizeof w->sort, s));
        GAHHG_TRY(mid.alloc((size_t)l0.sums.pairs / (SORT_THREAD + 1) + 1, s));
        GAHHG_TRY(longs.alloc((size_t)l0.sums.pairs / (SORT_WARP + 1) + 1, s));
        k_sort_lists<<<blocks_for(l0.nn), TPB, 0, s>>>(l0.cnt.ptr, l0.off.ptr, l0.nn, l0.list.ptr, mid.ptr, w->sort);
        k_sort_mid<<<sms * 8, TPB, 0, s>>>(l0.cnt.ptr, l0.off.ptr, l0.list.ptr, mid.ptr, w->sort, w->sort + 1,
                                           longs.ptr, w->sort + 2);
        k_sort_long<<<sms, SORT_TPB, 0, s>>>(l0.cnt.ptr, l0.off.ptr, l0.list.ptr, longs.ptr, w->sort + 2, w->sort + 3);
    }
    boxes.release();
    items.release();
    item_off.release();
    emask.release();
    hits.release();
    phase("l0 lists");

    // ---- level-0 labels and each polygon's label outside its domain
    int* bad = w->bad;
    DevArray<uint8_t> outl;
    GAHHG_TRY(outl.alloc(np, s));
    {
        LevelBuf& l0 = lv[0];
        std::vector<long long> pb(np + 1, 0), gb(np + 1, 0);
        std::vector<int4> oxy(np);
        for (int p = 0; p < np; p++) {
            const Geo& G0 = pg[p].g;
            const int W = G0.W, H = G0.H;
            pb[p + 1] = pb[p] + (long long)W * (H - 1) + (W - 1);
            gb[p + 1] = gb[p] + (W + 31) / 32;
            // the region outside the domain, from the nearest border cell
            int ix = 0, iy = 0, ox = 0, oy = 0;
            if (!G0.full_lon) {
                ox = -1;
            } else if (!G0.to_south) {
                oy = -1;
            } else if (!G0.to_north) {
                iy = H - 1;
                oy = H;
            } else {
                ox = INT_MIN;  // no outside region
            }
            oxy[p] = make_int4(ix, iy, ox, oy);
        }
        DevArray<long long> d_pb, d_gb;
        DevArray<int4> d_oxy;
        DevArray<uint8_t> par;
        GAHHG_TRY(upload(d_pb, pb, s));
        GAHHG_TRY(upload(d_gb, gb, s));
        GAHHG_TRY(upload(d_oxy, oxy, s));
        GAHHG_TRY(par.alloc(pb[np], s));
        GAHHG_TRY(l0.label.alloc(l0.nn, s));
        if (pb[np] > 0)
            k_l0_parity<<<blocks_for(pb[np]), TPB, 0, s>>>(ends, d_pg.ptr, d_pb.ptr, np, l0.cnt.ptr, l0.off.ptr,
                                                           l0.list.ptr, state.ptr, par.ptr, bad);
        k_l0_labels<<<(int)gb[np], 1024, 0, s>>>(d_pg.ptr, d_gb.ptr, d_pb.ptr, np, par.ptr, origin.ptr, l0.label.ptr);
        k_outside_label<<<blocks_for(np), TPB, 0, s>>>(ends, d_pg.ptr, np, d_oxy.ptr, l0.cnt.ptr, l0.off.ptr,
                                                       l0.list.ptr, l0.label.ptr, outl.ptr, bad);
    }
    state.release();
    phase("l0 labels");

    // ---- the levels: node words and leaves of one, then the next one's cells
    long long gnext = n0, leaf_total = 0, rec_total = 0;
    std::vector<int> leaf_base;
    std::vector<long long> rec_base;
    // node words, refined nodes and leaves of a level whose labels are known
    auto encode = [&](int lvl) -> gahhg_status {
        LevelBuf& b = lv[lvl];
        leaf_base.push_back((int)leaf_total);
        rec_base.push_back(rec_total);
        leaf_total += b.sums.leaves;
        rec_total += b.sums.recs;
        if (dbg)
            fprintf(stderr, "lattice level %d: %d cells, %lld edge entries, %d split, %d leaves of %lld entries\n",
                    lvl, b.nn, b.sums.pairs, b.sums.refined, b.sums.leaves, b.sums.recs);
        if (rec_total >= 0xFFFFFFFFll || leaf_total >= (long long)INDEX_MASK) {
            set_error("%stoo many leaves or edge records", prefix.c_str());
            return GAHHG_ERR_CAPACITY;
        }
        GAHHG_TRY(b.words.alloc(b.nn, s));
        GAHHG_TRY(b.rnode.alloc(b.sums.refined, s));
        GAHHG_TRY(b.lnode.alloc(b.sums.leaves, s));
        k_encode<<<blocks_for(b.nn), TPB, 0, s>>>(view(lvl), d_pg.ptr, (int)gnext, leaf_base[lvl], b.words.ptr,
                                                  b.rnode.ptr, b.lnode.ptr);
        return GAHHG_OK;
    };
    for (int lvl = 0;; lvl++) {
        LevelBuf& b = lv[lvl];
        if (lvl > 0) {
            // this level's lists and labels from the level above
            LevelBuf& up = lv[lvl - 1];
            const LevelView uv = view(lvl - 1);
            const int nref = up.sums.refined;
            GAHHG_TRY(b.list.alloc(b.sums.pairs, s));
            GAHHG_TRY(b.label.alloc(b.nn, s));
            k_child_fill<<<(nref + TPB / 32 - 1) / (TPB / 32), TPB, 0, s>>>(uv, up.rnode.ptr, nref, up.hit.ptr,
                                                                            b.cnt.ptr, b.off.ptr, b.cpar.ptr,
                                                                            b.list.ptr, b.label.ptr);
            k_child_exact<<<blocks_for(b.nn), TPB, 0, s>>>(ends, uv, d_pg.ptr, up.rnode.ptr, b.nn, b.ixy.ptr, b.cnt.ptr,
                                                           b.off.ptr, b.list.ptr, b.cpar.ptr, b.label.ptr, bad);
        }
        GAHHG_TRY(encode(lvl));
        const int nref = b.sums.refined;
        if (nref == 0) break;
        // the children: rectangles, pair tests, counts
        lv.emplace_back();
        LevelBuf& c = lv[lvl + 1];
        c.nn = nref * FAN * FAN;
        c.gstart = (int)gnext;
        gnext += c.nn;
        DevArray<int> longs;
        GAHHG_TRY(c.ixy.alloc(c.nn, s));
        if (np > 1) GAHHG_TRY(c.poly.alloc(c.nn, s));
        GAHHG_TRY(c.cnt.alloc(c.nn, s));
        GAHHG_TRY(c.cpar.alloc(c.nn, s));
        GAHHG_TRY(longs.alloc((size_t)b.sums.pairs / (PAIR_LONG + 1) + 1, s));
        GAHHG_TRY(b.hit.alloc(b.sums.pairs, s));
        GAHHG_CUDA_TRY(cudaMemsetAsync(w->sort, 0, sizeof w->sort, s));
        const PairArgs a{ends, d_pg.ptr, b.rnode.ptr, nref, c.ixy.ptr, c.poly.ptr, b.hit.ptr, c.cnt.ptr,
                         c.cpar.ptr, longs.ptr, w->sort};
        k_child_pairs<<<(c.nn + PAIR_TPB - 1) / PAIR_TPB, PAIR_TPB, 0, s>>>(a, view(lvl));
        k_child_pairs_long<<<sms * 2, TPB, 0, s>>>(a, view(lvl));
        GAHHG_CUDA_TRY(cudaGetLastError());
        GAHHG_TRY(scan(lvl + 1, gnext));
        if (too_long(lvl + 1)) {
            // edges closer to one another than the cells' margin: every child
            // lists nearly all of them, however small (8 entries and more for
            // one).  This level's cells stay leaves, as past the budgets.
            gnext -= c.nn;
            lv.pop_back();
            leaf_total = leaf_base.back();
            rec_total = rec_base.back();
            leaf_base.pop_back();
            rec_base.pop_back();
            GAHHG_TRY(scan_once(lvl, true));
            GAHHG_TRY(encode(lvl));
            break;
        }
    }
    const int nlev = (int)lv.size();
    L->nnodes = gnext;
    L->nleaves = leaf_total;
    L->nrecs = rec_total;
    phase("levels");

    // ---- the index: node words of all levels, leaves, records, summaries
    GAHHG_TRY(L->nodes.alloc(gnext, s));
    // one spare leaf: the grouped pass 2 copies leaf records in 16-byte units
    GAHHG_TRY(L->leaves.alloc(leaf_total + 1, s));
    GAHHG_TRY(L->recs.alloc(rec_total, s));
    GAHHG_TRY(L->eids.alloc(rec_total, s));
    GAHHG_TRY(L->aux.alloc(leaf_total, s));
    for (int lvl = 0; lvl < nlev; lvl++) {
        const LevelBuf& b = lv[lvl];
        GAHHG_CUDA_TRY(cudaMemcpyAsync(L->nodes.ptr + b.gstart, b.words.ptr, sizeof(uint32_t) * b.nn,
                                       cudaMemcpyDeviceToDevice, s));
        if (b.sums.leaves > 0)
            k_leaf_records<<<blocks_for(b.sums.leaves), TPB, 0, s>>>(ends, view(lvl), d_pg.ptr, b.lnode.ptr,
                                                                     b.sums.leaves, leaf_base[lvl], rec_base[lvl],
                                                                     L->leaves.ptr, L->recs.ptr, L->eids.ptr,
                                                                     L->aux.ptr, bad);
    }
    // coarse summaries, each polygon's from a 16-byte aligned word
    std::vector<long long> sc(np + 1, 0), soff(np + 1, 0);
    std::vector<int> cshift(np), SW(np), SH(np);
    L->swords.resize(np);
    for (int p = 0; p < np; p++) {
        summary_shape(pg[p].g.W, pg[p].g.H, &cshift[p], &SW[p], &SH[p]);
        L->swords[p] = (SW[p] * SH[p] + 15) / 16;
        sc[p + 1] = sc[p] + (long long)SW[p] * SH[p];
        soff[p + 1] = soff[p] + ((L->swords[p] + 3) & ~3);
    }
    {
        DevArray<long long> d_sc, d_soff;
        DevArray<int> d_cshift;
        GAHHG_TRY(upload(d_sc, sc, s));
        GAHHG_TRY(upload(d_soff, soff, s));
        GAHHG_TRY(upload(d_cshift, cshift, s));
        // (a bulk copy of a summary reads up to its 16-byte multiple, inside soff's padding)
        GAHHG_TRY(alloc_zero(L->summary, soff[np], s));
        k_summary<<<blocks_for(4 * sc[np]), TPB, 0, s>>>(L->nodes.ptr, d_pg.ptr, d_sc.ptr, d_cshift.ptr, d_soff.ptr, np,
                                                         outl.ptr, L->summary.ptr);
    }
    GAHHG_CUDA_TRY(cudaGetLastError());
    // ---- the last round trip: failures, origins, outside labels
    BuildWords hw;
    std::vector<int> h_origin(np);
    std::vector<uint8_t> h_out(np);
    GAHHG_CUDA_TRY(cudaMemcpyAsync(&hw, w, sizeof hw, cudaMemcpyDeviceToHost, s));
    GAHHG_CUDA_TRY(cudaMemcpyAsync(h_origin.data(), origin.ptr, sizeof(int) * np, cudaMemcpyDeviceToHost, s));
    GAHHG_CUDA_TRY(cudaMemcpyAsync(h_out.data(), outl.ptr, np, cudaMemcpyDeviceToHost, s));
    GAHHG_CUDA_TRY(cudaStreamSynchronize(s));
    phase("index");
    for (const LevelBuf& b : lv) L->scratch_bytes += (long long)b.bytes();
    for (int p = 0; p < np; p++) {
        const std::string who = prefix.empty() ? "exact index: " : prefix + "polygon " + std::to_string(p) + ": ";
        if (h_origin[p] == 0) {
            set_error("%sno outer-ring edge gives a reference point", who.c_str());
            return GAHHG_ERR_STATE;
        }
        if (h_origin[p] < 0) {
            set_error("%sa hub or the origin center coincides with a polygon vertex", who.c_str());
            return GAHHG_ERR_STATE;
        }
    }
    // a scan whose look-back ran out of time summed the late tile's counts
    // itself: its result is exact, the event is only counted
    g->stats.scan_fallbacks = hw.err.scan_lookback_timeout;
    if (hw.bad[0] || hw.bad[1]) {
        set_error("%s%d center/vertex coincidences, %d oversize leaves",
                  prefix.empty() ? "exact index: " : prefix.c_str(), hw.bad[0], hw.bad[1]);
        return GAHHG_ERR_DEVICE;
    }
    // ---- every polygon's query view
    L->views.resize(np);
    for (int p = 0; p < np; p++) {
        QueryView& Q = L->views[p];
        memset(&Q, 0, sizeof Q);
        set_view_geo(Q, pg[p].g);
        Q.outside = KIND_PURE | (uint32_t)h_out[p];
        Q.nodes = L->nodes.ptr + pg[p].top;
        Q.leaves = L->leaves.ptr;
        Q.recs = L->recs.ptr;
        Q.eids = L->eids.ptr;
        Q.ends = L->ends.ptr;
        Q.aux = L->aux.ptr;
        set_view_coarse(Q, pg[p].g, cshift[p], SW[p], SH[p]);
        Q.swords = L->swords[p];
        Q.summary = L->summary.ptr + soff[p];
        Q.nparts = 1;  // leaf windows: single-polygon queries set them
        Q.part_scale = 0.0f;
    }
    return GAHHG_OK;
}

}  // namespace

// The exact index of g's polygon, from the polygon's device copies.
gahhg_status lattice_build(Grid* g)
{
    LatticeSet* L = new LatticeSet();
    g->lattice = L;
    Polygon* P = const_cast<Polygon*>(g->poly);
    const int top = g->opts.lattice_top, leaf = g->opts.lattice_leaf;
    Builder b;
    b.L = L;
    GAHHG_TRY(b.run(g, &P, 1, &top, &leaf, P->d_pv, P->d_pe));
    set_leaf_windows(L->views[0], L->nleaves, L->nrecs);
    return GAHHG_OK;
}

// Exact indexes of polys[0 .. count) built together on g's stream (g lends
// the device, the stream and the scan state).
gahhg_status lattice_build_group(Grid* g, Polygon* const* polys, int count, const int* top_cells,
                                 const int* leaf_edges, LatticeSet** out)
{
    LatticeSet* L = new LatticeSet();
    *out = L;
    Builder b;
    b.L = L;
    b.prefix = "exact index group: ";
    return b.run(g, polys, count, top_cells, leaf_edges, nullptr, nullptr);
}

void lattice_free(LatticeSet* L)
{
    if (!L) return;
    L->release();
    delete L;
}

size_t lattice_bytes(const LatticeSet* L) { return L ? (size_t)L->bytes() : 0; }
size_t lattice_device_bytes(const LatticeSet* L) { return L ? (size_t)L->device_bytes() : 0; }
long long lattice_scratch_bytes(const LatticeSet* L) { return L ? L->scratch_bytes : 0; }
void lattice_view_write(const LatticeSet* L, int i, void* dst) { memcpy(dst, &L->views[i], sizeof(QueryView)); }
long long lattice_summary_words(const LatticeSet* L, int i) { return L ? L->swords[i] : 0; }

}  // namespace gahhg
