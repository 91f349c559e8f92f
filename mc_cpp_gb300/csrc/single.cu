// Single-system engine: the device side of FField_CUDA.
//
// Data layout in HBM (one system, n atoms):
//   pq[n]        double4_32a (x, y, z, q)      FP64 master coordinates + charge (32 B, aligned loads)
//   es[n]        double2 (eps, sig)        sqrt(eps*418.4) and MDBAS half-sigma
//   es14[n]      double2 (eps14, sig14)
//   fx[n]        uint4 (fx, fy, fz, parameter class)  fixed-point mirror for the mixed kernels
//   cls_of[n], cls[ncls]  parameter class of each atom and the classes' (q hi, q lo, eps, sig)
//   x64[n]       ulonglong4 (x, y, z as box fractions in 2^-64, class), FP64 periodic systems
//   pair64[ncls^2]   the class pairs' parameter products (fixed64.hpp)
//   esf[n]       float2 (eps, sig)
//   nbr[n*cap]   int   Verlet rows: partners j > i from the front, j < i from the back
//   nup[n], nlo[n]
//   cell_*       cell list of the last build
//   exclusion CSR (stored rows, and the full-mode effective rows), 1-4 pairs and per-atom 1-4 CSR
//   part[]       FP64 per-block partial sums (scratch), reduced in a fixed order by one block
//
// Kernels (all launched on the handle's stream):
//   k_cell_assign / k_cell_scan / k_cell_scatter / k_cell_sort / k_build_rows   Verlet build
//   k_energy_list<P>   switch energy over the half list (warp per row)        FField_MDBAS.cpp:336-424
//   k_energy_list64    the same in FP64 for periodic boxes, on 64-bit integer pair terms
//   k_energy_all*      full energy over all pairs (triangle of tiles)         FField_MDBAS.cpp:194-265
//   k_energy_all64     the same in FP64 for periodic boxes, on 64-bit integer pair terms
//   k_energy_tail<P>   1-4 pairs                                               FField_MDBAS.cpp:267-318,426-488
//                      bonds, Urey-Bradley, angles, dihedrals, impropers       FField_MDBAS.cpp:490-786
//                      and the fixed-order reduction of all partials into ener[10]
//   k_delta_e<P>       energy change of a moved atom set, one launch
//   k_commit           write accepted coordinates
#include <algorithm>
#include <array>
#include <climits>
#include <map>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "engine.hpp"
#include "fixed64.cuh"
#include "pair_math.cuh"
#include "single.hpp"

namespace mcg {

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) return fail(MCG_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

constexpr int NB_BLOCKS = 152 * 4;   // grid of the list-driven kernels: 4 CTAs per SM
constexpr int NB_THREADS = 256;
// largest grid of the bonded terms: a term per thread up to 155,648.  One, two and four CTAs per SM, us of a mixed energy:
// 100,002 water atoms 122, 115, 111; 36,000 64, 64, 63; 1,800 to 18,000 the same, and so FP64 (568, 568, 569 at 100,002)
constexpr int BD_BLOCKS = 152 * 4;
constexpr int MAX_MOVED = 1024;
constexpr int SORT_MAX = 2048;       // cells larger than this are sorted by one thread
constexpr int CLS_MAX = 1024;        // parameter classes the mixed pair kernel keeps in shared memory
// parameter classes whose pairs the FP64 kernel's table holds: 512 KB of products at 128, which stay in
// L2 with a few rows of the matrix in L1; a system of more classes forms them per pair (5 FP64 operations)
// (100,002 water atoms: 0.555 ms with 2 to 128 classes in the table, 0.647 formed per pair)
constexpr int CLS64_MAX = 128;

enum { PREC_F64 = 0, PREC_MIX = 1 };

// ------------------------------------------------------------------------------------------
// Verlet list build with a cell grid (replaces the O(N^2) List_nonBonded::update_verlet_list,
// List_nonBonded.cpp:836-915; same acceptance rule: r^2 <= (rc + skin)^2 in the reference's FP64
// arithmetic, not both frozen, not in the stored exclusion row of the lower index).
// Cells at least half the list radius wide: a neighbour within the radius lies within two cells
// along each axis, so an atom scans up to 5 x 5 x 5 cells (a whole axis when it has fewer than 5).
struct Grid {
    int nc[3];
    double lo[3], inv[3];   // PBC none: bounding-box origin and 1 / extent
    float csf[3];           // cell widths, rounded down
    int periodic;
};

// The five kernels of a list build follow each other as programmatic dependents, so a kernel's CTAs are
// placed while the one before it runs and begin at its end; each touches memory only behind this.  With
// that, the counters zeroed by the scan instead of two memsets, and the longest row written to mapped
// memory by the last CTA instead of a copy, a whole update takes 33 us at 864 argon atoms (47 without),
// 51 at 1,800 water atoms (70), 135 at 12,288 (146) and 650 at 100,002 (661).
__device__ __forceinline__ void list_step() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__global__ void k_cell_assign(const double4_32a* __restrict__ pq, int n, PbcDev pbc, Grid g, int* cell_of,
                              int* cell_count) {
    list_step();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4_32a p = pq[i];
    double c[3] = {p.x, p.y, p.z};
    int idx[3];
    for (int k = 0; k < 3; k++) {
        double u;
        if (g.periodic) { u = c[k] * pbc.rL[k]; u -= floor(u); }
        else u = (c[k] - g.lo[k]) * g.inv[k];
        int v = (int)(u * g.nc[k]);
        idx[k] = min(max(v, 0), g.nc[k] - 1);
    }
    int cell = (idx[2] * g.nc[1] + idx[1]) * g.nc[0] + idx[0];
    cell_of[i] = cell;
    atomicAdd(&cell_count[cell], 1);
}

// Exclusive scans by one block (cells are few) of the cell counts and of the cells' row-build tasks
// (runs of at most `run` home atoms), carried together in the halves of a 64-bit sum.  The counts are zero
// again afterwards, for the next build, and so are the row build's counters (max_row).
__global__ void k_cell_scan(int* cell_count, int ncell, int run, int* cell_start, int* cell_fill, int* task_start, int* max_row) {
    __shared__ unsigned long long sw[32];
    list_step();
    if (threadIdx.x < 3) max_row[threadIdx.x] = 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (int base = 0; base < ncell; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const unsigned v = i < ncell ? (unsigned)cell_count[i] : 0u;
        const unsigned long long own = (unsigned long long)((v + run - 1) / run) << 32 | v;
        unsigned long long s = own;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += up;
        }
        if (lane == 31) sw[w] = s;
        __syncthreads();
        if (w == 0) {
            unsigned long long t = sw[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long up = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += up;
            }
            sw[lane] = t;
        }
        __syncthreads();
        const unsigned long long at = carry + (w ? sw[w - 1] : 0ull) + s - own;
        if (i < ncell) { cell_start[i] = (int)(unsigned)at; cell_fill[i] = 0; cell_count[i] = 0; task_start[i] = (int)(at >> 32); }
        carry += sw[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) { cell_start[ncell] = (int)(unsigned)carry; task_start[ncell] = (int)(carry >> 32); }
}

__global__ void k_cell_scatter(const int* __restrict__ cell_of, int n, const int* __restrict__ cell_start,
                               int* cell_fill, int* cell_atoms) {
    list_step();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = cell_of[i];
    int slot = atomicAdd(&cell_fill[c], 1);
    cell_atoms[cell_start[c] + slot] = i;
}

// Sort each cell's atoms ascending so rows come out in a deterministic order, and write the cell's
// share of the candidates in cell order (fixed-point position, atom index), of the home atoms grouped by
// the octant of the cell they lie in (places in cell order), and of the row build's tasks: runs of at
// most `run` of these.  The grouping only decides which rows are built together.
__global__ void k_cell_sort(const int* __restrict__ cell_start, const int* __restrict__ task_start, int ncell, int run,
                            const uint4* __restrict__ fx, const double4_32a* __restrict__ pq, Grid g, int* cell_atoms, uint4* cell_pos,
                            int* home, int2* tasks) {
    __shared__ int sh[SORT_MAX];
    __shared__ uint8_t oct[SORT_MAX];
    int c = blockIdx.x;
    if (c >= ncell) return;
    list_step();
    int b = cell_start[c], e = cell_start[c + 1], m = e - b;
    for (int k = threadIdx.x; k * run < m; k += blockDim.x) tasks[task_start[c] + k] = make_int2(c, b + k * run);
    if (m > SORT_MAX) {
        if (threadIdx.x == 0)
            for (int i = b + 1; i < e; i++) {
                int v = cell_atoms[i], k = i - 1;
                while (k >= b && cell_atoms[k] > v) { cell_atoms[k + 1] = cell_atoms[k]; k--; }
                cell_atoms[k + 1] = v;
            }
        __syncthreads();
    } else if (m > 1) {
        int m2 = 1;
        while (m2 < m) m2 <<= 1;
        for (int i = threadIdx.x; i < m2; i += blockDim.x) sh[i] = i < m ? cell_atoms[b + i] : 0x7fffffff;
        __syncthreads();
        for (int k = 2; k <= m2; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = threadIdx.x; i < m2; i += blockDim.x) {
                    int l = i ^ j;
                    if (l > i) {
                        bool up = (i & k) == 0;
                        int a = sh[i], bb = sh[l];
                        if ((a > bb) == up) { sh[i] = bb; sh[l] = a; }
                    }
                }
                __syncthreads();
            }
        for (int i = threadIdx.x; i < m; i += blockDim.x) cell_atoms[b + i] = sh[i];
        __syncthreads();
    }
    for (int i = b + threadIdx.x; i < e; i += blockDim.x) {
        const int a = cell_atoms[i];
        uint4 p = fx[a];       // box fractions; without a box, FP32 distances from the atoms' lowest coordinates
        unsigned hx, hy, hz;   // the half of the cell along each axis
        if (g.periodic) {
            hx = (unsigned)((unsigned long long)p.x * (2 * g.nc[0]) >> 32);
            hy = (unsigned)((unsigned long long)p.y * (2 * g.nc[1]) >> 32);
            hz = (unsigned)((unsigned long long)p.z * (2 * g.nc[2]) >> 32);
        } else {
            const double4_32a q = pq[a];
            const float x = (float)(q.x - g.lo[0]), y = (float)(q.y - g.lo[1]), z = (float)(q.z - g.lo[2]);
            p = make_uint4(__float_as_uint(x), __float_as_uint(y), __float_as_uint(z), 0u);
            hx = (unsigned)(x * (float)g.inv[0] * (float)(2 * g.nc[0]));
            hy = (unsigned)(y * (float)g.inv[1] * (float)(2 * g.nc[1]));
            hz = (unsigned)(z * (float)g.inv[2] * (float)(2 * g.nc[2]));
        }
        p.w = (unsigned)a;
        cell_pos[i] = p;
        if (m <= SORT_MAX) {
            hx &= 1u; hy &= 1u; hz &= 1u;
            oct[i - b] = (uint8_t)(hz << 2 | hy << 1 | (hx ^ hy));   // neighbouring octants share a face
        } else {
            home[i] = i;
        }
    }
    if (m > SORT_MAX) return;
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int o = oct[i];
        int r = 0;
        for (int k = 0; k < m; k++) r += oct[k] < o || (oct[k] == o && k < i);
        home[b + r] = b + i;
    }
}

constexpr double LIST_EXTENT = 20.0;

struct ListParams {
    double cutnb2;
    int cap;
    int maxspan;
    // FP32 prefilter.  A pair whose FP32 r^2 lies below lo2 is inside, above hi2 outside; only the band between
    // takes the reference's FP64 test.  (A^2, or units of (L 2^-32)^2 in boxes of equal lengths.)  Without a box the
    // candidates hold FP32 coordinates, off by 2^-25 of the atoms' extent: up to an extent of LIST_EXTENT list radii
    // that moves a distance by 2e-6 of the radius, inside the margins; atoms spread farther are all in the band.
    float Ls[3];            // length of a unit of the candidates' coordinates (1 without a box)
    float lo2, hi2;
    float reach2;   // rows of cells farther than this (squared, with a margin) are not scanned
    int any_frozen;
};

__device__ __forceinline__ bool stored_excluded(int lo, int hi, const int* __restrict__ xs,
                                                const int* __restrict__ xd, int maxspan) {
    if (hi - lo > maxspan) return false;
    int b = xs[lo], e = xs[lo + 1];
    for (int k = b; k < e; k++) if (xd[k] == hi) return true;
    return false;
}

// A warp per task: up to A home atoms of one cell share the walk over the stencil's candidates, which
// lie in cell order (coalesced 16-byte loads, no index gather), 32 at a time.  The stencil's rows of
// cells become ranges of the candidates, dropped or trimmed where no home atom reaches; the ranges are
// walked as one sequence, the end of one with the beginning of the next, and the next 64 candidates load
// while these are tested.  A row lists its
// partners in the candidates' order, whatever the grouping.  A pair is first placed by its FP32 distance, in
// periodic boxes from the exact fixed-point mirrors (error ~2e-7 of (rc + skin)^2), without a box from FP32
// coordinates (at most 5e-6 of it, ListParams); the reference's FP64 distance decides only the pairs within
// 1e-4 of the list radius, so the rows are the reference's sets.
// Before the home atoms' tests the candidates pass one against the sphere around all of them, and the
// survivors (1,750 of 3,200 for four atoms of one octant of a water cell, 1,150 end in a row) are
// gathered in a ring, 32 at a time.  Bound by issue.  (One atom per warp with an index gather in front
// of every candidate took 1.48 ms on the 100,002-atom water box and 188 us at 12,288 atoms.  Two candidates
// per lane in the walk, and tasks from a counter instead of a third wave of CTAs, took a whole update of
// the former from 754 to 653 us.  Without a box, where every candidate took the FP64 test: 36,000 water atoms
// 1756 us, 299 with the FP32 coordinates.)
constexpr int ROW_WARPS = 4;
// CTAs of four warps launched per SM: what is resident with two home atoms (72 registers).  With four (96 registers) five
// are, and two start as others end: whole updates 136 us against 158 with five at 12,288 atoms, 274 against 280 at
// 36,000, 649 against 645 at 100,002.
constexpr int ROW_CTAS = 7;
constexpr int ROW_RING = 128;  // up to 63 pending candidates and 64 new ones

// The pairs the FP32 test does not decide: in the band around the list radius, or close in index (the atom
// itself, or perhaps excluded).
__device__ __noinline__ bool row_pair(const double4_32a* __restrict__ pq, const PbcDev& pbc, const ListParams& lp, const int* __restrict__ xs, const int* __restrict__ xd, int i, int j,
                                      bool exact) {
    if (j == i) return false;
    if (exact) {
        const double4_32a pi = pq[i], pj = pq[j];
        if (!(ref64_dist2(pi.x, pi.y, pi.z, pj.x, pj.y, pj.z, pbc) <= lp.cutnb2)) return false;
    }
    return !stored_excluded(min(i, j), max(i, j), xs, xd, lp.maxspan);
}

// a predicated store: the branch around an ordinary one costs more than the store
__device__ __forceinline__ void store_if(int* p, int v, bool pred) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.global.s32 [%0], %1;\n}" ::"l"(p), "r"(v), "r"((int)pred) : "memory");
}

template <int A, bool PERIODIC, bool ISO>
__global__ void __launch_bounds__(32 * ROW_WARPS) k_build_rows(const double4_32a* __restrict__ pq, const uint4* __restrict__ cell_pos,
                                                               const uint8_t* __restrict__ frozen, PbcDev pbc, Grid g,
                                                               ListParams lp, const int* __restrict__ cell_start,
                                                               const int* __restrict__ task_start, int ncell,
                                                               const int* __restrict__ home, const int2* __restrict__ tasks,
                                                               const int* __restrict__ xs,
                                                               const int* __restrict__ xd, int* nbr, int* nup, int* nlo,
                                                               int* max_row, int* longest_row) {
    __shared__ int2 s_range[ROW_WARPS][66];
    __shared__ uint4 s_ring[ROW_WARPS][ROW_RING];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    int2* range = s_range[wib];
    uint4* ring = s_ring[wib];
    list_step();
    const int ntask = task_start[ncell];
    const unsigned span2 = 2u * (unsigned)lp.maxspan;   // partners within maxspan in index are looked at
    int longest = 0;
    // the first task by the warp's place, the others from a counter (max_row[1]), each fetched while the one
    // before it is worked on: a grid of what is resident at once, without a last wave
    int task = blockIdx.x * ROW_WARPS + wib, after = 0;
    for (; task < ntask; task = __shfl_sync(0xffffffffu, after, 0)) {
        if (lane == 0) after = gridDim.x * ROW_WARPS + atomicAdd(max_row + 1, 1);
        const int2 tk = tasks[task];
        const int c = tk.x, m = min(A, cell_start[c + 1] - tk.y);
        const int ctr[3] = {c % g.nc[0], (c / g.nc[0]) % g.nc[1], c / (g.nc[0] * g.nc[1])};
        // the home atoms: candidate entries tk.y .. tk.y + m; a missing one repeats the first and is not stored
        uint32_t hx[A][3];
        int hi[A], up[A], back[A], first[A];
        int* row[A];
        unsigned fixed = 0;              // the frozen ones among them
#pragma unroll
        for (int k = 0; k < A; k++) {
            const uint4 p = cell_pos[home[tk.y + (k < m ? k : 0)]];
            hx[k][0] = p.x; hx[k][1] = p.y; hx[k][2] = p.z;
            hi[k] = (int)p.w;
            first[k] = hi[k] - lp.maxspan;
            up[k] = 0;
            back[k] = lp.cap - 1;
            row[k] = nbr + (size_t)p.w * lp.cap;
            if (lp.any_frozen) fixed |= (unsigned)(frozen[p.w] != 0) << k;
        }
        // per axis: the offsets scanned, and the home atoms' extent inside the cell (in cell widths) for
        // the distance from them to a cell d away along that axis.  FP32 throughout (FP64 here, at
        // GB300's FP64 rate, had cost more than the candidate tests): off by ~1e-6 cell widths, inside
        // the margin of lp.reach2.
        int dlo[3], dhi[3];
        bool whole[3];
        float pmin[3], pmax[3], ball2 = 0.f;
        uint32_t ball[3] = {0, 0, 0};
        {
            const uint4 q = cell_pos[home[tk.y + min(lane, m - 1)]];
            const uint32_t q3[3] = {q.x, q.y, q.z};
            double d3[3] = {0, 0, 0};
            if (!PERIODIC) { const double4_32a d = pq[q.w]; d3[0] = d.x; d3[1] = d.y; d3[2] = d.z; }
            for (int k = 0; k < 3; k++) {
                float p;
                if (PERIODIC) {   // the mirror holds the box fraction in units of 2^-32
                    p = (float)q3[k] * 2.3283064365386963e-10f * (float)g.nc[k] - (float)ctr[k];
                    if (p < -0.5f * g.nc[k]) p += (float)g.nc[k];       // fraction just below 1, stored as 0
                    else if (p > 0.5f * g.nc[k]) p -= (float)g.nc[k];
                } else {
                    p = (float)((d3[k] - g.lo[k]) * g.inv[k]) * (float)g.nc[k] - (float)ctr[k];
                }
                p = fminf(fmaxf(p, 0.f), 1.f);       // non-negative floats order as their bits
                pmin[k] = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(p)));
                pmax[k] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(p)));
                whole[k] = PERIODIC && g.nc[k] < 5;
                if (whole[k]) { dlo[k] = -ctr[k]; dhi[k] = g.nc[k] - 1 - ctr[k]; }
                else if (PERIODIC) { dlo[k] = -2; dhi[k] = 2; }
                else { dlo[k] = max(-2, -ctr[k]); dhi[k] = min(2, g.nc[k] - 1 - ctr[k]); }
            }
            // the sphere around the home atoms: the middle of their extent, and its radius
            float far2 = 0.f;
            for (int k = 0; k < 3; k++) {
                float e;
                if (PERIODIC) {
                    const int d = (int)(q3[k] - hx[0][k]);
                    const int mn = __reduce_min_sync(0xffffffffu, d), mx = __reduce_max_sync(0xffffffffu, d);
                    const int mid = mn + (int)((unsigned)(mx - mn) >> 1);
                    ball[k] = hx[0][k] + (uint32_t)mid;
                    e = (float)(d - mid) * lp.Ls[k];
                } else {
                    const float mn = __uint_as_float(__reduce_min_sync(0xffffffffu, q3[k])),
                                mx = __uint_as_float(__reduce_max_sync(0xffffffffu, q3[k])), mid = 0.5f * (mn + mx);
                    ball[k] = __float_as_uint(mid);
                    e = __uint_as_float(q3[k]) - mid;
                }
                far2 = fmaf(e, e, far2);
            }
            far2 = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(far2)));
            const float reach = sqrtf(lp.reach2) + sqrtf(far2);
            ball2 = lp.lo2 < 0.f ? lp.hi2 : reach * reach;
        }
        auto gap2 = [&](int k, int d) -> float {   // squared lower bound on |displacement| along axis k
            if (whole[k] || d == 0) return 0.f;
            const float w = (d > 0 ? (float)(d - 1) + (1.f - pmax[k]) : (float)(-d - 1) + pmin[k]) * g.csf[k];
            return w * w;
        };
        // the stencil's rows of cells along x (at most 5 x 5), one per lane, z outer and y inner: each
        // becomes one or two ranges of candidates, the wrapped part of a row first
        const int ny = dhi[1] - dlo[1] + 1, nrow = ny * (dhi[2] - dlo[2] + 1);
        int rb0 = 0, re0 = 0, rb1 = 0, re1 = 0;
        if (lane < nrow) {
            const int dy = dlo[1] + lane % ny, dz = dlo[2] + lane / ny;
            const float left = lp.reach2 - gap2(2, dz) - gap2(1, dy);
            if (left >= 0.f) {
                int x0 = dlo[0], x1 = dhi[0];
                while (x0 < 0 && gap2(0, x0) > left) x0++;
                while (x1 > 0 && gap2(0, x1) > left) x1--;
                int y = ctr[1] + dy, z = ctr[2] + dz;
                if (PERIODIC) { y = (y + g.nc[1]) % g.nc[1]; z = (z + g.nc[2]) % g.nc[2]; }
                const int rowc = (z * g.nc[1] + y) * g.nc[0];
                int a0 = ctr[0] + x0, a1 = ctr[0] + x1;   // both wrap only on a whole axis, which has none
                if (a0 < 0) { rb1 = cell_start[rowc + a0 + g.nc[0]]; re1 = cell_start[rowc + g.nc[0]]; a0 = 0; }
                if (a1 >= g.nc[0]) { rb1 = cell_start[rowc]; re1 = cell_start[rowc + a1 - g.nc[0] + 1]; a1 = g.nc[0] - 1; }
                rb0 = cell_start[rowc + a0];
                re0 = cell_start[rowc + a1 + 1];
            }
        }
        // the non-empty ranges in order; a walk over them takes 64 candidates at a time, two per lane, the
        // end of one range together with the beginning of the next
        const unsigned b1 = __ballot_sync(0xffffffffu, re1 > rb1), b0 = __ballot_sync(0xffffffffu, re0 > rb0);
        const int nrange = __popc(b1) + __popc(b0);
        __syncwarp();
        if (re1 > rb1) range[__popc(b1 & below) + __popc(b0 & below)] = make_int2(rb1, re1);
        if (re0 > rb0) range[__popc(b1 & (below << 1 | 1u)) + __popc(b0 & below)] = make_int2(rb0, re0);
        if (lane < 2) range[nrange + lane] = make_int2(0, 0);
        __syncwarp();
        constexpr uint32_t NONE = 0xffffffffu;
        int rg = 0;
        int2 cur = range[0], nxt = range[1];
        auto fetch = [&](uint4& c0, uint4& c1) {
            const int rem = cur.y - cur.x, skip = nxt.x - rem;   // at least 1 until the walk's end
            const int l1 = lane + 32;
            const int at0 = lane < rem ? cur.x + lane : skip + lane, at1 = l1 < rem ? cur.x + l1 : skip + l1;
            c0.w = c1.w = NONE;
            if (lane < rem || at0 < nxt.y) c0 = cell_pos[at0];
            if (l1 < rem || at1 < nxt.y) c1 = cell_pos[at1];
            if (rem > 64) {
                cur.x += 64;
            } else {
                cur = make_int2(min(skip + 64, nxt.y), nxt.y);
                rg++;
                nxt = range[min(rg + 1, nrange)];
                if (cur.x == cur.y && rg < nrange) {             // the next range was used up whole
                    cur = nxt;
                    rg++;
                    nxt = range[min(rg + 1, nrange)];
                }
            }
        };
        bool more = rg < nrange;
        uint4 n0 = make_uint4(0, 0, 0, NONE), n1 = n0;
        fetch(n0, n1);
        int head = 0, tail = 0;            // candidates within reach of the home atoms, pending in the ring
        // difference of two coordinates in the candidates' unit
        auto diff = [](uint32_t c, uint32_t h) {
            return PERIODIC ? __int2float_rn((int)(c - h)) : __uint_as_float(c) - __uint_as_float(h);
        };
        auto within = [&](const uint4& c) {
            const float dx = diff(c.x, ball[0]) * lp.Ls[0], dy = diff(c.y, ball[1]) * lp.Ls[1], dz = diff(c.z, ball[2]) * lp.Ls[2];
            return c.w != NONE && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= ball2;
        };
        while (more || head != tail) {
            if (more && head - tail < 64) {
                const uint4 c0 = n0, c1 = n1;
                more = rg < nrange;
                if (more) fetch(n0, n1);
                const bool in0 = within(c0), in1 = within(c1);
                const unsigned m0 = __ballot_sync(0xffffffffu, in0), m1 = __ballot_sync(0xffffffffu, in1);
                const int h1 = head + __popc(m0);
                if (in0) ring[(head + __popc(m0 & below)) & (ROW_RING - 1)] = c0;
                if (in1) ring[(h1 + __popc(m1 & below)) & (ROW_RING - 1)] = c1;
                head = h1 + __popc(m1);
                __syncwarp();
                if (more && head - tail < 32) continue;
            }
            uint4 cd = make_uint4(0, 0, 0, 0xffffffffu);
            if (lane < head - tail) cd = ring[(tail + lane) & (ROW_RING - 1)];
            tail = min(tail + 32, head);
            __syncwarp();
            const int j = (int)cd.w;      // -1 past the end
            // bit k: the candidate is in home atom k's row; close to it in index; in the band (one branch
            // for all that have to be looked at)
            unsigned in = 0, look = 0, band = 0;
            const float lo2 = j >= 0 ? lp.lo2 : -1.0f, hi2 = j >= 0 ? lp.hi2 : -1.0f;
#pragma unroll
            for (int k = 0; k < A; k++) {
                const float ux = diff(cd.x, hx[k][0]), uy = diff(cd.y, hx[k][1]), uz = diff(cd.z, hx[k][2]);
                float r2;
                if (ISO) {
                    r2 = fmaf(ux, ux, fmaf(uy, uy, uz * uz));   // in units of (L 2^-32)^2 in a box, as lo2 and hi2
                } else {
                    const float dx = ux * lp.Ls[0], dy = uy * lp.Ls[1], dz = uz * lp.Ls[2];
                    r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                }
                const unsigned near = r2 <= hi2 ? 1u << k : 0u;
                in |= near;
                band |= r2 < lo2 ? 0u : near;
                look |= (unsigned)(j - first[k]) <= span2 ? near : 0u;
            }
            // two frozen atoms are no pair: a look at the candidate's flag, once for all home atoms
            if (fixed && in && frozen[j]) { in &= ~fixed; look &= ~fixed; band &= ~fixed; }
            if (look | band) {
                for (unsigned l = look | band; l; l &= l - 1) {
                    const int k = __ffs(l) - 1;
                    int i = hi[0];
#pragma unroll
                    for (int q = 1; q < A; q++) if (k == q) i = hi[q];
                    if (!row_pair(pq, pbc, lp, xs, xd, i, j, band >> k & 1u)) in &= ~(1u << k);
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < A; k++) {
                const bool mine = in >> k & 1u, above = j > hi[k];
                const unsigned b = __ballot_sync(0xffffffffu, mine), bu = b & __ballot_sync(0xffffffffu, above);
                const int rank = __popc((above ? bu : b ^ bu) & below), at = up[k] + rank;
                // the front of the row grows up, its back down; a row that would pass its capacity is not stored
                const int off = above ? at : back[k] - rank;
                store_if(row[k] + off, j, mine && at <= back[k]);
                up[k] += __popc(bu);
                back[k] -= __popc(b ^ bu);
            }
        }
#pragma unroll
        for (int k = 0; k < A; k++)
            if (k < m) {
                const int lo = lp.cap - 1 - back[k];
                if (lane == 0) { nup[hi[k]] = up[k]; nlo[hi[k]] = lo; }
                longest = max(longest, up[k] + lo);
            }
    }
    if (lane == 0 && longest > 0) atomicMax(max_row, longest);
    __syncthreads();
    if (threadIdx.x == 0) {   // max_row[2] counts the CTAs done
        __threadfence();
        if (atomicAdd(max_row + 2, 1) == (int)gridDim.x - 1) *longest_row = atomicMax(max_row, 0);
    }
}

// ------------------------------------------------------------------------------------------
// Energies.
struct AtomsDev {
    const double4_32a* pq;
    const double2* es;
    const double2* es14;
    const uint4* fx;
    const float2* esf;
    const float2* esf14;
    const float2* qf;     // charge as float-float (hi, lo)
    float Ls[3], Lsl[3];  // box / 2^32 as float-float (mixed displacement scale)
    ulonglong4_32a* x64;  // 64-bit box fractions and parameter class (null: no 64-bit mirror)
    const Fix64Pair* pair64;   // products of the class pairs (null: formed per pair)
    int ncls64;
};

template <int P>
__device__ __forceinline__ void pair_energy(const AtomsDev& A, const PbcDev& pbc, const CutDev& cut, bool fourteen,
                                            double4_32a pi, uint4 fi, int i, double4_32a pj, uint4 fj, int j,
                                            bool apply_cut, double& el, double& vd) {
    if (P == PREC_F64) {
        double r2 = ref64_dist2(pi.x, pi.y, pi.z, pj.x, pj.y, pj.z, pbc);
        el = 0.0; vd = 0.0;
        if (apply_cut && r2 > cut.c2) return;
        double2 a = fourteen ? A.es14[i] : A.es[i];
        double2 b = fourteen ? A.es14[j] : A.es[j];
        ref64_pair(r2, pi.w, pj.w, a.x, b.x, a.y, b.y, apply_cut, cut, el, vd);
    } else {
        float dx, dy, dz;
        if (pbc.type != 0) {
            dx = fixed_delta(fi.x, fj.x, A.Ls[0], A.Lsl[0]);
            dy = fixed_delta(fi.y, fj.y, A.Ls[1], A.Lsl[1]);
            dz = fixed_delta(fi.z, fj.z, A.Ls[2], A.Lsl[2]);
        } else {
            dx = (float)(pj.x - pi.x); dy = (float)(pj.y - pi.y); dz = (float)(pj.z - pi.z);
        }
        float r2 = dx * dx + dy * dy + dz * dz;
        el = 0.0; vd = 0.0;
        if (apply_cut && r2 > cut.c2f) return;
        float2 a = fourteen ? A.esf14[i] : A.esf[i];
        float2 b = fourteen ? A.esf14[j] : A.esf[j];
        float s = a.y + b.y;
        float2 qa = A.qf[i], qb = A.qf[j];
        float qh, ql;
        ff_mul(qa.x, qa.y, qb.x, qb.y, qh, ql);
        float e1, v1;
        mixed_pair(r2, qh, ql, a.x * b.x, s * s, apply_cut, cut, e1, v1);
        el = e1; vd = v1;
    }
}

// Switch energy over the half list: a warp per row i, lanes over its j > i entries.
template <int P>
__global__ void __launch_bounds__(NB_THREADS) k_energy_list(AtomsDev A, int n, PbcDev pbc, CutDev cut,
                                                            const int* __restrict__ nbr, const int* __restrict__ nup,
                                                            int cap, double* part) {
    pair_kernel_begin();
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    double sel = 0.0, svd = 0.0;
    for (int i = warp; i < n; i += nwarps) {
        double4_32a pi = A.pq[i];
        uint4 fi = P == PREC_MIX ? A.fx[i] : make_uint4(0, 0, 0, 0);
        const int* row = nbr + (size_t)i * cap;
        int m = nup[i];
        F32Acc fe, fv;
        for (int k = lane; k < m; k += 32) {
            int j = row[k];
            double4_32a pj = P == PREC_F64 ? A.pq[j] : make_double4_32a(0, 0, 0, 0);
            uint4 fj = P == PREC_MIX ? A.fx[j] : make_uint4(0, 0, 0, 0);
            if (P == PREC_MIX && pbc.type == 0) pj = A.pq[j];
            double el, vd;
            pair_energy<P>(A, pbc, cut, false, pi, fi, i, pj, fj, j, true, el, vd);
            if (P == PREC_F64) { sel += el; svd += vd; }
            else { fe.add((float)el); fv.add((float)vd); }
        }
        if (P == PREC_MIX) { sel += fe.value(); svd += fv.value(); }
    }
    block_reduce2(sel, svd, part + 2 * blockIdx.x);
}

// The pair's parameters (Fix64Pair): from the table of class pairs, or formed here for a system of more
// than CLS64_MAX distinct parameter sets.
template <bool TABLE>
__device__ __forceinline__ void pair64_params(const AtomsDev& A, double ileff, int i, int j, int ci, int cj, double& qq,
                                              double& ee, unsigned long long& ms, int& es) {
    if (TABLE) {
        const ulonglong4_32a p = reinterpret_cast<const ulonglong4_32a*>(A.pair64)[ci * A.ncls64 + cj];
        qq = __longlong_as_double((long long)p.x);
        ee = __longlong_as_double((long long)p.y);
        ms = p.z;
        es = (int)p.w;
    } else {
        const double2 a = A.es[i], b = A.es[j];
        const double s = (a.y + b.y) * ileff;
        qq = A.pq[i].w * A.pq[j].w;
        ee = a.x * b.x;
        if (!fix64_mantissa(s * s, ms, es)) ee = __longlong_as_double(0x7ff8000000000000ll);   // NaN
    }
}

// FP64 switch energy over the half list for periodic boxes.  Bound by the integer and FP64 pipes
// (64-76 cycles of a scheduler per FP64 warp instruction, about 22 per 64-bit product), so:
//  - a warp per row places its entries by the FP32 distance of the fixed-point mirrors: beyond
//    rc (37% of a 14 A list at 12 A) they are dropped, the others go, with their row's atom, to one
//    of two rings in shared memory, inside ron (no switch factor) or not;
//  - a ring with 32 pairs is evaluated by all lanes at once, so no lane is idle at a row's end or at
//    the cutoff, and the switch is formed only for the pairs that need it;
//  - a pair's distance and powers are 64-bit integers (fixed64.cuh), with 3 FP64 operations.
// The FP32 placement has a margin of 1e-4 in r^2; a pair placed within rc that lies beyond takes a
// switch factor of exactly 0, and one placed outside ron that lies inside a factor of 1 to 2^-56.
// The rings are drained at one place in the code, after a chunk of E64_U entries per lane: with the
// evaluation inlined behind every entry the kernel stalled on instruction fetch (0.69 against 0.61 ms on
// the 100,002-atom water box).  That box takes 0.56 ms, 64 G pairs/s (4.2 ms with the pair terms in
// FP64, 0.53 with the sigmas' powers as doubles); ncu there: issue 60%, ALU 49%, FP64 pipe 42%, the rest
// latency of the gathers.  Three entries per lane in flight against two: 0.527 and 0.532 ms.  A grid of six
// CTAs per SM instead of four, whole energies: 59 against 62 us at 6,000 atoms, 132 against 117 at 18,000,
// 226 against 217 at 36,000, 626 against 568 at 100,002.
constexpr int E64_U = 3;
constexpr int E64_RING = 128;   // up to 31 pending pairs and 32 E64_U new ones

template <bool ISO, bool TABLE>
__global__ void __launch_bounds__(NB_THREADS) k_energy_list64(AtomsDev A, Fix64Geom G, PbcDev pbc, CutDev cut, int n,
                                                              const int* __restrict__ nbr, const int* __restrict__ nup,
                                                              int cap, double* part) {
    __shared__ int2 s_ring[NB_THREADS / 32][2][E64_RING];
    pair_kernel_begin();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const unsigned below = (1u << lane) - 1u;
    const double ileff = 1.0 / G.leff;
    int2* ring = s_ring[wib][0];              // inside ron, then the switched pairs at + E64_RING
    double sel = 0.0, svd = 0.0;
    int head0 = 0, tail0 = 0, head1 = 0, tail1 = 0;   // ring positions, warp-uniform
    int i = warp, k0 = 0, m = i < n ? nup[i] : 0;
    uint4 fi = i < n ? A.fx[i] : make_uint4(0, 0, 0, 0);
    for (;;) {
        const bool last = i >= n;
        if (!last) {
            const int* row = nbr + (size_t)i * cap;
            int j[E64_U];
            float r2[E64_U];
#pragma unroll
            for (int u = 0; u < E64_U; u++) {
                const int k = k0 + u * 32 + lane;
                j[u] = k < m ? row[k] : -1;
            }
#pragma unroll
            for (int u = 0; u < E64_U; u++) {
                const uint4 fj = j[u] >= 0 ? A.fx[j[u]] : fi;
                const float dx = fixed_delta(fi.x, fj.x, G.Ls[0], G.Ll[0]), dy = fixed_delta(fi.y, fj.y, G.Ls[1], G.Ll[1]),
                            dz = fixed_delta(fi.z, fj.z, G.Ls[2], G.Ll[2]);
                r2[u] = j[u] >= 0 ? fmaf(dx, dx, fmaf(dy, dy, dz * dz)) : 3.0e38f;
            }
#pragma unroll
            for (int u = 0; u < E64_U; u++) {
                const bool in = r2[u] < G.in2, sw = !in && r2[u] <= G.out2;
                const unsigned bi = __ballot_sync(0xffffffffu, in), bs = __ballot_sync(0xffffffffu, sw);
                if (in) ring[(head0 + __popc(bi & below)) & (E64_RING - 1)] = make_int2(i, j[u]);
                if (sw) ring[E64_RING + ((head1 + __popc(bs & below)) & (E64_RING - 1))] = make_int2(i, j[u]);
                head0 += __popc(bi);
                head1 += __popc(bs);
            }
            k0 += 32 * E64_U;
            if (k0 >= m) {
                i += nwarps;
                k0 = 0;
                if (i < n) { m = nup[i]; fi = A.fx[i]; }
            }
            __syncwarp();
        }
        // full rings, and what is left of them after the last row
        const int least = last ? 1 : 32;
        for (;;) {
            const bool sw = head0 - tail0 < least;
            if (sw && head1 - tail1 < least) break;
            const int at = sw ? E64_RING + ((tail1 + lane) & (E64_RING - 1)) : (tail0 + lane) & (E64_RING - 1);
            if (lane < (sw ? head1 - tail1 : head0 - tail0)) {
                const int2 p = ring[at];
                const ulonglong4_32a a = A.x64[p.x], b = A.x64[p.y];
                const Fix64Dist u = fix64_dist2<ISO>(G, a, b);
                double ys, w, ws, qq, ee;
                unsigned long long ms;
                int es;
                pair64_params<TABLE>(A, ileff, p.x, p.y, (int)a.w, (int)b.w, qq, ee, ms, es);
                if (fix64_terms(G, u, sw, ms, es, ys, w, ws)) {
                    sel = fma(qq, ys, sel);
                    svd = fma(ee, fma(w, ws, -ws), svd);
                } else {
                    double el, vd;
                    const uint4 f0 = make_uint4(0, 0, 0, 0);
                    pair_energy<PREC_F64>(A, pbc, cut, false, A.pq[p.x], f0, p.x, A.pq[p.y], f0, p.y, true, el, vd);
                    sel = fma(el, G.leff, sel);
                    svd += vd;
                }
            }
            if (sw) tail1 = min(tail1 + 32, head1);
            else tail0 = min(tail0 + 32, head0);
        }
        if (last) break;
        __syncwarp();
    }
    block_reduce2(sel * ileff, svd, part + 2 * blockIdx.x);
}

// One batch of U entries per lane of row i: the pair terms of k_energy_list_mix.
template <int U, bool ISO, bool TYPED>
__device__ __forceinline__ void mix_batch(const int (&j)[U], const uint4 (&fj)[U], float4 (&pj)[U], const float4* s_cls,
                                          int i, uint4 fi, float4 pi, int k0, int m, float Ls0, float Ls1, float Ls2,
                                          float Ll0, float Ll1, float Ll2, float L2h, float L2l, float c2, float n2,
                                          float k3, float& ch, float& cl, float& vs) {
    // the batch's terms are summed in FP32 (at most U per lane), then added to the row sums once;
    // a slot past the row's end or beyond rc takes r^2 = rc^2, where the switch polynomial is 0
    float th = 0.f, tl = 0.f;
#pragma unroll
    for (int u = 0; u < U; u++) {
        if (k0 + u * 32 >= m) break;   // warp-uniform: this and later slots are past the row
        if (TYPED) pj[u] = s_cls[fj[u].w];
        float r2;
        if (ISO) {
            const float ux = __int2float_rn((int)(fj[u].x - fi.x)), uy = __int2float_rn((int)(fj[u].y - fi.y)),
                        uz = __int2float_rn((int)(fj[u].z - fi.z));
            const float r2u = fmaf(ux, ux, fmaf(uy, uy, uz * uz));
            r2 = fmaf(r2u, L2h, r2u * L2l);
        } else {
            const float dx = fixed_delta(fi.x, fj[u].x, Ls0, Ll0), dy = fixed_delta(fi.y, fj[u].y, Ls1, Ll1),
                        dz = fixed_delta(fi.z, fj[u].z, Ls2, Ll2);
            r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        }
        r2 = (j[u] != i && r2 <= c2) ? r2 : c2;
        float rinv = rsqrtf(r2);
        rinv = rinv * fmaf(-0.5f * r2 * rinv, rinv, 1.5f);   // one Newton step
        const float uu = fmaxf(r2, n2);
        const float a = c2 - uu;
        const float f = a * a * fmaf(2.0f, uu, k3);
        const float g = rinv * f;
        th = fmaf(pj[u].x, g, th);
        tl = fmaf(pj[u].y, g, tl);
        const float y = (pi.w + pj[u].w) * rinv;
        const float x2 = y * y;
        const float x6 = x2 * x2 * x2;
        vs = fmaf(pj[u].z, fmaf(x6, x6, -x6) * f, vs);
    }
    float sm, er;
    two_sum(ch, th, sm, er);
    ch = sm;
    cl += tl + er;
}

// Mixed-precision switched energy over the half list for periodic boxes: the pair kernel.  A warp
// per row i, lanes over its j > i entries.  One 16-byte load per list entry (the fixed-point
// position: exact minimum-image displacement by 32-bit wrap-around, scaled by a float-float box
// length) and one 16-byte load per pair inside the cutoff (charge as float-float, eps, sig).
// The row's sums are factored: each lane sums q_j g (g = S(r^2)/r, float-float by TwoSum) and
// eps_j l S (l = x^12 - x^6, FP32) over its entries of row i, and at the row's end multiplies them
// by q_i (float-float) and eps_i into float-float totals; no FP64 arithmetic until the block sum.
// The switch is formed unscaled as A^2 B with A = rc^2 - u, B = 2u + rc^2 - 3 ron^2 and u = r^2
// raised to ron^2; inv_f1 = 1 / (that FP32 polynomial at ron^2) scales the block sums, so inner
// pairs have S = 1 exactly.  Same terms as mixed_pair (unscaled, k_energy_tail scales).
// U list entries in flight per lane; MINB resident CTAs per SM requested from the register
// allocator (occupancy against registers); the engine times the variants once and keeps the fastest.
// Without the class table (TYPED below), both gathers of an entry (position and parameters) are
// issued together, unconditionally: over pruned rows ~88% of the entries lie within rc, so the
// parameter load is rarely wasted and the two dependent gather phases become one.  A padded slot (past the row's end) reads atom i itself
// and is masked by its index.  Slots wholly past the row's end are skipped by a warp-uniform test.
// ISO (cubic boxes): r^2 is summed in fixed-point units (exact integer differences converted to
// FP32) and scaled once by the float-float square of the unit length, two instructions per entry
// instead of a float-float scale per axis.
// TYPED: the atoms' parameters come from a table of the system's distinct (q, eps, sig) classes
// in shared memory, indexed by the class the fixed-point mirror carries in w, so an entry costs
// one global gather (its position) instead of two.
template <int U, int MINB, bool ISO, bool TYPED>
__global__ void __launch_bounds__(NB_THREADS, MINB) k_energy_list_mix(const uint4* __restrict__ fx, const float4* __restrict__ prm,
                                                                      const float4* __restrict__ cls, int ncls,
                                                                      int n, float Ls0, float Ls1, float Ls2, float Ll0,
                                                                      float Ll1, float Ll2, float L2h, float L2l,
                                                                      CutDev cut, double inv_f1,
                                                                      const int* __restrict__ nbr,
                                                                      const int* __restrict__ nup, int cap, double* part) {
    extern __shared__ float4 s_cls[];
    pair_kernel_begin();
    if (TYPED) {
        for (int c = threadIdx.x; c < ncls; c += blockDim.x) s_cls[c] = cls[c];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const float c2 = cut.c2f, n2 = cut.n2f, k3 = c2 - 3.0f * n2;
    float EH = 0.0f, EL = 0.0f, VH = 0.0f, VL = 0.0f;   // this lane's totals, float-float
    for (int i = warp; i < n; i += nwarps) {
        const uint4 fi = fx[i];
        const float4 pi = prm[i];        // (q hi, q lo, eps, sig)
        const int* row = nbr + (size_t)i * cap;
        const int m = nup[i];
        float ch = 0.0f, cl = 0.0f, vs = 0.0f;
        for (int k0 = 0; k0 < m; k0 += 32 * U) {
            int j[U];
            uint4 fj[U];
            float4 pj[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int k = k0 + u * 32 + lane;
                j[u] = k < m ? row[k] : i;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                fj[u] = fx[j[u]];
                if (!TYPED) pj[u] = prm[j[u]];
            }
            mix_batch<U, ISO, TYPED>(j, fj, pj, s_cls, i, fi, pi, k0, m, Ls0, Ls1, Ls2, Ll0, Ll1, Ll2, L2h, L2l, c2, n2,
                                     k3, ch, cl, vs);
        }
        mix_row_flush(pi, ch, cl, vs, EH, EL, VH, VL);
    }
    block_reduce2(((double)EH + (double)EL) * inv_f1, ((double)VH + (double)VL) * inv_f1, part + 2 * blockIdx.x);
}

// Dynamic pruning of the half Verlet rows for the pair kernel: row i keeps, in its order, the
// partners j > i whose FP32 distance (the pair kernel's own fixed-point displacement) lies within
// the prune radius rp at the current positions.  While no atom has moved more than (rp - rc) / 2
// since, every list pair within rc is still in the pruned rows, so the pair kernel sums the same
// pairs over ~30% fewer entries (rc + skin = 14 A list, rp = 12.5 A).  The reference's stale-list
// set is kept: pruning only removes pairs, never adds one the Verlet build left out.  A warp per
// row, U entries in flight per lane, survivors compacted by ballot.
constexpr int PRUNE_U = 4;

__global__ void __launch_bounds__(NB_THREADS) k_prune_rows(const uint4* __restrict__ fx, int n, float Ls0, float Ls1,
                                                        float Ls2, float Ll0, float Ll1, float Ll2, float rp2,
                                                        const int* __restrict__ nbr, const int* __restrict__ nup,
                                                        int cap, int* __restrict__ prn, int* __restrict__ pnup,
                                                        unsigned long long* kept_total) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const unsigned below = (1u << lane) - 1u;
    unsigned long long kept = 0;
    for (int i = warp; i < n; i += nwarps) {
        const uint4 fi = fx[i];
        const int* row = nbr + (size_t)i * cap;
        int* out = prn + (size_t)i * cap;
        const int m = nup[i];
        int w = 0;
        for (int k0 = 0; k0 < m; k0 += 32 * PRUNE_U) {
            int j[PRUNE_U];
            uint4 fj[PRUNE_U];
#pragma unroll
            for (int u = 0; u < PRUNE_U; u++) {
                const int k = k0 + u * 32 + lane;
                j[u] = k < m ? row[k] : -1;
            }
#pragma unroll
            for (int u = 0; u < PRUNE_U; u++) fj[u] = j[u] >= 0 ? fx[j[u]] : fi;
#pragma unroll
            for (int u = 0; u < PRUNE_U; u++) {
                const float dx = fixed_delta(fi.x, fj[u].x, Ls0, Ll0), dy = fixed_delta(fi.y, fj[u].y, Ls1, Ll1),
                            dz = fixed_delta(fi.z, fj[u].z, Ls2, Ll2);
                const bool keep = j[u] >= 0 && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= rp2;
                const unsigned b = __ballot_sync(0xffffffffu, keep);
                if (keep) out[w + __popc(b & below)] = j[u];
                w += __popc(b);
            }
        }
        if (lane == 0) {
            pnup[i] = w;
            kept += (unsigned long long)w;
        }
    }
    if (lane == 0 && kept) atomicAdd(kept_total, kept);
}

// Full energy without a box, FP64: all pairs j > i not in the full-mode exclusion row of i, no cutoff.
// Triangular grid of TILE x TILE blocks; each thread owns one i and walks a shared-memory j tile with
// the reference's sorted-row cursor (FField_MDBAS.cpp:227-234).
constexpr int TILE = 128;

__global__ void __launch_bounds__(TILE) k_energy_all(AtomsDev A, int n, PbcDev pbc, CutDev cut,
                                                     const int* __restrict__ fxs, const int* __restrict__ fxd,
                                                     int ntile, double* part) {
    __shared__ double4_32a spq[TILE];
    pair_kernel_begin();
    // block -> (I, J) with I <= J, row-major over the upper triangle
    int b = blockIdx.x;
    int I = 0;
    while (b >= ntile - I) { b -= ntile - I; I++; }
    int J = I + b;
    int i = I * TILE + threadIdx.x;
    int jt = J * TILE + threadIdx.x;
    if (jt < n) spq[threadIdx.x] = A.pq[jt];
    __syncthreads();
    double sel = 0.0, svd = 0.0;
    if (i < n) {
        const double4_32a pi = A.pq[i];
        const uint4 f0 = make_uint4(0, 0, 0, 0);
        int cur = fxs[i];
        const int xe = fxs[i + 1], j0 = max(J * TILE, i + 1), jend = min(n, J * TILE + TILE);
        while (cur < xe && fxd[cur] < j0) cur++;
        for (int j = j0; j < jend; j++) {
            if (cur < xe && fxd[cur] == j) { cur++; continue; }
            double el, vd;
            pair_energy<PREC_F64>(A, pbc, cut, false, pi, f0, i, spq[j - J * TILE], f0, j, false, el, vd);
            sel += el;
            svd += vd;
        }
    }
    block_reduce2(sel, svd, part + 2 * blockIdx.x);
}

// The other full energies deal units of ALL_I rows (a thread each) against ALL_J columns staged in shared
// memory to the CTAs in turn; units are numbered over the upper triangle row tile by row tile.  Short
// columns, because a thread's walk along them is serial: a box of 1,536 atoms has 312 units (12 x 13 / 2
// = 78 with square tiles, for 152 SMs), and a CTA's partial sum covers all its units.
constexpr int ALL_I = 128, ALL_J = 32, ALL_STEP = ALL_I / ALL_J;

static long long all_units(int n) {
    const long long tiles = (n + ALL_I - 1) / ALL_I, c0 = (n + ALL_J - 1) / ALL_J;
    return tiles * c0 - ALL_STEP * tiles * (tiles - 1) / 2;
}

// Unit -> its row tile (returned) and first column; c0 column chunks in row tile 0, each next tile has
// ALL_STEP fewer.  The float estimate is put right by steps of one.
__device__ __forceinline__ int all_unit(long long unit, int c0, int& jb) {
    auto first = [&](int I) { return (long long)I * c0 - (long long)ALL_STEP * I * (I - 1) / 2; };
    const float b = c0 + 0.5f * ALL_STEP;
    int I = (int)((b - sqrtf(fmaxf(b * b - 2.0f * ALL_STEP * (float)unit, 0.0f))) / ALL_STEP);
    while (I > 0 && first(I) > unit) I--;
    while (first(I + 1) <= unit) I++;
    jb = I * ALL_I + (int)(unit - first(I)) * ALL_J;
    return I;
}

// TwoSum on both halves: s becomes s + v, c takes what that rounds off
__device__ __forceinline__ void two_sum_to(float2& s, float2& c, float2 v) {
    const float2 neg = make_float2(-1.0f, -1.0f);
    const float2 t = __fadd2_rn(s, v), b = __ffma2_rn(s, neg, t);
    c = __fadd2_rn(c, __fadd2_rn(__ffma2_rn(__ffma2_rn(b, neg, t), neg, s), __ffma2_rn(b, neg, v)));
    s = t;
}

// Mixed-precision full energy: the pair terms of mixed_pair without the switch for two columns at a time,
// the halves of float2 values, summed per thread and half as float-float over ALLMIX_FLUSH units, 64 pairs a
// half, in FP64 beyond: float-float holds 48 bits of its largest partial sum, and over thousands of pairs of one
// thread that showed (the Lennard-Jones energy of 36,864 argon atoms moved by 1.2e-14 with their order, by 2.2e-16
// so; 2% of the time).  A column that is not to count (excluded, not above the row, past the last atom) takes
// 1/r = 0, which makes its terms exactly 0.  Bound by the FP32 pipe.  The columns' positions and
// parameters come from shared memory, the row's and the next excluded atom stay in registers.
// Without a box a displacement is an FP64 difference rounded to FP32, and those are the bound.
// Whole energy calls, against a column at a time in square tiles with the exclusion row read at every
// column: 12,288 water atoms (75 M pairs) 171 us, was 227; 36,864 1384, was 1652 (one column at a time
// in these units: 1475); 4,096 argon atoms 37, was 56.
constexpr int ALLMIX_FLUSH = 4;
constexpr int ALLMIX_CTAS = 5;   // per SM; 3,000 water atoms, 36,864: 4 take 31 and 1388 us, 5 34 and 1360, 8 37 and 1359 (float-float throughout)

template <bool BOX>
__global__ void __launch_bounds__(ALL_I, ALLMIX_CTAS) k_energy_all_mix(AtomsDev A, int n,
                                                                       const int* __restrict__ fxs,
                                                                       const int* __restrict__ fxd, long long units,
                                                                       double* part) {
    __shared__ __align__(8) uint32_t sp[3][ALL_J];
    __shared__ double sd[3][BOX ? 1 : ALL_J];
    __shared__ __align__(8) float sprm[4][ALL_J];        // q hi, q lo, eps, sig
    pair_kernel_begin();
    const int c0 = (n + ALL_J - 1) / ALL_J;
    const float2 zero = make_float2(0.0f, 0.0f), neg = make_float2(-1.0f, -1.0f);
    auto both = [](float v) { return make_float2(v, v); };
    float2 eh = zero, el = zero, vh = zero, vl = zero;
    double sel = 0.0, svd = 0.0;
    auto flush = [&]() {
        sel += ((double)eh.x + (double)eh.y) + ((double)el.x + (double)el.y);
        svd += ((double)vh.x + (double)vh.y) + ((double)vl.x + (double)vl.y);
        eh = el = vh = vl = zero;
    };
    int since = 0;   // units since the float-float sums went to FP64
    for (long long unit = blockIdx.x; unit < units; unit += gridDim.x) {
        if (since++ == ALLMIX_FLUSH) { flush(); since = 1; }
        int jb;
        const int i = all_unit(unit, c0, jb) * ALL_I + threadIdx.x, je = min(n, jb + ALL_J);
        __syncthreads();
        if (threadIdx.x < ALL_J) {
            const int t = threadIdx.x, jt = min(jb + t, n - 1);
            if (BOX) {
                const uint4 f = A.fx[jt];
                sp[0][t] = f.x; sp[1][t] = f.y; sp[2][t] = f.z;
            } else {
                const double4_32a p = A.pq[jt];
                sd[0][t] = p.x; sd[1][t] = p.y; sd[2][t] = p.z;
            }
            const float2 q = A.qf[jt], e = A.esf[jt];
            sprm[0][t] = q.x; sprm[1][t] = q.y; sprm[2][t] = e.x; sprm[3][t] = e.y;
        }
        __syncthreads();
        if (i >= n) continue;
        uint4 fi = make_uint4(0, 0, 0, 0);
        double4_32a pi = make_double4_32a(0, 0, 0, 0);
        if (BOX) fi = A.fx[i];
        else pi = A.pq[i];
        const float2 qi = A.qf[i], ei = A.esf[i];
        int cur = fxs[i];
        const int xe = fxs[i + 1];
        while (cur < xe && fxd[cur] < jb) cur++;
        int next = cur < xe ? fxd[cur] : INT_MAX;     // the reference's sorted-row cursor (FField_MDBAS.cpp:227-234)
        for (int j = max(jb, (i + 1) & ~1); j < je; j += 2) {
            const int t = j - jb;
            bool on0 = j > i, on1 = j + 1 < je;
            if (next <= j + 1) {                 // rows hold partners above i only
                for (; next <= j + 1; next = ++cur < xe ? fxd[cur] : INT_MAX) {
                    if (next == j) on0 = false;
                    else on1 = false;
                }
            }
            auto col = [&](const float* v) { return *reinterpret_cast<const float2*>(v + t); };
            float2 dx, dy, dz;
            if (BOX) {
                auto diff = [&](int k, uint32_t f) {
                    const uint2 c = *reinterpret_cast<const uint2*>(&sp[k][t]);
                    const float2 d = make_float2(__int2float_rn((int)(c.x - f)), __int2float_rn((int)(c.y - f)));
                    return __ffma2_rn(d, both(A.Ls[k]), __fmul2_rn(d, both(A.Lsl[k])));
                };
                dx = diff(0, fi.x); dy = diff(1, fi.y); dz = diff(2, fi.z);
            } else {
                auto diff = [&](int k, double p) { return make_float2((float)(sd[k][t] - p), (float)(sd[k][t + 1] - p)); };
                dx = diff(0, pi.x); dy = diff(1, pi.y); dz = diff(2, pi.z);
            }
            const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy)));
            float2 y = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
            y = __fmul2_rn(y, __ffma2_rn(__fmul2_rn(__fmul2_rn(both(-0.5f), r2), y), y, both(1.5f)));   // one Newton step
            y.x = on0 ? y.x : 0.0f;
            y.y = on1 ? y.y : 0.0f;
            // the float-float charge product (ff_mul)
            const float2 qh = col(sprm[0]), ql = col(sprm[1]);
            const float2 ph = __fmul2_rn(both(qi.x), qh), nph = __fmul2_rn(both(-qi.x), qh);
            const float2 pl = __fadd2_rn(__ffma2_rn(both(qi.x), qh, nph), __ffma2_rn(both(qi.x), ql, __fmul2_rn(both(qi.y), qh)));
            two_sum_to(eh, el, __ffma2_rn(ph, y, __fmul2_rn(pl, y)));
            const float2 s = __fadd2_rn(both(ei.y), col(sprm[3]));
            const float2 x2 = __fmul2_rn(__fmul2_rn(s, s), __fmul2_rn(y, y)), x6 = __fmul2_rn(__fmul2_rn(x2, x2), x2);
            const float2 l = __ffma2_rn(x6, x6, __fmul2_rn(neg, x6));
            two_sum_to(vh, vl, __fmul2_rn(__fmul2_rn(both(ei.x), col(sprm[2])), l));
        }
    }
    flush();
    block_reduce2(sel, svd, part + 2 * blockIdx.x);
}

// FP64 full energy for periodic boxes, on 64-bit integer pair terms (fixed64.cuh): three FP64
// operations a pair, about 230 cycles of a scheduler's FP64 pipe per warp, beside some 150 integer
// and FP32 ones.
// 12,288 atoms (75 M pairs): the whole energy call takes 0.62 ms, 3.78 ms with the pair terms in FP64 (0.57 with the
// sigmas' powers as doubles, whose rounding all pairs of two classes share).  ncu: FP64 pipe 62%, ALU 50%, issue 59%.
constexpr int A64_CTAS = 10;   // per SM; 8, whole calls: 632 against 620 us at 12,288 atoms, 91.7 against 89.3 at 4,096, alike below

template <bool ISO, bool TABLE>
__global__ void __launch_bounds__(ALL_I, A64_CTAS) k_energy_all64(AtomsDev A, Fix64Geom G, PbcDev pbc, CutDev cut, int n,
                                                        const int* __restrict__ fxs, const int* __restrict__ fxd,
                                                        long long units, double* part) {
    __shared__ ulonglong4_32a sx[ALL_J];
    pair_kernel_begin();
    const double ileff = 1.0 / G.leff;
    const int c0 = (n + ALL_J - 1) / ALL_J;
    double sel = 0.0, svd = 0.0;
    for (long long unit = blockIdx.x; unit < units; unit += gridDim.x) {
        int jb;
        const int i = all_unit(unit, c0, jb) * ALL_I + threadIdx.x, je = min(n, jb + ALL_J);
        __syncthreads();
        if (threadIdx.x < ALL_J && jb + threadIdx.x < n) sx[threadIdx.x] = A.x64[jb + threadIdx.x];
        __syncthreads();
        if (i >= n) continue;
        const ulonglong4_32a a = A.x64[i];
        int cur = fxs[i];
        const int xe = fxs[i + 1], j0 = max(jb, i + 1);
        while (cur < xe && fxd[cur] < j0) cur++;
        int next = cur < xe ? fxd[cur] : n;      // the reference's sorted-row cursor (FField_MDBAS.cpp:227-234)
        for (int j = jb; j < je; j++) {
            if (j <= i) continue;
            if (j == next) {
                cur++;
                next = cur < xe ? fxd[cur] : n;
                continue;
            }
            const ulonglong4_32a bj = sx[j - jb];
            const Fix64Dist u = fix64_dist2<ISO, true>(G, a, bj);
            double ys, w, ws, qq, ee;
            unsigned long long ms;
            int es;
            pair64_params<TABLE>(A, ileff, i, j, (int)a.w, (int)bj.w, qq, ee, ms, es);
            if (fix64_terms(G, u, false, ms, es, ys, w, ws)) {
                sel = fma(qq, ys, sel);
                svd = fma(ee, fma(w, ws, -ws), svd);
            } else {
                double el, vd;
                const uint4 f0 = make_uint4(0, 0, 0, 0);
                pair_energy<PREC_F64>(A, pbc, cut, false, A.pq[i], f0, i, A.pq[j], f0, j, false, el, vd);
                sel = fma(el, G.leff, sel);
                svd += vd;
            }
        }
    }
    block_reduce2(sel * ileff, svd, part + 2 * blockIdx.x);
}

// ---- bonded terms (FP64, device math library) ---------------------------------------------
struct BondedDev {
    const BondT* bonds; int nb;
    const BondT* ubs; int nu;
    const AngleT* angles; int na;
    const TorsT* dihes; int nd;
    const TorsT* imprs; int ni;
};

__device__ __forceinline__ void crd(const double4_32a* pq, int i, double c[3]) {
    double4_32a p = pq[i]; c[0] = p.x; c[1] = p.y; c[2] = p.z;
}
__device__ __forceinline__ void apply_pbc(double d[3], const PbcDev& p) {
    if (p.type != 0) for (int k = 0; k < 3; k++) d[k] = ref64_mic(d[k], p.L[k], p.rL[k]);
}

// crd_of: coordinates of atom i, with moved atoms taken from the proposal.
struct CrdSrc {
    const double4_32a* pq;
    const int* mv_idx; const double* mv_xyz; int m;   // sorted moved atoms (may be m = 0)
    __device__ __forceinline__ void get(int i, double c[3]) const {
        int lo = 0, hi = m - 1;
        while (lo <= hi) {
            int mid = (lo + hi) >> 1, v = mv_idx[mid];
            if (v == i) { c[0] = mv_xyz[3 * mid]; c[1] = mv_xyz[3 * mid + 1]; c[2] = mv_xyz[3 * mid + 2]; return; }
            if (v < i) lo = mid + 1; else hi = mid - 1;
        }
        crd(pq, i, c);
    }
};

__device__ double bond_e(const BondT& b, const CrdSrc& S, const PbcDev& pbc, bool morse_ok) {
    double di[3], dj[3];
    S.get(b.a, di); S.get(b.b, dj);
    double d = sqrt(ref64_dist2(di[0], di[1], di[2], dj[0], dj[1], dj[2], pbc));
    if (morse_ok && b.type == 1) {
        double ma = exp(-b.beta * (d - b.r0));
        return b.k * (ma * ma - 2. * ma) + b.k;
    }
    return 0.5 * b.k * (d - b.r0) * (d - b.r0);
}

// The angle and torsion terms need an angle's deviation from its reference, or the cosine of a
// multiple of it, and both follow from sines and cosines: the library's acos, atan2 and cos are
// some 100 FP64 operations each, at 64 cycles of a scheduler's FP64 pipe per warp.  The general form
// (out of line) stays for what the short one does not cover: an angle more than 2^-6 off its reference
// or nearly straight, a multiplicity that is not an integer of 0 to 6, three atoms in line.  With a grid
// of two CTAs per SM instead of 64 in all this took the bonded terms of 100,002 water atoms from 31 us
// (46 before the minimum image went to integer compares) to 12; a term per thread (BD_BLOCKS) came after.

// asin(s) for |s| <= 2^-6: the Taylor series to s^9 (the next term is below 2^-64 of s)
__device__ __forceinline__ double asin_small(double s) {
    const double z = s * s;
    const double p = fma(z, fma(z, fma(z, 35.0 / 1152.0, 5.0 / 112.0), 3.0 / 40.0), 1.0 / 6.0);
    return fma(s * z, p, s);
}
__device__ __forceinline__ bool below_abs(double v, unsigned hi) { return ((unsigned)__double2hiint(v) & 0x7fffffffu) < hi; }   // NaN: false
constexpr unsigned HI_2M6 = 0x3f900000u;        // 2^-6
constexpr unsigned HI_ALMOST1 = 0x3feff800u;    // 1 - 2^-10

__device__ __noinline__ double angle_general(double dot, double r2ab, double r2bc, double theta0) {
    return acos(dot / (sqrt(r2ab) * sqrt(r2bc))) - theta0;
}

__device__ __forceinline__ double angle_e(const AngleT& a, const CrdSrc& S, const PbcDev& pbc) {
    double di[3], dj[3], dk[3], dab[3], dbc[3];
    S.get(a.a, di); S.get(a.b, dj); S.get(a.c, dk);
    const double r2ab = ref64_dist2(di[0], di[1], di[2], dj[0], dj[1], dj[2], pbc, dab);
    const double r2bc = ref64_dist2(dk[0], dk[1], dk[2], dj[0], dj[1], dj[2], pbc, dbc);
    const double dot = fma(dab[0], dbc[0], fma(dab[1], dbc[1], dab[2] * dbc[2]));
    const double c = dot * rsqrt64(r2ab * r2bc);
    const double u = fma(-c, c, 1.0);
    // sin(theta - theta0); a small one is a small deviation, theta and theta0 both well inside (0, pi)
    const double s = fma(u * rsqrt64(u), a.cos0, -(c * a.sin0));
    const double th = below_abs(c, HI_ALMOST1) && below_abs(s, HI_2M6) ? asin_small(s) : angle_general(dot, r2ab, r2bc, a.theta0);
    return 0.5 * a.k * th * th;
}

// the deviation of a harmonic torsion, or the angle itself
__device__ __noinline__ double tors_general(const TorsT& t, double sinp, double cosp) {
    double phi = atan2(sinp, cosp);
    if (t.type == 2) {
        phi = phi - t.phi0;
        phi = phi - ref64_rint(phi / TWOPI) * TWOPI;
        return 0.5 * t.k * phi * phi;
    }
    return t.k * (1. + cos(t.mult * phi - t.phi0));
}

__device__ __forceinline__ double tors_e(const TorsT& t, const CrdSrc& S, const PbcDev& pbc) {
    double di[3], dj[3], dk[3], dl[3], dab[3], dbc[3], dcd[3], pb[3], pc[3];
    S.get(t.a, di); S.get(t.b, dj); S.get(t.c, dk); S.get(t.d, dl);
    for (int k = 0; k < 3; k++) { dab[k] = di[k] - dj[k]; dcd[k] = dk[k] - dl[k]; }
    apply_pbc(dab, pbc); apply_pbc(dcd, pbc);
    const double rbc = sqrt(ref64_dist2(dk[0], dk[1], dk[2], dj[0], dj[1], dj[2], pbc, dbc));
    auto cross = [](const double* x, const double* y, double* z) {
        z[0] = fma(x[1], y[2], -(x[2] * y[1]));
        z[1] = fma(x[2], y[0], -(x[0] * y[2]));
        z[2] = fma(x[0], y[1], -(x[1] * y[0]));
    };
    auto dot = [](const double* x, const double* y) { return fma(x[0], y[0], fma(x[1], y[1], x[2] * y[2])); };
    double pcb[3];
    cross(dab, dbc, pb);
    cross(dbc, dcd, pc);
    cross(pc, pb, pcb);
    // sin phi and cos phi times |pb| |pc| |bc|
    const double sn = dot(dbc, pcb), cn = dot(pb, pc) * rbc;
    const double u = fma(sn, sn, cn * cn);
    if (!((unsigned)__double2hiint(u) - 0x00100000u < 0x7fe00000u)) {   // three atoms in line, or not finite: the reference's quotients
        const double q = sqrt(dot(pb, pb)) * sqrt(dot(pc, pc));
        return tors_general(t, sn / (q * rbc), dot(pb, pc) / q);
    }
    const double inv = rsqrt64(u), s1 = sn * inv, c1 = cn * inv;
    if (t.type == 2) {
        const double s = fma(s1, t.cos0, -(c1 * t.sin0)), c = fma(c1, t.cos0, s1 * t.sin0);   // of phi - phi0
        if (!(below_abs(s, HI_2M6) && __double2hiint(c) >= 0)) return tors_general(t, s1, c1);
        const double d = asin_small(s);
        return 0.5 * t.k * d * d;
    }
    if (t.nmult < 0) return tors_general(t, s1, c1);
    double s = 0.0, c = 1.0;                            // of n phi, by the addition theorem
    for (int n = 0; n < t.nmult; n++) {
        const double cc = fma(c, c1, -(s * s1));
        s = fma(s, c1, c * s1);
        c = cc;
    }
    return t.k * (1.0 + fma(c, t.cos0, s * t.sin0));
}

// The rest of an energy beside the pair kernel, in one launch: bonded terms (blocks below nbd), 1-4
// pairs (the n14b blocks behind), and the sums.  It is launched as the pair kernel's programmatic
// dependent: once every CTA of that has started (pair_kernel_begin) this one's begin too where they
// fit, so the FP64 terms run beside the pair kernel, and only the last block to finish waits for the
// pair kernel's partial sums.  That block adds all partials in a fixed order.
// Whole energy calls against separate kernels for bonded terms, 1-4 pairs and sums: 864 argon atoms
// 29.6 -> 24.5 us, 12,288 water atoms in full mode 579 -> 566, 100,002 in FP64 577 -> 539.  The packed
// group kernels of the mixed energy leave no registers beside them (2 x 256 threads of 128): 122 either way.
template <int P>
__global__ void __launch_bounds__(256) k_energy_tail(BondedDev B, int nbd, AtomsDev A, PbcDev pbc, CutDev cut,
                                                     const int2* __restrict__ p14, int n14, int n14b, const double* nb, int nnb,
                                                     double* part, unsigned* ticket, double* out) {
    __shared__ double sh[9][8];
    __shared__ bool s_last;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    double* bd = part;                    // five sums per bonded block, then two per 1-4 block
    double* s14 = part + 5 * nbd;
    if ((int)blockIdx.x < nbd) {
        double e[5] = {0, 0, 0, 0, 0};
        const CrdSrc S{A.pq, nullptr, nullptr, 0};
        const int total = B.nb + B.na + B.nu + B.nd + B.ni;
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < total; k += nbd * blockDim.x) {
            int t = k;
            if (t < B.nb) { e[0] += bond_e(B.bonds[t], S, pbc, true); continue; }
            t -= B.nb;
            if (t < B.na) { e[1] += angle_e(B.angles[t], S, pbc); continue; }
            t -= B.na;
            if (t < B.nu) { e[2] += bond_e(B.ubs[t], S, pbc, false); continue; }
            t -= B.nu;
            if (t < B.nd) { e[3] += tors_e(B.dihes[t], S, pbc); continue; }
            t -= B.nd;
            e[4] += tors_e(B.imprs[t], S, pbc);
        }
        for (int c = 0; c < 5; c++) {
            // a warp holds terms of one kind or two: the others' sums are zero without the five additions
            double v = __any_sync(0xffffffffu, __double_as_longlong(e[c]) != 0) ? warp_sum(e[c]) : 0.0;
            if (l == 0) sh[c][w] = v;
        }
        __syncthreads();
        if (threadIdx.x < 5) {
            double s = 0.0;
            for (int k = 0; k < (int)(blockDim.x >> 5); k++) s += sh[threadIdx.x][k];
            bd[5 * blockIdx.x + threadIdx.x] = s;
            __threadfence();
        }
    } else if ((int)blockIdx.x < nbd + n14b) {
        const int b = blockIdx.x - nbd;
        double sel = 0.0, svd = 0.0;
        for (int k = b * blockDim.x + threadIdx.x; k < n14; k += n14b * blockDim.x) {
            int2 p = p14[k];
            double el, vd;
            uint4 fi = P == PREC_MIX ? A.fx[p.x] : make_uint4(0, 0, 0, 0);
            uint4 fj = P == PREC_MIX ? A.fx[p.y] : make_uint4(0, 0, 0, 0);
            pair_energy<P>(A, pbc, cut, true, A.pq[p.x], fi, p.x, A.pq[p.y], fj, p.y, cut.mode == 1, el, vd);
            sel += el; svd += vd;
        }
        block_reduce2(sel, svd, s14 + 2 * b);
        if (threadIdx.x == 0) __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;   // uniform over the block
    __threadfence();
    // The partial sums, eight loads in flight: 1-4 elec and vdw and the five bonded components by a warp
    // each, then, when the pair kernel has ended, its two by four warps each: only those are left to do
    // after it (up to 1,520 partial sums; a warp per component took 63 against 60 us for a full FP64
    // energy of 3,000 atoms, 56.5 against 54.5 for a mixed one of a peptide box of 18,040).
    auto sum = [](const double* src, int count, int step, int k0, int dk) {
        double v = 0.0;
#pragma unroll 8
        for (int k = k0; k < count; k += dk) v += __ldcg(src + (size_t)k * step);
        return warp_sum(v);
    };
    if (w < 7) {
        const double v = w < 2 ? sum(s14 + w, n14b, 2, l, 32) : sum(bd + (w - 2), nbd, 5, l, 32);
        if (l == 0) sh[2 + w][0] = v;
    }
    pair_kernel_wait();
    const double v = sum(nb + (w & 1), nnb, 2, 32 * (w >> 1) + l, 128);
    if (l == 0) sh[w & 1][w >> 1] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        const double K = CHGCHARMM * KCALTOIU;
        double elec = K * ((sh[0][0] + sh[0][1]) + (sh[0][2] + sh[0][3]));
        double vdw = 4.0 * ((sh[1][0] + sh[1][1]) + (sh[1][2] + sh[1][3]));
        elec += K * sh[2][0];
        vdw += 4.0 * sh[3][0];
        double bond = sh[4][0], ang = sh[5][0], ub = sh[6][0], dihe = sh[7][0], impr = sh[8][0];
        double pot = elec + vdw + bond + ang + ub + dihe + impr;
        out[0] = pot + 0.0; out[1] = pot; out[2] = 0.0; out[3] = elec; out[4] = vdw;
        out[5] = bond; out[6] = ang; out[7] = ub; out[8] = dihe; out[9] = impr;
        *ticket = 0u;
    }
}

// ------------------------------------------------------------------------------------------
// Energy change of a moved set.  Blocks b < m*S take moved atom mv[b / S] against slice b % S of
// its partners (Verlet row in switch mode, every atom in full mode) and of its 1-4 partners; the blocks
// behind them take the listed bonded terms, a block per kind present.  Pairs with both atoms moved are
// counted once, by the lower index.
// Bound by latency: the longest chain of dependent FP64 operations (64 cycles each on GB300, whatever a
// warp's active lanes) between the launch and the result.  So FP64 pairs take their old and new energy on
// two lanes, rows spread until a thread has one such term, bonded kinds run on blocks of their own with
// the old terms on one warp and the new ones on the other, and a thread's contributions become one number
// before the sums across lanes, warps and blocks.  The last block to finish sums the partials (a fixed
// order, so de is reproducible) and writes de (iu).
// A water move took 18 us (FP64 or mixed) with both sides of a pair and of all bonded terms on one
// thread, three sums per block and two more block sums at the end; 11 and 10 now.  A move of a chain atom
// with its dihedrals took 46 to 73 us before this and the shorter bonded terms; 14 to 19 now.
constexpr int DE_KINDS = 5;   // bonds, angles, Urey-Bradley, dihedrals, impropers
struct MoveDev {
    int m;
    const int* idx;        // sorted moved atoms
    const double* xyz;     // their proposed coordinates (3 per atom)
    const int* terms;      // bonded terms touching them, kind after kind
    int nkind;             // kinds present, each with the end of its terms
    int kind[DE_KINDS], kend[DE_KINDS];
};

// A small proposal travels inside the launch (kernel parameter space, read through the constant
// cache), so that a trial move costs one launch and no copy; m = 0 means it was staged in device
// memory and MoveDev points there.
constexpr int INL_M = 32, INL_T = 192;
struct MoveInline {
    int m;
    int idx[INL_M];
    int terms[INL_T];
    double xyz[3 * INL_M];
};

// sum over the block; thread 0 has it
__device__ __forceinline__ double block_sum(double v, double* s) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) v += s[w];
    return v;
}

// M: the moved atoms the shared arrays hold (a small proposal's block asks for little shared memory)
template <int P, int M>
__global__ void __launch_bounds__(256) k_delta_e(AtomsDev A, int n, PbcDev pbc, CutDev cut, const __grid_constant__ MoveDev mv,
                                                 const int* __restrict__ nbr, const int* __restrict__ nup,
                                                 const int* __restrict__ nlo, int cap,
                                                 const int* __restrict__ fxs, const int* __restrict__ fxd,
                                                 const int* __restrict__ c14s, const int* __restrict__ c14d,
                                                 BondedDev B, int S, double* part, unsigned* ticket, double* out,
                                                 const __grid_constant__ MoveInline inl) {
    __shared__ int s_idx[M];
    __shared__ double s_xyz[3 * M];
    __shared__ uint4 s_fx[P == PREC_MIX ? M : 1];
    __shared__ double s_sum[8];
    __shared__ bool s_last;
    const int* idx = inl.m > 0 ? inl.idx : mv.idx;
    const double* xyz = inl.m > 0 ? inl.xyz : mv.xyz;
    const int* terms = inl.m > 0 ? inl.terms : mv.terms;
    const int m = mv.m;
    for (int k = threadIdx.x; k < m; k += blockDim.x) s_idx[k] = idx[k];
    for (int k = threadIdx.x; k < 3 * m; k += blockDim.x) {
        const double v = xyz[k];
        s_xyz[k] = v;
        if (P == PREC_MIX && pbc.type != 0) reinterpret_cast<uint32_t*>(s_fx + k / 3)[k % 3] = to_fixed(v, pbc.rL[k % 3]);
    }
    __syncthreads();
    auto slot = [&](int j) -> int {
        int lo = 0, hi = m - 1;
        while (lo <= hi) {
            int mid = (lo + hi) >> 1, v = s_idx[mid];
            if (v == j) return mid;
            if (v < j) lo = mid + 1; else hi = mid - 1;
        }
        return -1;
    };
    double del = 0.0, dvd = 0.0, dbd = 0.0;
    const bool sw = cut.mode == 1;
    if ((int)blockIdx.x < m * S) {
        const int ka = blockIdx.x / S;
        const int k0 = (blockIdx.x % S) * blockDim.x + threadIdx.x, kstep = S * blockDim.x;
        const int a = s_idx[ka];
        const double4_32a ao = A.pq[a];
        const double4_32a an = make_double4_32a(s_xyz[3 * ka], s_xyz[3 * ka + 1], s_xyz[3 * ka + 2], ao.w);
        const uint4 f0 = make_uint4(0, 0, 0, 0);
        const uint4 fo = P == PREC_MIX ? A.fx[a] : f0;
        const uint4 fn = P == PREC_MIX ? s_fx[ka] : f0;
        CutDev cutx = cut;   // full mode: no cutoff and no switch
        if (!sw) { cutx.c2f = 1.0e30f; cutx.n2f = 1.0e30f; }   // "no cutoff": finite, so c2 - 3 n2 stays finite
        float ma[3] = {0.f, 0.f, 0.f};   // the exact move of a, as the fixed-point mirror sees it
        if (P == PREC_MIX) {
            if (pbc.type != 0) {
                ma[0] = fixed_delta(fo.x, fn.x, A.Ls[0], A.Lsl[0]);
                ma[1] = fixed_delta(fo.y, fn.y, A.Ls[1], A.Lsl[1]);
                ma[2] = fixed_delta(fo.z, fn.z, A.Ls[2], A.Lsl[2]);
            } else {
                ma[0] = (float)(an.x - ao.x); ma[1] = (float)(an.y - ao.y); ma[2] = (float)(an.z - ao.z);
            }
        }
        // FP64: the old (side 0, subtracted) or new energy of the pair
        auto visit64 = [&](int j, bool fourteen, bool apply_cut, int side) {
            const int sj = slot(j);
            if (sj >= 0 && j < a) return;       // counted by the lower index's block
            double4_32a pa = ao, pj = A.pq[j];
            if (side) {
                pa = an;
                if (sj >= 0) { pj.x = s_xyz[3 * sj]; pj.y = s_xyz[3 * sj + 1]; pj.z = s_xyz[3 * sj + 2]; }
            }
            double e, v;
            pair_energy<PREC_F64>(A, pbc, cut, fourteen, pa, f0, a, pj, f0, j, apply_cut, e, v);
            del += side ? e : -e;
            dvd += side ? v : -v;
        };
        auto visit = [&](int j, bool fourteen, bool apply_cut) {
            int sj = slot(j);
            if (sj >= 0 && j < a) return;       // counted by the lower index's block
            double4_32a jo = pbc.type != 0 ? make_double4_32a(0, 0, 0, 0) : A.pq[j];
            uint4 gjo = A.fx[j];
            double4_32a jn = jo;
            uint4 gjn = gjo;
            if (sj >= 0) { jn.x = s_xyz[3 * sj]; jn.y = s_xyz[3 * sj + 1]; jn.z = s_xyz[3 * sj + 2]; gjn = s_fx[sj]; }
            {
                // d_old = j_old - a_old, d_new = j_new - a_new = d_old - m
                float d[3], m[3];
                if (pbc.type != 0) {
                    d[0] = fixed_delta(fo.x, gjo.x, A.Ls[0], A.Lsl[0]); d[1] = fixed_delta(fo.y, gjo.y, A.Ls[1], A.Lsl[1]); d[2] = fixed_delta(fo.z, gjo.z, A.Ls[2], A.Lsl[2]);
                } else {
                    d[0] = (float)(jo.x - ao.x); d[1] = (float)(jo.y - ao.y); d[2] = (float)(jo.z - ao.z);
                }
                // d_new by minimum image; m = d_old - d_new is taken from the exact move of a when
                // only a moved (so the analytic difference keeps its accuracy), and the pair is
                // differenced directly when the move carries it across half the box
                float dn[3];
                if (pbc.type != 0) {
                    dn[0] = fixed_delta(fn.x, gjn.x, A.Ls[0], A.Lsl[0]); dn[1] = fixed_delta(fn.y, gjn.y, A.Ls[1], A.Lsl[1]); dn[2] = fixed_delta(fn.z, gjn.z, A.Ls[2], A.Lsl[2]);
                } else {
                    dn[0] = (float)(jn.x - an.x); dn[1] = (float)(jn.y - an.y); dn[2] = (float)(jn.z - an.z);
                }
                bool flip = false;
                if (sj >= 0) { m[0] = d[0] - dn[0]; m[1] = d[1] - dn[1]; m[2] = d[2] - dn[2]; }
                else {
                    m[0] = ma[0]; m[1] = ma[1]; m[2] = ma[2];
                    for (int t = 0; t < 3; t++) flip |= fabsf(d[t] - m[t] - dn[t]) > 1.0f;
                }
                float2 pa = fourteen ? A.esf14[a] : A.esf[a];
                float2 pb = fourteen ? A.esf14[j] : A.esf[j];
                float s = pa.y + pb.y;
                float2 qa = A.qf[a], qb = A.qf[j];
                float qh, ql;
                ff_mul(qa.x, qa.y, qb.x, qb.y, qh, ql);
                float qk = (float)(CHGCHARMM * KCALTOIU) * (qh + ql);
                int np_ = 0;
                if (!flip) {
                    dbd += (double)mixed_pair_delta(d[0], d[1], d[2], m[0], m[1], m[2], qk, 4.0f * pa.x * pb.x, s * s,
                                                    apply_cut ? cut : cutx, np_);
                } else {
                    float e0, v0, e1, v1;
                    const CutDev& cc = apply_cut ? cut : cutx;
                    const float u0 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2], u1 = dn[0] * dn[0] + dn[1] * dn[1] + dn[2] * dn[2];
                    e0 = v0 = e1 = v1 = 0.f;
                    if (!apply_cut || u0 <= cc.c2f) mixed_pair(u0, qh, ql, pa.x * pb.x, s * s, apply_cut, cc, e0, v0);
                    if (!apply_cut || u1 <= cc.c2f) mixed_pair(u1, qh, ql, pa.x * pb.x, s * s, apply_cut, cc, e1, v1);
                    dbd += (double)(CHGCHARMM * KCALTOIU) * ((double)e1 - (double)e0) + 4.0 * ((double)v1 - (double)v0);
                }
            }
        };
        // partner k of a's 1-4 pairs, of its row, or of all atoms; FP64: k = 2 partner + side
        constexpr int SIDES = P == PREC_F64 ? 2 : 1;
        auto at = [&](int k, int j, bool fourteen) {
            if (P == PREC_F64) visit64(j, fourteen, sw, k & 1);
            else visit(j, fourteen, sw);
        };
        if (sw) {
            const int* row = nbr + (size_t)a * cap;
            const int u = nup[a], l = nlo[a];
            for (int k = k0; k < SIDES * (u + l); k += kstep) {
                const int t = k / SIDES;
                at(k, t < u ? row[t] : row[cap - 1 - (t - u)], false);
            }
        } else {
            for (int k = k0; k < SIDES * n; k += kstep) {
                const int j = k / SIDES;
                if (j == a) continue;
                const int lo_ = min(a, j), hi_ = max(a, j);
                bool ex = false;
                for (int x = fxs[lo_]; x < fxs[lo_ + 1]; x++) if (fxd[x] == hi_) { ex = true; break; }
                if (!ex) at(k, j, false);
            }
        }
        const int c0 = c14s[a], c1 = c14s[a + 1];
        for (int k = k0; k < SIDES * (c1 - c0); k += kstep) at(k, c14d[c0 + k / SIDES], true);
        dbd = fma(CHGCHARMM * KCALTOIU, del, fma(4.0, dvd, dbd));
    } else {
        const int q = blockIdx.x - m * S, kind = mv.kind[q];
        const int warp = threadIdx.x >> 5, side = warp & 1;
        const CrdSrc src{A.pq, s_idx, s_xyz, side ? m : 0};
        for (int k = (q ? mv.kend[q - 1] : 0) + 32 * (warp >> 1) + (threadIdx.x & 31); k < mv.kend[q]; k += blockDim.x / 2) {
            const int t = terms[k];
            double e;
            if (kind == 0) e = bond_e(B.bonds[t], src, pbc, true);
            else if (kind == 1) e = angle_e(B.angles[t], src, pbc);
            else if (kind == 2) e = bond_e(B.ubs[t], src, pbc, false);
            else if (kind == 3) e = tors_e(B.dihes[t], src, pbc);
            else e = tors_e(B.imprs[t], src, pbc);
            dbd += side ? e : -e;
        }
    }
    const double sum = block_sum(dbd, s_sum);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = sum;
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {   // uniform over the block
        __threadfence();
        double v = 0.0;
        for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) v += __ldcg(part + b);
        __syncthreads();
        v = block_sum(v, s_sum);
        if (threadIdx.x == 0) {
            out[0] = v;
            *ticket = 0u;
        }
    }
}

__device__ __forceinline__ void store_x64(ulonglong4_32a* x64, const double4_32a& p, const PbcDev& pbc, int sh, unsigned cls) {
    *x64 = make_ulonglong4_32a(to_fixed64(p.x, pbc.L[0], pbc.rL[0], sh), to_fixed64(p.y, pbc.L[1], pbc.rL[1], sh),
                               to_fixed64(p.z, pbc.L[2], pbc.rL[2], sh), cls);
}

// A thread per coordinate: a coordinate's mirrors are some 25 dependent FP64 operations, at 64 cycles each.
__global__ void k_commit(int m, const int* idx, const double* xyz, double4_32a* pq, uint4* fx, ulonglong4_32a* x64,
                         int sh, PbcDev pbc, const __grid_constant__ MoveInline inl) {
    if (inl.m > 0) { idx = inl.idx; xyz = inl.xyz; }
    const int t = blockIdx.x * blockDim.x + threadIdx.x, k = t / 3, c = t - 3 * k;
    if (k >= m) return;
    const int a = idx[k];
    const double v = xyz[t];
    reinterpret_cast<double*>(pq + a)[c] = v;
    if (pbc.type != 0) {
        reinterpret_cast<uint32_t*>(fx + a)[c] = to_fixed(v, pbc.rL[c]);
        if (x64) reinterpret_cast<unsigned long long*>(x64 + a)[c] = to_fixed64(v, pbc.L[c], pbc.rL[c], sh);
    }
}

// Fixed-point mirrors of an atom from its FP64 master; w carries the atom's parameter class.
__device__ __forceinline__ void store_mirrors(int i, const double4_32a& p, unsigned cls, uint4* fx, ulonglong4_32a* x64, int sh,
                                              const PbcDev& pbc) {
    uint4 f;
    if (pbc.type != 0) { f.x = to_fixed(p.x, pbc.rL[0]); f.y = to_fixed(p.y, pbc.rL[1]); f.z = to_fixed(p.z, pbc.rL[2]); }
    else { f.x = f.y = f.z = 0; }
    f.w = cls;
    fx[i] = f;
    if (x64) store_x64(x64 + i, p, pbc, sh, cls);
}

__global__ void k_fix_all(int n, const double4_32a* __restrict__ pq, const int* __restrict__ cls_of, uint4* fx,
                          ulonglong4_32a* x64, int sh, PbcDev pbc) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) store_mirrors(i, pq[i], (unsigned)cls_of[i], fx, x64, sh, pbc);
}

// New coordinates of every atom, x, y and z after one another in page-locked host memory (read once,
// coalesced, over the host link): the masters and their mirrors.
__global__ void k_take_coords(int n, const double* __restrict__ xyz, double4_32a* pq, const int* __restrict__ cls_of, uint4* fx,
                              ulonglong4_32a* x64, int sh, PbcDev pbc) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4_32a p = make_double4_32a(xyz[i], xyz[n + i], xyz[2 * (size_t)n + i], pq[i].w);
    pq[i] = p;
    store_mirrors(i, p, (unsigned)cls_of[i], fx, x64, sh, pbc);
}

// ==========================================================================================
// Host side of the engine.
template <typename T>
static int dalloc(T** p, size_t count) {
    *p = nullptr;
    if (count == 0) count = 1;
    cudaError_t e = cudaMalloc((void**)p, count * sizeof(T));
    if (e != cudaSuccess) {
        cudaGetLastError();   // reported here, not left for the next call's launches
        return fail(MCG_ECUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e));
    }
    return MCG_OK;
}

template <typename T>
static int dupload(T** p, const std::vector<T>& v, cudaStream_t st) {
    int rc = dalloc(p, v.size());
    if (rc) return rc;
    if (!v.empty()) CK(cudaMemcpyAsync(*p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
    return MCG_OK;
}

SingleEngine::~SingleEngine() { release(); }

void SingleEngine::release() {
    void* ptrs[] = {d_pq, d_es, d_es14, d_fx, d_esf, d_esf14, d_qf, d_prmf, d_frozen, d_xs, d_xd, d_fxs, d_fxd, d_p14, d_c14s,
                    d_c14d, d_bonds, d_ubs, d_angles, d_dihes, d_imprs, d_nbr, d_nup, d_nlo, d_cell_of,
                    d_cell_count, d_cell_start, d_cell_fill, d_task_start, d_tasks, d_cell_atoms, d_cell_pos, d_home, d_part, d_ticket, d_maxrow,
                    d_stage, d_prn, d_pnup, d_pkept, d_cls_of, d_cls, d_x64, d_pair64};
    for (void* p : ptrs) if (p) cudaFree(p);
    for (cudaEvent_t& e : ev_prune) if (e) { cudaEventDestroy(e); e = nullptr; }
    if (h_stage) cudaFreeHost(h_stage);
    host_x = host_y = host_z = nullptr;   // inside h_stage
    if (h_map) cudaFreeHost(h_map);
    h_map = nullptr; d_map = nullptr;
    if (stream) cudaStreamDestroy(stream);
    d_pq = nullptr; stream = nullptr; h_stage = nullptr;
}

int SingleEngine::init(const HostSystem& h) {
    hs = h;
    n = hs.n;
    any_frozen = std::any_of(hs.frozen.begin(), hs.frozen.end(), [](uint8_t f) { return f != 0; });
    CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    pbc.type = hs.pbc;
    for (int k = 0; k < 3; k++) { pbc.L[k] = hs.L[k]; pbc.rL[k] = hs.rL[k]; }
    cut.mode = hs.cut;
    cut.c2 = hs.rc * hs.rc;
    cut.n2 = hs.ron * hs.ron;
    {
        double d = cut.c2 - cut.n2;
        cut.sw2 = 1. / (d * d * d);
    }
    cut.c2f = (float)cut.c2; cut.n2f = (float)cut.n2; cut.sw2f = (float)cut.sw2;
    std::vector<double4_32a> pq(n);
    std::vector<double2> es(n), es14(n);
    std::vector<float2> esf(n), esf14(n), qf(n);
    std::vector<float4> prmf(n);
    for (int i = 0; i < n; i++) {
        pq[i] = make_double4_32a(hs.x[i], hs.y[i], hs.z[i], hs.q[i]);
        es[i] = make_double2(hs.eps[i], hs.sig[i]);
        es14[i] = make_double2(hs.eps14[i], hs.sig14[i]);
        esf[i] = make_float2((float)hs.eps[i], (float)hs.sig[i]);
        esf14[i] = make_float2((float)hs.eps14[i], (float)hs.sig14[i]);
        float qh = (float)hs.q[i];
        qf[i] = make_float2(qh, (float)(hs.q[i] - (double)qh));
        prmf[i] = make_float4(qf[i].x, qf[i].y, esf[i].x, esf[i].y);
    }
    // parameter classes: the distinct (q hi, q lo, eps, sig) of the mixed pair kernel, in first-seen
    // order; more than CLS_MAX (CLS64_MAX) classes leave the table empty (the kernel gathers per atom)
    std::vector<int> cls_of(n, 0);
    std::vector<float4> cls;
    std::vector<Fix64Pair> pair64;
    if (uses_fix64()) {   // FP64: the distinct (q, eps, sig) and the products of every pair of them
        fix64 = hs.cut == MCG_CUT_SWITCH ? fix64_geom(hs.L, hs.rc, hs.ron) : fix64_geom_full(hs.L);
        std::map<std::array<double, 3>, int> seen;
        std::vector<std::array<double, 3>> par;
        for (int i = 0; i < n && (int)par.size() <= CLS64_MAX; i++) {
            const std::array<double, 3> key{hs.q[i], hs.eps[i], hs.sig[i]};
            auto it = seen.find(key);
            if (it == seen.end()) {
                it = seen.emplace(key, (int)par.size()).first;
                par.push_back(key);
            }
            cls_of[i] = it->second;
        }
        if ((int)par.size() <= CLS64_MAX) {
            ncls64 = (int)par.size();
            for (const auto& a : par)
                for (const auto& b : par) pair64.push_back(fix64_pair(a[0], a[1], a[2], b[0], b[1], b[2], fix64.leff));
        } else {
            std::fill(cls_of.begin(), cls_of.end(), 0);
        }
    } else {
        std::map<std::array<uint32_t, 4>, int> seen;
        for (int i = 0; i < n && (int)cls.size() <= CLS_MAX; i++) {
            std::array<uint32_t, 4> key;
            memcpy(key.data(), &prmf[i], sizeof(float4));
            auto it = seen.find(key);
            if (it == seen.end()) {
                it = seen.emplace(key, (int)cls.size()).first;
                cls.push_back(prmf[i]);
            }
            cls_of[i] = it->second;
        }
        if ((int)cls.size() > CLS_MAX) {
            cls.clear();
            std::fill(cls_of.begin(), cls_of.end(), 0);
        }
        ncls = (int)cls.size();
    }
    int rc;
    if ((rc = dupload(&d_cls_of, cls_of, stream)) || (rc = dupload(&d_cls, cls, stream))) return rc;
    if ((rc = dupload(&d_pq, pq, stream)) || (rc = dupload(&d_es, es, stream)) || (rc = dupload(&d_es14, es14, stream)) ||
        (rc = dupload(&d_esf, esf, stream)) || (rc = dupload(&d_esf14, esf14, stream)) || (rc = dupload(&d_qf, qf, stream)) ||
        (rc = dupload(&d_prmf, prmf, stream)) ||
        (rc = dupload(&d_frozen, hs.frozen, stream)) || (rc = dupload(&d_xs, hs.exclStart, stream)) ||
        (rc = dupload(&d_xd, hs.exclData, stream)) || (rc = dupload(&d_fxs, hs.fexclStart, stream)) ||
        (rc = dupload(&d_fxd, hs.fexclData, stream)))
        return rc;
    if ((rc = dalloc(&d_fx, n))) return rc;
    if (uses_fix64() && ((rc = dalloc(&d_x64, n)) || (ncls64 > 0 && (rc = dupload(&d_pair64, pair64, stream))))) return rc;
    if (uses_pair_variants() && ncls > 0) {   // groups of the group-pair kernels (residue runs of <= 4 atoms)
        if ((rc = grp.setup(hs.resid))) return rc;
        grp_setup = true;
    }
    // 1-4 pairs and their per-atom CSR (both directions) for the ΔE kernel
    n14 = (int)hs.pairs14.size() / 2;
    std::vector<int2> p14(n14);
    std::vector<std::vector<int>> adj(n);
    for (int k = 0; k < n14; k++) {
        p14[k] = make_int2(hs.pairs14[2 * k], hs.pairs14[2 * k + 1]);
        adj[p14[k].x].push_back(p14[k].y);
        adj[p14[k].y].push_back(p14[k].x);
    }
    std::vector<int> c14s(n + 1, 0), c14d;
    for (int i = 0; i < n; i++) { c14s[i] = (int)c14d.size(); c14d.insert(c14d.end(), adj[i].begin(), adj[i].end()); }
    c14s[n] = (int)c14d.size();
    if ((rc = dupload(&d_p14, p14, stream)) || (rc = dupload(&d_c14s, c14s, stream)) || (rc = dupload(&d_c14d, c14d, stream)))
        return rc;
    if ((rc = dupload(&d_bonds, hs.bonds, stream)) || (rc = dupload(&d_ubs, hs.ubs, stream)) ||
        (rc = dupload(&d_angles, hs.angles, stream)) || (rc = dupload(&d_dihes, hs.dihes, stream)) ||
        (rc = dupload(&d_imprs, hs.imprs, stream)))
        return rc;
    // per-atom bonded-term index for ΔE (kind, index)
    term_start.assign(n + 1, 0);
    std::vector<std::vector<int>> tl(n);
    auto addt = [&](int atom, int kind, int idx) { tl[atom].push_back(kind); tl[atom].push_back(idx); };
    for (int k = 0; k < (int)hs.bonds.size(); k++) { addt(hs.bonds[k].a, 0, k); addt(hs.bonds[k].b, 0, k); }
    for (int k = 0; k < (int)hs.angles.size(); k++) { const AngleT& a = hs.angles[k]; addt(a.a, 1, k); addt(a.b, 1, k); addt(a.c, 1, k); }
    for (int k = 0; k < (int)hs.ubs.size(); k++) { addt(hs.ubs[k].a, 2, k); addt(hs.ubs[k].b, 2, k); }
    for (int k = 0; k < (int)hs.dihes.size(); k++) { const TorsT& t = hs.dihes[k]; addt(t.a, 3, k); addt(t.b, 3, k); addt(t.c, 3, k); addt(t.d, 3, k); }
    for (int k = 0; k < (int)hs.imprs.size(); k++) { const TorsT& t = hs.imprs[k]; addt(t.a, 4, k); addt(t.b, 4, k); addt(t.c, 4, k); addt(t.d, 4, k); }
    term_data.clear();
    for (int i = 0; i < n; i++) { term_start[i] = (int)term_data.size() / 2; term_data.insert(term_data.end(), tl[i].begin(), tl[i].end()); }
    term_start[n] = (int)term_data.size() / 2;
    // scratch: partial sums and the ΔE ticket
    ntile = (n + TILE - 1) / TILE;
    size_t nparts = std::max<size_t>({(size_t)152 * std::max(A64_CTAS, ALLMIX_CTAS), (size_t)ntile * (ntile + 1) / 2, (size_t)MAX_MOVED + 1});
    part_cap = nparts * 3 + 2 * 64 + 5 * BD_BLOCKS + 16;
    if ((rc = dalloc(&d_part, part_cap)) || (rc = dalloc(&d_ticket, 2)) ||
        (rc = dalloc(&d_maxrow, 3)))
        return rc;
    CK(cudaMemsetAsync(d_ticket, 0, 2 * sizeof(unsigned), stream));
    // staging for moves: idx (sorted), xyz, terms
    stage_bytes = (size_t)MAX_MOVED * (4 + 24) + 64 * 1024 * 8;
    CK(cudaMallocHost(&h_stage, stage_bytes + sizeof(double) * 3 * (size_t)n));
    host_x = (double*)((char*)h_stage + stage_bytes);
    host_y = host_x + n;
    host_z = host_y + n;
    std::copy(hs.x.begin(), hs.x.end(), host_x);
    std::copy(hs.y.begin(), hs.y.end(), host_y);
    std::copy(hs.z.begin(), hs.z.end(), host_z);
    // results the host reads after a sync: de at [0, 4), the ten energy terms at [8, 18)
    CK(cudaHostAlloc((void**)&h_map, 32 * sizeof(double), cudaHostAllocMapped));
    CK(cudaHostGetDevicePointer((void**)&d_map, h_map, 0));
    if ((rc = dalloc((char**)&d_stage, stage_bytes))) return rc;
    k_fix_all<<<(n + 255) / 256, 256, 0, stream>>>(n, d_pq, d_cls_of, d_fx, d_x64, fix64.sh, pbc);
    CK(cudaGetLastError());
    if (hs.cut == MCG_CUT_SWITCH) {
        if ((rc = build_list())) return rc;
    }
    CK(cudaStreamSynchronize(stream));
    return MCG_OK;
}

// The switched nonbonded kernel over the half list (FP64, or mixed: the dedicated pair kernel for
// periodic boxes).
int SingleEngine::launch_nonbonded(double* nbp) {
    AtomsDev A = atoms();
    if (uses_fix64()) {
        const int blocks = std::min(NB_BLOCKS, (n + NB_THREADS / 32 - 1) / (NB_THREADS / 32));
#define MCG_LIST64(ISO_, TAB_)                                                                                        \
    k_energy_list64<ISO_, TAB_><<<blocks, NB_THREADS, 0, stream>>>(A, fix64, pbc, cut, n, d_nbr, d_nup, cap, nbp)
        if (fix64.iso && ncls64) MCG_LIST64(true, true);
        else if (fix64.iso) MCG_LIST64(true, false);
        else if (ncls64) MCG_LIST64(false, true);
        else MCG_LIST64(false, false);
#undef MCG_LIST64
        return blocks;
    }
    if (hs.prec == MCG_PREC_FP64)
        k_energy_list<PREC_F64><<<NB_BLOCKS, NB_THREADS, 0, stream>>>(A, n, pbc, cut, d_nbr, d_nup, cap, nbp);
    else if (pbc.type != 0)
        return launch_pair_variant(pair_variant < 0 ? 0 : pair_variant, nbp);
    else
        k_energy_list<PREC_MIX><<<NB_BLOCKS, NB_THREADS, 0, stream>>>(A, n, pbc, cut, d_nbr, d_nup, cap, nbp);
    return NB_BLOCKS;
}

static const int kListVariants = 4;
static const int kGroupFirst = kListVariants + ClusterPairs::kVariants;   // first group-pair variant

int SingleEngine::pair_kernel_count() { return kGroupFirst + GroupPairs::kVariants; }

int SingleEngine::launch_pair_variant(int v, double* nbp) {
    if (v >= kGroupFirst)
        return grp.launch_energy(stream, v - kGroupFirst, d_fx, d_cls, ncls, group_geom(), nbp);
    if (v >= kListVariants) {
        launches += 1;   // the pack kernel in front of the cluster kernel
        return clp.launch_energy(stream, v - kListVariants, d_fx, d_prmf, cluster_geom(), nbp);
    }
    AtomsDev A = atoms();
    const double inv_f1 = cluster_geom().inv_f1;
    // the pruned rows when they are current (prepare_pair_kernel prunes before every launch that
    // needs it), else the Verlet rows
    const bool pr = prune_buf > 0.0 && !prune_dirty && d_prn;
    const int* rows = pr ? d_prn : d_nbr;
    const int* lens = pr ? d_pnup : d_nup;
    // cubic boxes: r^2 in fixed-point units scaled by the float-float square of the unit length
    const bool iso = A.Ls[0] == A.Ls[1] && A.Ls[1] == A.Ls[2] && A.Lsl[0] == A.Lsl[1] && A.Lsl[1] == A.Lsl[2];
    const double l2 = (double)A.Ls[0] + (double)A.Lsl[0];
    const double l2sq = l2 * l2;
    const float L2h = (float)l2sq, L2l = (float)(l2sq - (double)L2h);
    int blocks = 0;
#define MCG_LIST_MIX_ONE(U_, B_, ISO_, TY_)                                                                  \
    blocks = 152 * B_;                                                                                        \
    k_energy_list_mix<U_, B_, ISO_, TY_><<<152 * B_, NB_THREADS, TY_ ? sizeof(float4) * ncls : 0, stream>>>( \
        d_fx, d_prmf, d_cls, ncls, n, A.Ls[0], A.Ls[1], A.Ls[2], A.Lsl[0], A.Lsl[1], A.Lsl[2], L2h, L2l, cut, inv_f1, \
        rows, lens, cap, nbp);
#define MCG_LIST_MIX(U_, B_)                                                                                   \
    if (iso && ncls > 0) { MCG_LIST_MIX_ONE(U_, B_, true, true) }                                             \
    else if (iso) { MCG_LIST_MIX_ONE(U_, B_, true, false) }                                                   \
    else if (ncls > 0) { MCG_LIST_MIX_ONE(U_, B_, false, true) }                                              \
    else { MCG_LIST_MIX_ONE(U_, B_, false, false) }
    // grids sized to the residency each variant asks for (NB_THREADS threads per CTA)
    switch (v) {
    case 0: MCG_LIST_MIX(4, 4) break;
    case 1: MCG_LIST_MIX(5, 4) break;
    case 2: MCG_LIST_MIX(3, 5) break;
    default: MCG_LIST_MIX(6, 4) break;
    }
#undef MCG_LIST_MIX
#undef MCG_LIST_MIX_ONE
    return blocks;
}

// Times every pair-kernel variant on the current system (3 launches each) and keeps the fastest;
// the cluster-pair variants take part when the cluster list was built.
void SingleEngine::tune_pair_kernel() {
    cudaEvent_t a, b;
    pair_variant = 0;
    if (cudaEventCreate(&a) != cudaSuccess) return;
    if (cudaEventCreate(&b) != cudaSuccess) { cudaEventDestroy(a); return; }
    float best = 3.0e38f;
    const int nv = pair_kernel_count();
    int timed = 0;
    for (int v = 0; v < nv; v++) {
        if (v >= kListVariants && v < kGroupFirst && !clp.ok) continue;
        if (v >= kGroupFirst && !grp.ok) continue;
        timed++;
        launch_pair_variant(v, d_part);
        cudaEventRecord(a, stream);
        for (int r = 0; r < 3; r++) launch_pair_variant(v, d_part);
        cudaEventRecord(b, stream);
        float ms = 0.f;
        if (cudaEventSynchronize(b) != cudaSuccess || cudaEventElapsedTime(&ms, a, b) != cudaSuccess) continue;
        if (ms < best) { best = ms; pair_variant = v; }
    }
    launches += 4 * timed;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
}

int SingleEngine::set_pair_kernel(int v) {
    if (v < -1 || v >= pair_kernel_count()) return fail(MCG_EINVAL, "pair-kernel variant out of range");
    if (v >= 0 && !uses_pair_variants())
        return fail(MCG_ENOTSUP, "pair-kernel variants apply to the mixed periodic switch energy");
    if (v >= kGroupFirst) {
        if (!grp_setup) return fail(MCG_ENOTSUP, "the group-pair kernels need the parameter-class table");
        int rc = ensure_pruned();
        if (!rc) rc = ensure_groups();
        if (rc) return rc;
        if (!grp.ok) return fail(MCG_ENOTSUP, "the group-pair rows could not be built for this system");
    } else if (v >= kListVariants) {
        int rc = ensure_clusters();
        if (rc) return rc;
        if (!clp.ok) return fail(MCG_ENOTSUP, "the cluster-pair list could not be built for this system");
    }
    pair_variant = v;
    return MCG_OK;
}

// The group-pair rows of the rows the per-atom list kernels read (pruned rows when pruning is on),
// rebuilt on first use after those rows changed.  A system whose group rows overflow the build's
// limits keeps the other kernels.
int SingleEngine::ensure_groups() {
    if (!grp_setup || !grp_dirty) return MCG_OK;
    if (int rc = need_list()) return rc;
    grp_dirty = false;
    const bool pr = prune_buf > 0.0 && !prune_dirty && d_prn;
    const int grc = grp.build(stream, pr ? d_prn : d_nbr, pr ? d_pnup : d_nup, cap);
    launches += grp.build_launches;
    grp.build_launches = 0;
    if (grc == MCG_ECUDA) return grc;
    if (grc != MCG_OK) set_error("");
    return MCG_OK;
}

GroupGeom SingleEngine::group_geom() const {
    const ClusterGeom C = cluster_geom();
    GroupGeom G;
    for (int k = 0; k < 3; k++) { G.Ls[k] = C.Ls[k]; G.Ll[k] = C.Ll[k]; }
    G.iso = G.Ls[0] == G.Ls[1] && G.Ls[1] == G.Ls[2] && G.Ll[0] == G.Ll[1] && G.Ll[1] == G.Ll[2];
    const double l2 = (double)G.Ls[0] + (double)G.Ll[0];
    const double l2sq = l2 * l2;
    G.L2h = (float)l2sq;
    G.L2l = (float)(l2sq - (double)G.L2h);
    G.c2 = C.c2;
    G.n2 = C.n2;
    G.k3 = C.k3;
    G.inv_f1 = C.inv_f1;
    G.D = C.c2 - C.n2;
    G.inv_p1 = 1.0 / (double)((G.D * G.D) * std::fmaf(G.D, -2.0f, 3.0f * G.D));
    const double lmin = std::min(pbc.L[0], std::min(pbc.L[1], pbc.L[2]));
    G.emax = (float)(0.5 * lmin - std::sqrt((double)C.c2) - 1e-3);
    return G;
}

int SingleEngine::group_stats(int64_t* groups, int64_t* entries, int64_t* mask_pairs) {
    *groups = *entries = *mask_pairs = 0;
    if (!grp_setup) return MCG_OK;
    int rc = ensure_pruned();
    if (!rc) rc = ensure_groups();
    if (rc) return rc;
    if (grp.ok) { *groups = grp.ngroup; *entries = grp.nentries; *mask_pairs = grp.nbits; }
    return MCG_OK;
}

bool SingleEngine::uses_pair_variants() const {
    return hs.prec == MCG_PREC_MIXED && pbc.type != 0 && hs.cut == MCG_CUT_SWITCH;
}

// The cluster-pair form of the current Verlet list, built on first use after a list build (the
// tuner's first timing, a cluster variant chosen, or the statistics asked for).  A system whose
// clusters do not fit the build's shared-memory limits keeps the per-atom list kernels only.
int SingleEngine::ensure_clusters() {
    if (!clp_dirty) return MCG_OK;
    if (int rc = need_list()) return rc;
    clp_dirty = false;
    const int crc = clp.build(stream, d_fx, n, hs.L, d_nbr, d_nup, d_nlo, cap);
    launches += clp.build_launches;
    clp.build_launches = 0;
    if (crc == MCG_OK) return ensure_part((size_t)2 * clp.ncl + 2 * 64 + 5 * BD_BLOCKS + 16);
    if (crc == MCG_ECUDA) return crc;
    set_error("");
    return MCG_OK;
}

// Before a launch of the mixed periodic switch energy: the first use times every variant (the
// cluster list built for it); a chosen cluster variant has its list brought up to date.  Runs
// before the caller takes the partial-sum buffer, which the cluster build may grow.
int SingleEngine::prepare_pair_kernel() {
    int rc = need_list();
    if (rc || !uses_pair_variants()) return rc;
    if ((rc = ensure_pruned())) return rc;
    if (pair_variant < 0) {
        if ((rc = ensure_clusters())) return rc;
        if ((rc = ensure_groups())) return rc;
        tune_pair_kernel();
    }
    if (pair_variant >= kGroupFirst) {
        if ((rc = ensure_groups())) return rc;
        if (!grp.ok) pair_variant = 0;
    } else if (pair_variant >= kListVariants) {
        if ((rc = ensure_clusters())) return rc;
        if (!clp.ok) pair_variant = 0;
    }
    return MCG_OK;
}

// Prunes the Verlet rows for the pair kernel when they are stale: after a list build, a change of
// the buffer, or once an atom has moved more than half the buffer (less 1e-3 A) from its position
// at the last prune (host-side positions, minimum image).  The prune runs on the handle's stream
// between event records, so its device time can be read back without a synchronisation here.
int SingleEngine::ensure_pruned() {
    if (prune_buf <= 0.0 || !prune_dirty) return MCG_OK;
    int rc = need_list();
    if (rc) return rc;
    if (prn_cap != cap) {   // the pruned rows share the Verlet rows' stride
        if (d_prn) cudaFree(d_prn);
        d_prn = nullptr;
        prn_cap = 0;
        if ((rc = dalloc(&d_prn, (size_t)n * cap))) return rc;
        prn_cap = cap;
    }
    if (!d_pnup && (rc = dalloc(&d_pnup, n))) return rc;
    if (!d_pkept && (rc = dalloc(&d_pkept, 1))) return rc;
    for (cudaEvent_t& e : ev_prune)
        if (!e) CK(cudaEventCreate(&e));
    const AtomsDev A = atoms();
    const double rp = hs.rc + prune_buf;
    const float rp2 = (float)(rp * rp * (1.0 + 1e-5));   // above any FP32 rounding of r^2
    CK(cudaMemsetAsync(d_pkept, 0, sizeof(unsigned long long), stream));
    CK(cudaEventRecord(ev_prune[0], stream));
    k_prune_rows<<<NB_BLOCKS, NB_THREADS, 0, stream>>>(d_fx, n, A.Ls[0], A.Ls[1], A.Ls[2], A.Lsl[0], A.Lsl[1], A.Lsl[2],
                                                       rp2, d_nbr, d_nup, cap, d_prn, d_pnup, d_pkept);
    CK(cudaGetLastError());
    CK(cudaEventRecord(ev_prune[1], stream));
    prune_x.assign(host_x, host_x + n);
    prune_y.assign(host_y, host_y + n);
    prune_z.assign(host_z, host_z + n);
    const double lim = std::max(0.0, 0.5 * prune_buf - 1e-3);
    prune_lim2 = lim * lim;
    prune_dirty = false;
    grp_dirty = grp_setup;    // the group rows follow the pruned rows
    prunes++;
    launches += 1;
    return MCG_OK;
}

// An atom's coordinates changed on the host side: the pruned rows go stale once it is further
// than the limit from where it was at the last prune.
void SingleEngine::note_moved(int a) {
    double d2 = 0.0;
    const double p[3] = {host_x[a] - prune_x[a], host_y[a] - prune_y[a], host_z[a] - prune_z[a]};
    for (int k = 0; k < 3; k++) {
        const double d = p[k] - hs.L[k] * std::nearbyint(p[k] / hs.L[k]);
        d2 += d * d;
    }
    if (!(d2 <= prune_lim2)) prune_dirty = true;
}

int SingleEngine::set_prune_buffer(double buffer) {
    if (!(buffer >= 0.0) || !std::isfinite(buffer)) return fail(MCG_EINVAL, "prune buffer must be finite and >= 0");
    if (buffer > 0.0 && !uses_pair_variants())
        return fail(MCG_ENOTSUP, "pruning applies to the mixed periodic switch energy");
    prune_buf = buffer;
    prune_dirty = true;
    grp_dirty = grp_setup;
    return MCG_OK;
}

int SingleEngine::prune_stats(int64_t* entries, int64_t* nprunes, float* last_ms) {
    *entries = 0;
    *nprunes = prunes;
    *last_ms = 0.f;
    if (prunes == 0 || !d_pkept) return MCG_OK;
    unsigned long long k = 0;
    CK(cudaMemcpyAsync(&k, d_pkept, sizeof(k), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    CK(cudaEventElapsedTime(last_ms, ev_prune[0], ev_prune[1]));
    *entries = (int64_t)k;
    return MCG_OK;
}

int SingleEngine::cluster_stats(int64_t* clusters, int64_t* cluster_pairs, int64_t* mask_pairs) {
    *clusters = *cluster_pairs = *mask_pairs = 0;
    if (!uses_pair_variants()) return MCG_OK;
    int rc = ensure_clusters();
    if (rc) return rc;
    if (clp.ok) { *clusters = clp.ncl; *cluster_pairs = clp.npairs; *mask_pairs = clp.nbits; }
    return MCG_OK;
}

ClusterGeom SingleEngine::cluster_geom() const {
    ClusterGeom G;
    AtomsDev A = atoms();
    for (int k = 0; k < 3; k++) {
        G.Ls[k] = A.Ls[k];
        G.Ll[k] = A.Lsl[k];
        G.Lf[k] = (float)hs.L[k];
        G.iLf[k] = (float)(1.0 / hs.L[k]);
        G.lim[k] = (float)(hs.L[k] - hs.rc - 0.01);
    }
    G.c2 = cut.c2f;
    G.n2 = cut.n2f;
    G.k3 = cut.c2f - 3.0f * cut.n2f;
    const float pr = (float)(hs.rc + 0.01);
    G.prune2 = pr * pr;
    // the FP32 switch polynomial at u = ron^2, as the kernel forms it
    const float a = G.c2 - G.n2;
    const float aa = a * a;
    const float bb = std::fmaf(2.0f, G.n2, G.k3);
    const float f1 = aa * bb;
    G.inv_f1 = 1.0 / (double)f1;
    return G;
}

int SingleEngine::ensure_part(size_t count) {
    if (count <= part_cap) return MCG_OK;
    if (d_part) cudaFree(d_part);
    d_part = nullptr;
    part_cap = 0;
    int rc = dalloc(&d_part, count);
    if (rc) return rc;
    part_cap = count;
    return MCG_OK;
}

int SingleEngine::time_nonbonded(int reps, float* ms) {
    if (hs.cut != MCG_CUT_SWITCH) return fail(MCG_ENOTSUP, "the pair-kernel timing covers the switch mode");
    {
        int rc = prepare_pair_kernel();
        if (rc) return rc;
    }
    cudaEvent_t a, b;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    launch_nonbonded(d_part);                       // warm
    CK(cudaEventRecord(a, stream));
    for (int r = 0; r < reps; r++) launch_nonbonded(d_part);
    CK(cudaEventRecord(b, stream));
    CK(cudaEventSynchronize(b));
    CK(cudaEventElapsedTime(ms, a, b));
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    launches += reps + 1;
    return MCG_OK;
}

int SingleEngine::time_nonbonded_flushed(int reps, float* ms) {
    if (hs.cut != MCG_CUT_SWITCH) return fail(MCG_ENOTSUP, "the pair-kernel timing covers the switch mode");
    {
        int rc = prepare_pair_kernel();
        if (rc) return rc;
    }
    constexpr size_t kFlush = (size_t)256 << 20;   // twice the L2
    unsigned char* junk = nullptr;
    CK(cudaMalloc(&junk, kFlush));
    cudaEvent_t a, b;
    if (cudaEventCreate(&a) != cudaSuccess) { cudaFree(junk); return fail(MCG_ECUDA, "cudaEventCreate"); }
    if (cudaEventCreate(&b) != cudaSuccess) { cudaEventDestroy(a); cudaFree(junk); return fail(MCG_ECUDA, "cudaEventCreate"); }
    float total = 0.0f;
    cudaError_t e = cudaSuccess;
    for (int r = 0; r < reps && e == cudaSuccess; r++) {
        e = cudaMemsetAsync(junk, r & 0xff, kFlush, stream);
        if (e == cudaSuccess) e = cudaEventRecord(a, stream);
        if (e == cudaSuccess) launch_nonbonded(d_part);
        if (e == cudaSuccess) e = cudaEventRecord(b, stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(b);
        float t = 0.0f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&t, a, b);
        total += t;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(junk);
    if (e != cudaSuccess) return fail(MCG_ECUDA, std::string("flushed pair-kernel timing: ") + cudaGetErrorString(e));
    launches += reps;
    *ms = total;
    return MCG_OK;
}

AtomsDev SingleEngine::atoms() const {
    AtomsDev A;
    A.x64 = d_x64; A.pair64 = d_pair64; A.ncls64 = ncls64;
    A.pq = d_pq; A.es = d_es; A.es14 = d_es14; A.fx = d_fx; A.esf = d_esf; A.esf14 = d_esf14; A.qf = d_qf;
    for (int k = 0; k < 3; k++) {
        const double ls = hs.L[k] / 4294967296.0;
        A.Ls[k] = (float)ls;
        A.Lsl[k] = (float)(ls - (double)A.Ls[k]);
    }
    return A;
}

BondedDev SingleEngine::bonded() const {
    return BondedDev{d_bonds, (int)hs.bonds.size(), d_ubs, (int)hs.ubs.size(), d_angles, (int)hs.angles.size(),
                     d_dihes, (int)hs.dihes.size(), d_imprs, (int)hs.imprs.size()};
}

// Rows that a failed build left short (no memory for longer ones) are not read: their counts run past them.
int SingleEngine::need_list() const {
    return hs.cut != MCG_CUT_SWITCH || list_ok ? MCG_OK : fail(MCG_ECUDA, "no Verlet list: the last list update failed");
}

int SingleEngine::build_list() {
    const double rl = hs.rc + hs.dcut;
    Grid g;
    g.periodic = hs.pbc != MCG_PBC_NONE;
    double ext[3];
    if (g.periodic) {
        for (int k = 0; k < 3; k++) { ext[k] = hs.L[k]; g.lo[k] = 0; g.inv[k] = 0; }
    } else {
        for (int k = 0; k < 3; k++) {
            const double* c = k == 0 ? host_x : (k == 1 ? host_y : host_z);
            double lo = *std::min_element(c, c + n), hi = *std::max_element(c, c + n);
            ext[k] = std::max(hi - lo, 1e-6);
            g.lo[k] = lo;
            g.inv[k] = 1.0 / ext[k] * (1.0 - 1e-12);
        }
    }
    for (int k = 0; k < 3; k++) g.nc[k] = std::max(1, (int)std::floor(2.0 * ext[k] / rl));
    while ((long long)g.nc[0] * g.nc[1] * g.nc[2] > (1 << 20))
        for (int k = 0; k < 3; k++) g.nc[k] = std::max(1, g.nc[k] / 2);
    for (int k = 0; k < 3; k++) g.csf[k] = (float)(ext[k] / g.nc[k] * (1.0 - 1e-6));
    int ncell = g.nc[0] * g.nc[1] * g.nc[2];
    const bool iso = g.periodic && hs.L[0] == hs.L[1] && hs.L[1] == hs.L[2];
    // home atoms that share a walk: four share more of it, two leave fewer warps idle in a small system.  A whole
    // update with two and four, us: 33, 37 (864 argon atoms), 42, 39 (4,000 argon), 51, 57 (1,800 water atoms), 83, 86
    // (4,500), 100, 106 (6,000), 104, 113 (8,193), 158, 120 (9,600), 167, 136 (12,288), 185, 182 (18,000), 751, 649
    // (100,002); eight were slower up to 36,000.  The line is at 8,192
    const int run = n < 8192 ? 2 : 4;
    int rc;
    if (ncell > ncell_cap) {
        ncell_cap = 0;             // an allocation that fails leaves them to the next build
        int** const per_cell[] = {&d_cell_count, &d_cell_start, &d_cell_fill, &d_task_start};
        for (int** p : per_cell) {
            if (*p) cudaFree(*p);
            if ((rc = dalloc(p, ncell + 1))) return rc;
        }
        CK(cudaMemsetAsync(d_cell_count, 0, sizeof(int) * (ncell + 1), stream));   // every scan leaves it zero
        if (d_tasks) cudaFree(d_tasks);
        if ((rc = dalloc(&d_tasks, (size_t)n / 2 + ncell + 1))) return rc;
        ncell_cap = ncell;
    }
    if (!d_cell_of) {
        if ((rc = dalloc(&d_cell_of, n)) || (rc = dalloc(&d_cell_atoms, n)) || (rc = dalloc(&d_cell_pos, n)) || (rc = dalloc(&d_home, n)) || (rc = dalloc(&d_nup, n)) || (rc = dalloc(&d_nlo, n)))
            return rc;
    }
    if (cap == 0) {
        // initial capacity from the density of the list sphere, grown on overflow below
        double vol = g.periodic ? hs.L[0] * hs.L[1] * hs.L[2] : 0.0;
        double est = g.periodic ? (4.0 / 3.0 * PI * rl * rl * rl) * n / vol : n;
        cap = (int)std::min<double>(n, est * 1.3 + 64);
        cap = (cap + 31) & ~31;
    }
    if (!d_nbr && (rc = dalloc(&d_nbr, (size_t)n * cap))) {
        cap = 0;
        return rc;
    }
    list_ok = false;   // until the rows are whole
    ListParams lp{rl * rl, cap, hs.maxExclSpan, {0, 0, 0}, 0.f, 0.f, 0.f, any_frozen};
    {
        // equal box lengths: r^2 stays in the mirrors' own units
        double t = hs.rc + hs.dcut;  // (cutoff + deltacut)^2 as List_nonBonded.cpp:842-843
        lp.cutnb2 = t * t;
        const AtomsDev A = atoms();
        for (int k = 0; k < 3; k++) lp.Ls[k] = g.periodic ? A.Ls[k] : 1.0f;
        const double unit2 = iso ? (hs.L[0] / 4294967296.0) * (hs.L[0] / 4294967296.0) : 1.0;
        lp.lo2 = (float)(lp.cutnb2 * (1.0 - 1e-4) / unit2);
        lp.hi2 = (float)(lp.cutnb2 * (1.0 + 1e-4) / unit2);
        lp.reach2 = (float)(lp.cutnb2 * (1.0 + 1e-5) + 1e-2);
        if (!g.periodic && std::max(ext[0], std::max(ext[1], ext[2])) > LIST_EXTENT * t) { lp.lo2 = -1.0f; lp.hi2 = HUGE_VALF; }
    }
    for (int attempt = 0; attempt < 3; attempt++) {
        cudaLaunchAttribute after[1];
        after[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        after[0].val.programmaticStreamSerializationAllowed = 1;
        auto launch = [&](auto kernel, int blocks, int threads, auto... args) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(blocks);
            cfg.blockDim = dim3(threads);
            cfg.stream = stream;
            cfg.attrs = after;
            cfg.numAttrs = 1;
            return cudaLaunchKernelEx(&cfg, kernel, args...);
        };
        CK(launch(k_cell_assign, (n + 255) / 256, 256, d_pq, n, pbc, g, d_cell_of, d_cell_count));
        CK(launch(k_cell_scan, 1, 1024, d_cell_count, ncell, run, d_cell_start, d_cell_fill, d_task_start, d_maxrow));
        CK(launch(k_cell_scatter, (n + 255) / 256, 256, d_cell_of, n, d_cell_start, d_cell_fill, d_cell_atoms));
        // a CTA per cell: 128 threads, or 512 where cells hold hundreds of atoms (3,000 in one cell: 82 us an update with
        // 512 threads, 100 with 128)
        CK(launch(k_cell_sort, ncell, n / ncell >= 256 ? 512 : 128, d_cell_start, d_task_start, ncell, run, d_fx, d_pq, g, d_cell_atoms, d_cell_pos, d_home, d_tasks));
        const int blocks = std::min((n / run + ncell + ROW_WARPS - 1) / ROW_WARPS, 152 * ROW_CTAS);
#define MCG_ROWS(A_, P_, I_)                                                                                          \
    CK(launch(k_build_rows<A_, P_, I_>, blocks, 32 * ROW_WARPS, d_pq, d_cell_pos, d_frozen, pbc, g, lp, d_cell_start, \
              d_task_start, ncell, d_home, d_tasks, d_xs, d_xd, d_nbr, d_nup, d_nlo, d_maxrow, (int*)(d_map + 24)))
        if (!g.periodic && run == 4) MCG_ROWS(4, false, true);
        else if (!g.periodic) MCG_ROWS(2, false, true);
        else if (iso && run == 4) MCG_ROWS(4, true, true);
        else if (iso) MCG_ROWS(2, true, true);
        else if (run == 4) MCG_ROWS(4, true, false);
        else MCG_ROWS(2, true, false);
#undef MCG_ROWS
        CK(cudaStreamSynchronize(stream));
        const int maxrow = *(volatile int*)(h_map + 24);
        last_max_row = maxrow;
        if (maxrow <= cap) {
            clp_dirty = uses_pair_variants();   // the cluster form follows on first use
            prune_dirty = true;                 // and so do the pruned rows
            grp_dirty = grp_setup;              // and the group rows
            list_ok = true;
            return MCG_OK;
        }
        cudaFree(d_nbr);
        d_nbr = nullptr;
        cap = ((int)(maxrow * 1.1) + 32 + 31) & ~31;
        lp.cap = cap;
        if ((rc = dalloc(&d_nbr, (size_t)n * cap))) {
            cap = 0;               // the next build begins at the estimate again
            return rc;
        }
    }
    return fail(MCG_ECAPACITY, "Verlet row capacity could not be grown");
}

int SingleEngine::energy(double ener[10]) {
    if (hs.cut == MCG_CUT_SWITCH) {
        int rc = prepare_pair_kernel();
        if (rc) return rc;
    }
    AtomsDev A = atoms();
    double* nbp = d_part;
    int nnb = 0;
    if (hs.cut == MCG_CUT_SWITCH) {
        nnb = launch_nonbonded(nbp);
    } else {
        const long long units = all_units(n);
        if (uses_fix64()) {
            nnb = (int)std::min<long long>(units, 152 * A64_CTAS);
#define MCG_ALL64(ISO_, TAB_)                                                                                         \
    k_energy_all64<ISO_, TAB_><<<nnb, ALL_I, 0, stream>>>(A, fix64, pbc, cut, n, d_fxs, d_fxd, units, nbp)
            if (fix64.iso && ncls64) MCG_ALL64(true, true);
            else if (fix64.iso) MCG_ALL64(true, false);
            else if (ncls64) MCG_ALL64(false, true);
            else MCG_ALL64(false, false);
#undef MCG_ALL64
        } else if (hs.prec == MCG_PREC_FP64) {
            nnb = ntile * (ntile + 1) / 2;
            k_energy_all<<<nnb, TILE, 0, stream>>>(A, n, pbc, cut, d_fxs, d_fxd, ntile, nbp);
        } else {
            nnb = (int)std::min<long long>(units, 152 * ALLMIX_CTAS);
            if (pbc.type != 0) k_energy_all_mix<true><<<nnb, ALL_I, 0, stream>>>(A, n, d_fxs, d_fxd, units, nbp);
            else k_energy_all_mix<false><<<nnb, ALL_I, 0, stream>>>(A, n, d_fxs, d_fxd, units, nbp);
        }
    }
    const BondedDev B = bonded();
    const int nterm = B.nb + B.na + B.nu + B.nd + B.ni;
    const int nbd = std::min(BD_BLOCKS, (nterm + 255) / 256), n14b = std::min(64, (n14 + 255) / 256);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::max(1, nbd + n14b));
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute beside[1];
    beside[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    beside[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = beside;
    cfg.numAttrs = 1;
    double* rest = nbp + 2 * (size_t)nnb;
    if (hs.prec == MCG_PREC_FP64)
        CK(cudaLaunchKernelEx(&cfg, k_energy_tail<PREC_F64>, B, nbd, A, pbc, cut, (const int2*)d_p14, n14, n14b,
                              (const double*)nbp, nnb, rest, d_ticket + 1, d_map + 8));
    else
        CK(cudaLaunchKernelEx(&cfg, k_energy_tail<PREC_MIX>, B, nbd, A, pbc, cut, (const int2*)d_p14, n14, n14b,
                              (const double*)nbp, nnb, rest, d_ticket + 1, d_map + 8));
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(stream));
    for (int k = 0; k < 10; k++) ener[k] = ((volatile double*)h_map)[8 + k];
    launches += 2;
    return MCG_OK;
}

// Whether v[0 .. n) holds an infinity or NaN: an exponent of all ones carries into the sign bit.
static bool any_nonfinite(const double* v, int n) {
    uint64_t carry = 0;
    for (int i = 0; i < n; i++) {
        uint64_t b;
        memcpy(&b, v + i, sizeof b);
        carry |= (b & 0x7ff0000000000000ull) + 0x0010000000000000ull;
    }
    return carry >> 63;
}

// The coordinates go into the page-locked mirror and are taken from there by one kernel.  One core's
// passes over memory are the bound (about 25 GB/s each), so the blocks are checked, copied and compared
// with the last prune's positions while they are in cache, in loops that vectorise (before: interleaved
// with the charges in a fresh vector, copied from pageable memory, the mirror beside it; 100,002 atoms
// 328 -> 182 us).
int SingleEngine::set_coords(const double* x, const double* y, const double* z) {
    for (int i0 = 0; i0 < n; i0 += 1024) {
        const int m = std::min(n - i0, 1024);
        const double *bx = x + i0, *by = y + i0, *bz = z + i0;
        if (any_nonfinite(bx, m) || any_nonfinite(by, m) || any_nonfinite(bz, m)) {
            int i = i0;
            while (std::isfinite(x[i]) && std::isfinite(y[i]) && std::isfinite(z[i])) i++;
            const int rc = get_coords(host_x, host_y, host_z);   // the device still has what the mirror held
            return rc ? rc : fail(MCG_EINVAL, "non-finite coordinate at atom " + std::to_string(i));
        }
        memcpy(host_x + i0, bx, sizeof(double) * m);
        memcpy(host_y + i0, by, sizeof(double) * m);
        memcpy(host_z + i0, bz, sizeof(double) * m);
        if (prune_dirty) continue;
        // a plain displacement within the limit is a wrapped one within it: only other blocks are looked
        // at.  The squares are not negative, so one above the limit borrows into the sign bit.
        const double *px = prune_x.data() + i0, *py = prune_y.data() + i0, *pz = prune_z.data() + i0;
        uint64_t lim, far = 0;
        memcpy(&lim, &prune_lim2, sizeof lim);
        for (int i = 0; i < m; i++) {
            const double dx = bx[i] - px[i], dy = by[i] - py[i], dz = bz[i] - pz[i], d2 = dx * dx + dy * dy + dz * dz;
            uint64_t u;
            memcpy(&u, &d2, sizeof u);
            far |= lim - u;
        }
        for (int i = 0; far >> 63 && i < m && !prune_dirty; i++) note_moved(i0 + i);
    }
    k_take_coords<<<(n + 255) / 256, 256, 0, stream>>>(n, host_x, d_pq, d_cls_of, d_fx, d_x64, fix64.sh, pbc);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(stream));
    return MCG_OK;
}

int SingleEngine::get_coords(double* x, double* y, double* z) {
    std::vector<double4_32a> pq(n);
    CK(cudaMemcpyAsync(pq.data(), d_pq, sizeof(double4_32a) * n, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    for (int i = 0; i < n; i++) { x[i] = pq[i].x; y[i] = pq[i].y; z[i] = pq[i].z; }
    return MCG_OK;
}

int SingleEngine::delta_e(int m, const int* atoms_in, const double* nx, const double* ny, const double* nz, double* de) {
    pending_m = 0;   // a new proposal replaces the pending one, also when it is rejected
    if (int rc = need_list()) return rc;
    if (m <= 0 || m > MAX_MOVED) return fail(MCG_EINVAL, "moved-set size must be in [1, 1024]");
    // sort the moved set (keeps proposal coordinates paired), reject duplicates
    std::vector<int> ord(m);
    std::iota(ord.begin(), ord.end(), 0);
    std::sort(ord.begin(), ord.end(), [&](int a, int b) { return atoms_in[a] < atoms_in[b]; });
    // staged as [idx: m ints | xyz: 3m doubles | terms: 2 ints each], packed so that one small
    // copy carries the proposal; the device copy stays in place for commit()
    const size_t off_xyz = ((size_t)4 * m + 15) & ~(size_t)15, off_terms = off_xyz + (size_t)24 * m;
    char* st = (char*)h_stage;
    int* idx = (int*)st;
    double* xyz = (double*)(st + off_xyz);
    int* terms = (int*)(st + off_terms);
    for (int k = 0; k < m; k++) {
        int a = atoms_in[ord[k]];
        if (a < 0 || a >= n) return fail(MCG_EINVAL, "moved atom index out of range");
        if (k > 0 && a == idx[k - 1]) return fail(MCG_EINVAL, "duplicate moved atom");
        double px = nx[ord[k]], py = ny[ord[k]], pz = nz[ord[k]];
        if (!std::isfinite(px) || !std::isfinite(py) || !std::isfinite(pz)) return fail(MCG_EINVAL, "non-finite proposal");
        idx[k] = a;
        xyz[3 * k] = px; xyz[3 * k + 1] = py; xyz[3 * k + 2] = pz;
    }
    // bonded terms touching the moved set, each once, kind after kind
    stamp++;
    int nt = 0;
    const size_t tcap = (stage_bytes - 64 - off_terms) / 8;
    for (std::vector<int>& v : term_kind) v.clear();
    for (int k = 0; k < m; k++) {
        int a = idx[k];
        for (int t = term_start[a]; t < term_start[a + 1]; t++) {
            int kind = term_data[2 * t], ti = term_data[2 * t + 1];
            size_t gk = (size_t)ti * 5 + kind;
            if (gk >= term_seen.size()) term_seen.resize(gk + 1, 0);
            if (term_seen[gk] == stamp) continue;
            term_seen[gk] = stamp;
            if ((size_t)nt++ >= tcap) return fail(MCG_ECAPACITY, "too many bonded terms in one move");
            term_kind[kind].push_back(ti);
        }
    }
    MoveDev mv{};
    mv.m = m;
    mv.idx = (const int*)d_stage;
    mv.xyz = (const double*)((char*)d_stage + off_xyz);
    mv.terms = (const int*)((char*)d_stage + off_terms);
    int* tend = terms;
    for (int k = 0; k < DE_KINDS; k++) {
        if (term_kind[k].empty()) continue;
        tend = std::copy(term_kind[k].begin(), term_kind[k].end(), tend);
        mv.kind[mv.nkind] = k;
        mv.kend[mv.nkind++] = (int)(tend - terms);
    }
    MoveInline inl;
    inl.m = 0;
    if (m <= INL_M && nt <= INL_T) {
        inl.m = m;
        memcpy(inl.idx, idx, 4 * (size_t)m);
        memcpy(inl.xyz, xyz, 24 * (size_t)m);
        memcpy(inl.terms, terms, 4 * (size_t)nt);
    } else {
        CK(cudaMemcpyAsync(d_stage, h_stage, off_terms + (size_t)nt * 4, cudaMemcpyHostToDevice, stream));
    }
    AtomsDev A = atoms();
    BondedDev B = bonded();
    // slices per moved atom: about one partner (FP64: one side of one) per thread for a Verlet row (64
    // threads), about four per thread over all atoms in full mode (256 threads), at most two blocks per SM in all
    const bool sw = hs.cut == MCG_CUT_SWITCH;
    const int threads = sw ? 64 : 256;
    const int span = (sw ? cap : n) * (hs.prec == MCG_PREC_FP64 ? 2 : 1);
    int S = (span + (sw ? 64 : 1024) - 1) / (sw ? 64 : 1024);
    S = std::max(1, std::min(S, std::max(1, 304 / m)));
    S = std::min(S, std::max(1, MAX_MOVED / m));   // m*S + 5 partials fit the scratch
#define MCG_DELTA(P_, M_)                                                                                             \
    k_delta_e<P_, M_><<<m * S + mv.nkind, threads, 0, stream>>>(A, n, pbc, cut, mv, d_nbr, d_nup, d_nlo, cap, d_fxs,  \
                                                                d_fxd, d_c14s, d_c14d, B, S, d_part, d_ticket, d_map, inl)
    if (hs.prec == MCG_PREC_FP64) {
        if (inl.m) MCG_DELTA(PREC_F64, INL_M);
        else MCG_DELTA(PREC_F64, MAX_MOVED);
    } else {
        if (inl.m) MCG_DELTA(PREC_MIX, INL_M);
        else MCG_DELTA(PREC_MIX, MAX_MOVED);
    }
#undef MCG_DELTA
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(stream));   // de lands in mapped host memory
    *de = ((volatile double*)h_map)[0];
    pending_m = m;
    pending_inline = inl.m > 0;
    pending_off_xyz = off_xyz;
    pending_idx.assign(idx, idx + m);
    pending_xyz.assign(xyz, xyz + 3 * m);
    launches += 1;
    return MCG_OK;
}

// ---- device-resident Metropolis run (MC_metropolis::run, src/MC_metropolis.cpp:80-165) ---------
// For translation moves of atom sets without bonded terms in a periodic switched system, with no
// per-step output: the whole step runs on the device, a launch covering the steps up to the next
// list update (MC_metropolis.cpp:151).  The random numbers are the reference's: the raw 32-bit words of
// the host's std::mt19937, turned into doubles as libstdc++'s generate_canonical<double, 53> does
// (two words, w0 + w1 2^32 rounded once, times 2^-64; a result of 1 becomes the largest double
// below 1) and into uniform_real_distribution values as (b - a) u + a, every operation rounded on
// its own as the reference's uncontracted host code rounds it.
constexpr int RP_MAXT = SingleEngine::kReplayMaxTypes;   // move types
constexpr int RP_MAXM = SingleEngine::kReplayMaxAtoms;   // atoms of one move

bool SingleEngine::replay_fits(const std::vector<MoveKind>& moves) {
    if (moves.empty() || (int)moves.size() > RP_MAXT) return false;
    for (const MoveKind& mk : moves)
        for (int k = 0; k < mk.ninst(); k++) {
            int m = 0;
            for (int r = mk.rstart[k]; r < mk.rstart[k + 1]; r++) m += mk.ranges[2 * r + 1] - mk.ranges[2 * r] + 1;
            if (m > RP_MAXM) return false;
        }
    return true;
}
struct ReplayTables {
    int nmvtyp;
    int ninst[RP_MAXT];           // instances of each move type
    int ibase[RP_MAXT];           // first global instance of each type
    int each[RP_MAXT];            // dmax adjustment period (0: never), MC::adjust_dmax (MC.cpp:165-173)
    double target[RP_MAXT];       // target acceptance, percent
    const int* inst_first;        // per global instance: its first (first, last) atom range; one past the end last
    const int* ranges;            // (first, last) atom pairs
    int ninst_all, nranges;       // sizes of the two (instances + 1 entries, nranges pairs)
};
struct ReplayState {
    double etot;
    long long acc;
    long long cursor;             // random words consumed from the launch's buffer
    int steps_done;               // the last step completed
    int status;                   // 0 ok; 1 out of random words (resume after steps_done); 2 move too large
    double dmax[RP_MAXT];
    int acc_tmp[RP_MAXT];
};

__device__ __forceinline__ double rp_canonical(const uint32_t* __restrict__ w, long long& cur) {
    const double sum = __dadd_rn((double)w[cur], __dmul_rn((double)w[cur + 1], 4294967296.0));
    cur += 2;
    const double r = __dmul_rn(sum, 5.421010862427522170037264e-20);   // 2^-64
    return r >= 1.0 ? 0.99999999999999988898 : r;                       // nextafter(1, 0)
}

// Energy of one pair (iu), the FP64 terms of ref64_pair with the factors of the total folded in: qa, ea are
// the moved atom's charge and eps times K and 4, sw the switch's 1 / (rc^2 - ron^2)^3, 3 ron^2 - rc^2 and
// bounds.  Comparisons of non-negative doubles are comparisons of their bits, on the integer pipe.
__device__ __forceinline__ double rp_pair(double4_32a a, double4_32a b, double2 ea, double2 eb, double qa, const PbcDev& pbc,
                                          const CutDev& cut, double k3s, double sw2s) {
    const double dx = ref64_mic(__dsub_rn(b.x, a.x), pbc.L[0], pbc.rL[0]), dy = ref64_mic(__dsub_rn(b.y, a.y), pbc.L[1], pbc.rL[1]),
                 dz = ref64_mic(__dsub_rn(b.z, a.z), pbc.L[2], pbc.rL[2]);
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const long long u = __double_as_longlong(r2);
    if (u > __double_as_longlong(cut.c2)) return 0.0;
    const double rt = rsqrt64(r2);
    const double x = (ea.y + eb.y) * rt, x2 = x * x, x6 = x2 * x2 * x2;
    double e = fma(ea.x * eb.x, fma(x6, x6, -x6), qa * b.w * rt);
    if (u > __double_as_longlong(cut.n2)) {
        const double s1 = cut.c2 - r2;
        e *= s1 * s1 * fma(sw2s, r2, k3s);
    }
    return e;
}

// One thread-block cluster of RP_CL CTAs of RP_NT threads runs the steps.  On GB300 a warp's FP64
// instruction holds its scheduler's narrow FP64 pipe for tens of cycles whatever its active lanes,
// so a step costs about (warps per scheduler) x (the dependent FP64 operations of one thread):
//  - the proposal's uniforms (move type, instance and RP_TRIES unit-ball tries at once) are formed
//    by the lanes of warp 0 in one pass, and the first accepted try is picked by ballot;
//  - the dE terms are spread one per thread over the cluster's schedulers (CTAs first, then warps,
//    then lanes), the old and the new energy of a pair on different threads;
//  - each warp's sum goes to every CTA's shared memory at once, and behind the step's one cluster
//    barrier every CTA adds the cluster's 32 sums by the same shuffles and takes the same decision;
//  - every CTA commits the move itself (the same values to the same places), so its next reads need no
//    barrier across the cluster.  A CTA can be at most at the next step's barrier while another still
//    commits, and reads positions only before that barrier; the exchanged sums alternate between two
//    buffers for the same reason.  The fixed-point mirrors, which only list builds read, follow before
//    those (k_fix_all);
//  - the decision compares in FP32 unless the draw is within 1e-4 of the threshold (an FP64 exp is some
//    twenty dependent FP64 operations).
// The launch's random words, and the move-instance tables when they fit, are copied into each
// CTA's shared memory first: the proposal's loads are then shared-memory loads, not L2 round trips.
// While the four warps of a CTA take the dE terms, a fifth forms the next step's uniforms: the next
// step's words start at this step's post-proposal cursor, or 2 words later when this step draws an
// acceptance uniform, so 27 uniforms from that cursor cover both cases; the warp forms both cases'
// move type, instance and RP_TRIES unit-ball tries.  The next proposal picks the case its cursor
// matches and only scales, orders and wraps; when none of those tries lies in the ball it goes on
// with the following ones as before.  The same operations on the same words: the same proposals.
// Measured on the 864-atom argon box (moves per second, host work included): 49.8k with one
// 256-thread CTA (its ~200 dE terms at two warps per scheduler), 89.9k with the cluster and the
// words read from global memory, 94.8k with them in shared memory, 99.9k with the fifth warp.
// In runs of 500 steps, 92k so far, 107k with the FP64 operations of ref64_mic and rsqrt64, 142k with one
// barrier and one sum a step, 152k with the terms off the fifth warp's scheduler and its draw used, 163k with
// shorter list builds, 169k with the words and the state in page-locked memory (three copies a launch before).
constexpr int RP_CL = 8;
constexpr int RP_NT = 128;
constexpr int RP_TRIES = 8;
constexpr int RP_SPEC = 32;            // a fifth warp: the next step's uniforms, formed during this step's dE
constexpr int RP_WORDS = 8192;        // random words of one launch, staged in each CTA's shared memory
constexpr int RP_TAB = 3072;          // ints of the instance tables staged with them when they fit
static_assert(RP_CL * RP_NT / 32 == 32, "the decision adds the cluster's warp sums as one warp");

__device__ __forceinline__ double rp_canonical_at(const uint32_t* __restrict__ w, long long at) {
    long long cur = at;
    return rp_canonical(w, cur);
}

__global__ void __cluster_dims__(RP_CL, 1, 1) __launch_bounds__(RP_NT + RP_SPEC)
    k_replay(AtomsDev A, double4_32a* pq, PbcDev pbc, CutDev cut, const int* __restrict__ nbr,
             const int* __restrict__ nup, const int* __restrict__ nlo, int cap, const int* __restrict__ c14s,
             const int* __restrict__ c14d, ReplayTables T, const uint32_t* __restrict__ words, long long nwords,
             const __grid_constant__ ReplayState init, ReplayState* st, int s0, int s1, double beta) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ ReplayState S;
    __shared__ int s_idx[RP_MAXM];
    __shared__ double s_xyz[3 * RP_MAXM];
    __shared__ double s_r[3];
    __shared__ int s_m, s_type, s_stop, s_acc;
    __shared__ long long s_cur;
    __shared__ double s_cl[2][RP_CL * RP_NT / 32];   // every warp's sum, of this step and the other
    __shared__ __align__(16) uint32_t s_words[RP_WORDS];
    __shared__ int s_tab[RP_TAB];
    // the next step's uniforms, both cases (0: no acceptance draw in this step, 1: one)
    __shared__ double s_sx[2 * RP_TRIES], s_sy[2 * RP_TRIES], s_sz[2 * RP_TRIES], s_sq[2 * RP_TRIES];
    __shared__ int s_st[2], s_sg[2], s_sok;
    __shared__ double s_alpha;      // this step's acceptance uniform, when the fifth warp could form it
    __shared__ long long s_sbase;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = RP_NT / 32, G = RP_CL * RP_NT;
    for (int i = tid; i < (int)(nwords >> 2); i += blockDim.x)
        reinterpret_cast<uint4*>(s_words)[i] = reinterpret_cast<const uint4*>(words)[i];
    const bool tab_sh = T.ninst_all + 2 * T.nranges <= RP_TAB;
    if (tab_sh) {
        for (int i = tid; i < T.ninst_all; i += blockDim.x) s_tab[i] = T.inst_first[i];
        for (int i = tid; i < 2 * T.nranges; i += blockDim.x) s_tab[T.ninst_all + i] = T.ranges[i];
    }
    if (tid == 0) s_sok = 0;
    const double k3s = (cut.c2 - 3.0 * cut.n2) * cut.sw2, sw2s = 2.0 * cut.sw2;
    const int* inst_first = tab_sh ? s_tab : T.inst_first;
    const int* ranges = tab_sh ? s_tab + T.ninst_all : T.ranges;
    const int rank = (int)cluster.block_rank();
    // this thread's place in the order the terms are dealt: CTAs first, then the lanes of warps 1 and 2, then
    // those of 3 and 0.  Up to 512 terms (255 partners of one atom) leave warp 0's scheduler to the fifth warp
    const int gslot = rank + RP_CL * (2 * lane + (warp == 1 || warp == 2 ? warp - 1 : 64 + (warp == 0)));
    if (tid == 0) S = init;
    cluster.sync();   // every CTA of the cluster is running before any writes into its shared memory
    for (int step = s0 + 1; step <= s1; step++) {
        if (warp == 0) {
            // the proposal (MC.cpp:142-156): type and instance from the words at cur and cur + 2,
            // unit-ball tries of 3 uniforms each from cur + 4 on (6 words a try), RP_TRIES at a time
            const long long cur = S.cursor;
            bool out = cur + 256 > nwords;
            int t = 0, m = 0, first = -1;
            int sv = -1;   // the case of the uniforms formed during the previous step that matches cur
            if (!out && s_sok) sv = cur == s_sbase ? 0 : (cur == s_sbase + 2 ? 1 : -1);
            if (!out) {
                int g;
                if (sv >= 0) {
                    t = s_st[sv];
                    g = s_sg[sv];
                } else {
                    double u = 0.0;
                    if (lane < 2) u = rp_canonical_at(s_words, cur + 2 * lane);
                    const double u0 = __shfl_sync(0xffffffffu, u, 0), u1 = __shfl_sync(0xffffffffu, u, 1);
                    t = (int)__dmul_rn((double)T.nmvtyp, u0);
                    g = T.ibase[t] + (int)__dmul_rn((double)T.ninst[t], u1);
                }
                if (lane == 0) {
                    for (int r = inst_first[g]; r < inst_first[g + 1]; r++)
                        for (int a = ranges[2 * r]; a <= ranges[2 * r + 1]; a++) {
                            if (m < RP_MAXM) s_idx[m] = a;
                            m++;
                        }
                }
                m = __shfl_sync(0xffffffffu, m, 0);
                int pass0 = 0;
                if (sv >= 0) {   // the first RP_TRIES tries, formed in advance
                    const unsigned ok = __ballot_sync(0xffffffffu, lane < RP_TRIES && s_sq[sv * RP_TRIES + lane] <= 1.0);
                    if (ok) {
                        const int k = __ffs(ok) - 1;
                        first = k;
                        if (lane < 3) {   // a component per lane: one product's latency
                            const int e = sv * RP_TRIES + k;
                            s_r[lane] = __dmul_rn(lane == 0 ? s_sx[e] : lane == 1 ? s_sy[e] : s_sz[e], S.dmax[t]);
                        }
                    }
                    pass0 = 1;
                }
                for (int pass = pass0; first < 0; pass++) {
                    const long long cb = cur + 4 + 6LL * RP_TRIES * pass;
                    if (cb + 6LL * RP_TRIES + 2 > nwords) { out = true; break; }   // the pass and the acceptance draw
                    double v = 0.0;
                    if (lane < 3 * RP_TRIES) v = __dadd_rn(__dmul_rn(rp_canonical_at(s_words, cb + 2 * lane), 2.0), -1.0);
                    const double x = __shfl_sync(0xffffffffu, v, (3 * lane) & 31);
                    const double y = __shfl_sync(0xffffffffu, v, (3 * lane + 1) & 31);
                    const double z = __shfl_sync(0xffffffffu, v, (3 * lane + 2) & 31);
                    const double q = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
                    const unsigned ok = __ballot_sync(0xffffffffu, lane < RP_TRIES && q <= 1.0);
                    if (ok) {
                        const int k = __ffs(ok) - 1;
                        first = pass * RP_TRIES + k;
                        if (lane == k) {
                            const double dm = S.dmax[t];
                            s_r[0] = __dmul_rn(x, dm); s_r[1] = __dmul_rn(y, dm); s_r[2] = __dmul_rn(z, dm);
                        }
                    }
                }
            }
            if (lane == 0) {
                s_stop = 0;
                if (out) { s_stop = 1; S.status = 1; }
                else if (m > RP_MAXM) { s_stop = 1; S.status = 2; }
                else {
                    for (int i = 1; i < m; i++) {        // ascending atom order (the partner lookup bisects)
                        const int v = s_idx[i];
                        int k = i - 1;
                        while (k >= 0 && s_idx[k] > v) { s_idx[k + 1] = s_idx[k]; k--; }
                        s_idx[k + 1] = v;
                    }
                    s_m = m;
                    s_type = t;
                    s_cur = cur + 4 + 6LL * (first + 1);
                }
            }
            __syncwarp();
            if (!out && m <= RP_MAXM)
                for (int i = lane; i < 3 * m; i += 32) {   // the moved atoms' new positions, wrapped
                    const int k = i / 3, c = i - 3 * k;
                    const double4_32a p = pq[s_idx[k]];
                    const double pc = c == 0 ? p.x : (c == 1 ? p.y : p.z);
                    s_xyz[i] = ref64_mic(__dadd_rn(pc, s_r[c]), pbc.L[c], pbc.rL[c]);   // PerConditions::applyPBC
                }
        }
        __syncthreads();
        if (s_stop) break;   // the same in every CTA: each formed the same proposal from the same words
        if (warp == NW) {
            // the next step's uniforms (words from b = this step's post-proposal cursor): type and
            // instance of case v from uniforms v and v + 1, try k from v + 2 + 3k .. v + 4 + 3k
            const long long b = s_cur;
            const bool ok = b + 54 <= nwords;
            double c = 0.0;
            if (ok && lane < 27) c = rp_canonical_at(s_words, b + 2 * lane);
            const double cn = __shfl_sync(0xffffffffu, c, (lane + 1) & 31);
            if (lane < 2) {
                const int tv = (int)__dmul_rn((double)T.nmvtyp, c);
                s_st[lane] = tv;
                s_sg[lane] = T.ibase[tv] + (int)__dmul_rn((double)T.ninst[tv], cn);
            }
            const int i0 = (lane >> 3) + 2 + 3 * (lane & 7);
            const double cx = __shfl_sync(0xffffffffu, c, i0 & 31), cy = __shfl_sync(0xffffffffu, c, (i0 + 1) & 31),
                         cz = __shfl_sync(0xffffffffu, c, (i0 + 2) & 31);
            if (lane < 2 * RP_TRIES) {
                const double x = __dadd_rn(__dmul_rn(cx, 2.0), -1.0), y = __dadd_rn(__dmul_rn(cy, 2.0), -1.0),
                             z = __dadd_rn(__dmul_rn(cz, 2.0), -1.0);
                s_sx[lane] = x; s_sy[lane] = y; s_sz[lane] = z;
                s_sq[lane] = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
            }
            if (lane == 0) { s_sbase = b; s_sok = ok ? 1 : 0; s_alpha = c; }   // uniform 0 is the draw, if there is one
        }
        // dE of the moved set over its Verlet partners and 1-4 pairs, FP64 (as k_delta_e): term
        // (k, t, side) of the moved atoms' partner lists, numbered in list order, goes to the thread
        // whose gslot it equals modulo G; side 0 is the old pair energy (subtracted), 1 the new
        const int m = s_m;
        auto slot = [&](int j) -> int {
            int lo = 0, hi = m - 1;
            while (lo <= hi) {
                const int mid = (lo + hi) >> 1, v = s_idx[mid];
                if (v == j) return mid;
                if (v < j) lo = mid + 1; else hi = mid - 1;
            }
            return -1;
        };
        double val = 0.0;
        int base = 0;
        for (int k = 0; k < m && warp < NW; k++) {
            const int a = s_idx[k];
            const int* row = nbr + (size_t)a * cap;
            const int u = nup[a], l = nlo[a], n14 = c14s[a + 1] - c14s[a];
            const int cnt = u + l + n14;
            int q = (gslot - 2 * base) % G;
            if (q < 0) q += G;
            if (q < 2 * cnt) {
                const double4_32a po = pq[a], pn = make_double4_32a(s_xyz[3 * k], s_xyz[3 * k + 1], s_xyz[3 * k + 2], po.w);
                const double qa = CHGCHARMM * KCALTOIU * po.w;
                for (; q < 2 * cnt; q += G) {
                    const int t = q >> 1, side = q & 1;
                    const bool fourteen = t >= u + l;
                    const int j = fourteen ? c14d[c14s[a] + t - u - l] : (t < u ? row[t] : row[cap - 1 - (t - u)]);
                    const int sj = slot(j);
                    if (sj >= 0 && j < a) continue;   // a pair of moved atoms, counted at its lower atom
                    double4_32a jj = pq[j];
                    if (side && sj >= 0) { jj.x = s_xyz[3 * sj]; jj.y = s_xyz[3 * sj + 1]; jj.z = s_xyz[3 * sj + 2]; }
                    double2 ea = fourteen ? A.es14[a] : A.es[a];
                    const double2 eb = fourteen ? A.es14[j] : A.es[j];
                    ea.x *= 4.0;
                    const double e = rp_pair(side ? pn : po, jj, ea, eb, qa, pbc, cut, k3s, sw2s);
                    val += side ? e : -e;
                }
            }
            base += cnt;
        }
        double* cl = s_cl[step & 1];
        if (warp < NW) {
            if (__any_sync(0xffffffffu, __double_as_longlong(val) != 0)) val = warp_sum(val);
            if (lane < RP_CL) *cluster.map_shared_rank(cl + rank * NW + warp, lane) = val;
        }
        cluster.sync();
        if (warp == 0) {
            const double de = warp_sum(cl[lane]);
            if (lane == 0) {
                // MC_metropolis::apply_criterion (MC_metropolis.cpp:175-204); exp is CUDA's (at most 1 ulp
                // from the exact value) where the host loop calls glibc's: the two runs can part only on a
                // uniform within an ulp of the threshold
                long long cur = s_cur;
                bool accepted;
                if (de <= 2.220446049250313e-16) accepted = true;
                else {
                    const double alpha = s_sok ? s_alpha : rp_canonical_at(s_words, cur);
                    cur += 2;
                    const float af = (float)alpha, ef = __expf((float)(-beta * de));   // off by less than 1e-5
                    accepted = fabsf(af - ef) > 1e-4f ? af < ef : alpha < exp(-beta * de);
                }
                S.cursor = cur;
                const int t = s_type;
                if (accepted) {
                    S.acc_tmp[t]++;
                    S.etot += de;
                    S.acc++;
                }
                for (int tt = 0; tt < T.nmvtyp; tt++) {
                    if (T.each[tt] != 0 && (step % T.each[tt]) == 0) {
                        const double ratio = (double)S.acc_tmp[tt] / (double)T.each[tt];
                        S.dmax[tt] = ratio > T.target[tt] / 100 ? S.dmax[tt] * 1.10 : S.dmax[tt] * 0.9;
                        S.acc_tmp[tt] = 0;
                    }
                }
                S.steps_done = step;
                s_acc = accepted ? 1 : 0;
            }
        }
        __syncthreads();
        if (s_acc) {
            for (int i = tid; i < 3 * m; i += blockDim.x) reinterpret_cast<double*>(pq + s_idx[i / 3])[i % 3] = s_xyz[i];
            __syncthreads();   // the commit before the next step's proposal
        }
    }
    cluster.sync();   // no CTA leaves while another may still write into its shared memory
    if (tid == 0 && rank == 0) *st = S;
}

bool SingleEngine::replay_cluster_ok() {
    static int ok = -1;
    if (ok < 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(RP_CL);
        cfg.blockDim = dim3(RP_NT + RP_SPEC);
        int nclusters = 0;
        ok = cudaOccupancyMaxActiveClusters(&nclusters, k_replay, &cfg) == cudaSuccess && nclusters >= 1 ? 1 : 0;
        if (!ok) cudaGetLastError();
    }
    return ok == 1;
}

int SingleEngine::metropolis_device(std::mt19937& gen, const std::vector<MoveKind>& moves, double beta, int nsteps,
                                    double* etot, int64_t* n_accepted) {
    const int nt = (int)moves.size();
    if (nt < 1 || nt > RP_MAXT) return fail(MCG_ENOTSUP, "device run: 1 to 8 move types");
    if (int rc = need_list()) return rc;
    ReplayTables T{};
    ReplayState S{};
    std::vector<int> first, ranges;
    T.nmvtyp = nt;
    for (int t = 0; t < nt; t++) {
        const MoveKind& mk = moves[t];
        T.ninst[t] = mk.ninst();
        T.ibase[t] = (int)first.size();
        T.each[t] = mk.each;
        T.target[t] = mk.target;
        S.dmax[t] = mk.dmax;
        const int rb = (int)ranges.size() / 2;
        for (int k = 0; k < mk.ninst(); k++) first.push_back(rb + mk.rstart[k]);
        ranges.insert(ranges.end(), mk.ranges.begin(), mk.ranges.end());
    }
    first.push_back((int)ranges.size() / 2);
    S.etot = *etot;
    constexpr long long W = RP_WORDS;        // random words per launch
    // In the page-locked staging memory: a launch's words and the state it leaves, which the kernel reads
    // and writes there (few and once a launch), and the instance tables on their way to the device; tables
    // larger than it get their own memory.
    uint32_t* const w = (uint32_t*)h_stage;
    ReplayState* const left = (ReplayState*)(w + W);
    static_assert(sizeof(ReplayState) <= 256, "place of the tables");
    const size_t tab_at = sizeof(uint32_t) * W + 256, nfirst = first.size();
    first.insert(first.end(), ranges.begin(), ranges.end());
    const size_t tab_bytes = sizeof(int) * first.size();
    pending_m = 0;                           // the staged proposal makes way
    int* d_tab = nullptr;
    int rc = MCG_OK;
    auto done = [&](int r) {
        // the run keeps pq current; the mirrors, which it does not read, follow here
        k_fix_all<<<(n + 255) / 256, 256, 0, stream>>>(n, d_pq, d_cls_of, d_fx, d_x64, fix64.sh, pbc);
        launches++;
        if (cudaStreamSynchronize(stream) != cudaSuccess && r == MCG_OK) r = fail(MCG_ECUDA, "device run: mirrors");
        if (d_tab) cudaFree(d_tab);
        return r;
    };
    const bool staged = tab_at + tab_bytes <= stage_bytes;
    if (!staged && (rc = dalloc(&d_tab, first.size()))) return done(rc);
    int* const tab = staged ? (int*)d_stage : d_tab;
    if (staged) memcpy((char*)h_stage + tab_at, first.data(), tab_bytes);
    if (cudaMemcpyAsync(tab, staged ? (const void*)((char*)h_stage + tab_at) : first.data(), tab_bytes, cudaMemcpyHostToDevice, stream) !=
        cudaSuccess)
        return done(fail(MCG_ECUDA, "device run: table upload"));
    T.inst_first = tab;
    T.ranges = tab + nfirst;
    T.ninst_all = (int)nfirst;
    T.nranges = (int)ranges.size() / 2;
    std::vector<uint32_t> stash;     // the generator's next words, drawn while the previous launch ran
    size_t stash_at = 0;
    long long filled = 0;
    int step = 0;
    while (step < nsteps) {
        // the words not consumed yet, then the generator's next ones (from the stash first)
        const long long keep = filled - S.cursor;
        if (keep > 0 && S.cursor > 0) std::memmove(w, w + S.cursor, sizeof(uint32_t) * (size_t)keep);
        filled = std::max(0LL, keep);
        const int s1 = std::min(nsteps, (step / 50 + 1) * 50);     // up to the next list update
        // a step takes 17 words on average; a launch that ran out of them goes on with a full buffer
        const long long need = S.status == 1 ? W : std::min(W, 32LL * (s1 - step) + 512);
        while (filled < need) w[filled++] = stash_at < stash.size() ? stash[stash_at++] : gen();
        S.cursor = 0;
        S.status = 0;
        k_replay<<<RP_CL, RP_NT + RP_SPEC, 0, stream>>>(atoms(), d_pq, pbc, cut, d_nbr, d_nup, d_nlo, cap, d_c14s, d_c14d, T,
                                              w, filled & ~3LL, S, left, step, s1, beta);
        launches++;
        // while the launch runs: the generator's next words, in order, for the next buffer
        stash.erase(stash.begin(), stash.begin() + (long)stash_at);
        stash_at = 0;
        while ((long long)stash.size() < need) stash.push_back(gen());
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(stream) != cudaSuccess)
            return done(fail(MCG_ECUDA, "device run: replay kernel"));
        memcpy(&S, left, sizeof S);
        if (S.status == 2) return done(fail(MCG_ENOTSUP, "device run: a move of more than 64 atoms"));
        step = S.steps_done;
        if (S.status == 0 && step % 50 == 0) {
            k_fix_all<<<(n + 255) / 256, 256, 0, stream>>>(n, d_pq, d_cls_of, d_fx, d_x64, fix64.sh, pbc);
            launches++;
            if ((rc = update_lists())) return done(rc);
        }
    }
    // host mirror of the coordinates
    std::vector<double4_32a> pqh((size_t)n);
    if (cudaMemcpy(pqh.data(), d_pq, sizeof(double4_32a) * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess)
        return done(fail(MCG_ECUDA, "device run: coordinates"));
    for (int a = 0; a < n; a++) { host_x[a] = pqh[a].x; host_y[a] = pqh[a].y; host_z[a] = pqh[a].z; }
    prune_dirty = true;
    pending_m = 0;
    *etot = S.etot;
    *n_accepted = S.acc;
    return done(MCG_OK);
}

int SingleEngine::commit() {
    if (pending_m <= 0) return fail(MCG_EINVAL, "no pending proposal to commit");
    // the pending proposal is still staged on the device: only delta_e and a device run write d_stage,
    // and each replaces the pending proposal.  Stream order puts the update before any later
    // call's work, so the host does not wait for it.
    const int* didx = (const int*)d_stage;
    const double* dxyz = (const double*)((char*)d_stage + pending_off_xyz);
    MoveInline inl;
    inl.m = 0;
    if (pending_inline) {
        inl.m = pending_m;
        memcpy(inl.idx, pending_idx.data(), 4 * (size_t)pending_m);
        memcpy(inl.xyz, pending_xyz.data(), 24 * (size_t)pending_m);
    }
    k_commit<<<(3 * pending_m + 127) / 128, 128, 0, stream>>>(pending_m, didx, dxyz, d_pq, d_fx, d_x64, fix64.sh, pbc, inl);
    CK(cudaGetLastError());
    for (int k = 0; k < pending_m; k++) {
        int a = pending_idx[k];
        host_x[a] = pending_xyz[3 * k]; host_y[a] = pending_xyz[3 * k + 1]; host_z[a] = pending_xyz[3 * k + 2];
        if (!prune_dirty) note_moved(a);
    }
    pending_m = 0;
    launches += 1;
    return MCG_OK;
}

bool SingleEngine::pending_matches(int m, const int* atoms, const double* x, const double* y, const double* z) const {
    if (pending_m != m) return false;
    for (int k = 0; k < m; k++) {
        const int a = atoms[k];
        if (pending_idx[k] != a || pending_xyz[3 * k] != x[a] || pending_xyz[3 * k + 1] != y[a] ||
            pending_xyz[3 * k + 2] != z[a])
            return false;
    }
    return true;
}

int SingleEngine::update_lists() {
    if (hs.cut != MCG_CUT_SWITCH) return MCG_OK;
    int rc = build_list();
    launches += 5;
    return rc;
}

int SingleEngine::get_pairlist(int* counts, int* entries, int64_t cap_entries, int64_t* total) {
    if (hs.cut != MCG_CUT_SWITCH) {
        for (int i = 0; i < n; i++) counts[i] = 0;
        if (total) *total = 0;
        return MCG_OK;
    }
    if (int rc = need_list()) return rc;
    std::vector<int> up(n);
    CK(cudaMemcpyAsync(up.data(), d_nup, sizeof(int) * n, cudaMemcpyDeviceToHost, stream));
    std::vector<int> rows((size_t)n * cap);
    CK(cudaMemcpyAsync(rows.data(), d_nbr, sizeof(int) * (size_t)n * cap, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    int64_t t = 0;
    for (int i = 0; i < n; i++) { counts[i] = up[i]; t += up[i]; }
    if (total) *total = t;
    if (entries && cap_entries >= t) {
        int64_t p = 0;
        for (int i = 0; i < n; i++) {
            int* r = rows.data() + (size_t)i * cap;
            std::sort(r, r + up[i]);
            memcpy(entries + p, r, sizeof(int) * up[i]);
            p += up[i];
        }
    }
    return MCG_OK;
}

}  // namespace mcg
