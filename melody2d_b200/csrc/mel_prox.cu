// Update_proximity (Code/Proximity.h:48-473) on the device, for one model or for several models
// (the members of a batch) with the same launches.
//
// Stages (all integer bookkeeping deterministic, geometry bit-identical to the reference):
//   boxes_kernel       border boxes inflated by the detection distance and their period shifts
//                      (Code/Proximity.h:63-109), one warp per border; segment-block and superblock
//                      boxes for pruning, one warp per superblock
//   neighbour_kernel or cl_*   (body, border) overlap with periodic shifts and de-duplication
//                      (Code/Proximity.h:112-169), one warp per body
//   tasks_kernel       tasks and slots per body and their offsets: one task per (slave body, slave
//                      border, neighbour, piece of the border) in the reference's loop order, then
//                      self tasks per (slave body, border, piece); a slot per (task, slave border node)
//   [host read-back]   task and slot totals of every member
//   find_kernel        accepted candidates: a thread per slot tests the master's boxes, then a warp per
//                      slot that is near one tests the segments; candidates are listed in any order
//                      and counted per task
//   scan               task offsets in the new list
//   [host read-back]   contact totals of every member
//   bucket_kernel, write_kernel   the candidates by task; one warp per candidate finds its place in
//                      the task (slave border node, then segment order, the reference's) and writes the
//                      contact element, with the history of the first matching old element of the
//                      same slave border node (Code/Proximity.h:269-284)
//   inc_fill_kernel, bodies_kernel   incoming ranges, contact ranges and the vgap carry per body
// Every kernel reads a table of member jobs (mel_prox_job), or its own argument when there is one
// member; the host driver is at the end.
//
// What bounds it: latency.  A run is some fifteen short launches, each a chain of dependent loads.
// Measured on B200, an update with its launch gaps and read-backs: 4x4 lattice 370 -> 95 us, 50
// grains 486 -> 135 us, 700 grains 582 -> 175 us, against forty launches in which a thread per slot
// walked its segments itself, once to count (68 us) and once to write (155 us).
#include <cstdio>
#include <cstring>
#include <utility>
#include <vector>
#include <algorithm>
#include "mel_internal.h"
#include "mel_geometry.cuh"
#include "mel_prox_host.h"
#include "mel_dependent.cuh"

// total: where the sum of all entries goes as well (a pinned host word), or NULL
struct mel_scan_job { const int* in; int* out; int n; int* sums; int* total; };

namespace mel {

// ---------------------------------------------------------------------------------------------
// exclusive scans of int arrays, several per launch (deterministic; one launch up to SCAN_ITEMS
// entries, three above).  Job j scans in[0..n) into out[0..n] (out[n] = total); blocks [bpre[j],
// bpre[j+1]) of a launch serve job j.  A few jobs travel as the kernel's argument.
// ---------------------------------------------------------------------------------------------
#define SCAN_BLOCK 1024
#define SCAN_PER 8
#define SCAN_ITEMS (SCAN_BLOCK * SCAN_PER)
#define SCAN_INLINE 4
struct scan_args { const mel_scan_job* J; const int* bpre; int nj; mel_scan_job job[SCAN_INLINE]; int pre[SCAN_INLINE + 1]; };
__device__ __forceinline__ int block_job(const int* bpre, int nj)
{
    int lo = 0, hi = nj;                  // largest j with bpre[j] <= blockIdx.x
    while (hi - lo > 1) { int mid = (lo + hi) >> 1; if (bpre[mid] <= (int)blockIdx.x) lo = mid; else hi = mid; }
    return lo;
}

// exclusive prefix of v over the block and the block's total; s: one int per warp
__device__ __forceinline__ int block_scan(int v, int* s, int& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) s[warp] = incl;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int w = 0; w < nw; w++) { if (w < warp) before += s[w]; total += s[w]; }
    return before + incl - v;
}

__global__ void __launch_bounds__(SCAN_BLOCK) scan_block_kernel(const __grid_constant__ scan_args A)
{
    __shared__ int s[SCAN_BLOCK / 32];
    grid_wait();
    grid_release();
    const int j = block_job(A.J ? A.bpre : A.pre, A.nj);
    const mel_scan_job job = A.J ? A.J[j] : A.job[j];
    const int lb = blockIdx.x - (A.J ? A.bpre : A.pre)[j];
    const int i0 = lb * SCAN_ITEMS + threadIdx.x * SCAN_PER;
    int v[SCAN_PER], sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) { v[k] = i0 + k < job.n ? job.in[i0 + k] : 0; sum += v[k]; }
    int total, at = block_scan(sum, s, total);
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) { if (i0 + k <= job.n) job.out[i0 + k] = at; at += v[k]; }
    if (threadIdx.x == SCAN_BLOCK - 1) {
        job.sums[lb] = total;
        if (job.total) *job.total = total;
    }
}
// adds the scanned block totals (in) to out[0..n) block by block
__global__ void __launch_bounds__(SCAN_BLOCK) scan_add_kernel(const __grid_constant__ scan_args A)
{
    grid_wait();
    grid_release();
    const int j = block_job(A.J ? A.bpre : A.pre, A.nj);
    const mel_scan_job job = A.J ? A.J[j] : A.job[j];
    const int lb = blockIdx.x - (A.J ? A.bpre : A.pre)[j];
    for (int i = lb * SCAN_ITEMS + threadIdx.x; i < min((lb + 1) * SCAN_ITEMS, job.n); i += SCAN_BLOCK) job.out[i] += job.in[lb];
}

} // namespace mel

namespace mel {

// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void aabb_item(const mel_dev& d, double* aabb, int* shmin, int* shmax, int g, int lane)
{
    if (g >= d.nbd) return;
    int b = d.bd_body[g];
    if (d.b_status[b] == MEL_STATUS_INACTIVE) return;
    double dd = d.b_dist[3 * b + 1];
    int n0 = d.b_node0[b];
    double xmin = 1.e100, xmax = -1.e100, ymin = 1.e100, ymax = -1.e100;
    bool nonfinite = false;          // the comparisons below pass over NaN, so it is tested apart
    const int e1 = d.bd_e0[g + 1];
    for (int e = d.bd_e0[g] + lane; e < e1; e += 8 * 32) {      // eight entries in flight a lane
        int nd[8];
        double2 p[8];
#pragma unroll
        for (int k = 0; k < 8; k++) nd[k] = e + 32 * k < e1 ? d.e_node[e + 32 * k] : -1;
#pragma unroll
        for (int k = 0; k < 8; k++) p[k] = nd[k] >= 0 ? d.x[n0 + nd[k]] : make_double2(0., 0.);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (nd[k] < 0) continue;
            nonfinite |= !isfinite(p[k].x) || !isfinite(p[k].y);
            if (p[k].x - dd < xmin) xmin = p[k].x - dd;
            if (p[k].x + dd > xmax) xmax = p[k].x + dd;
            if (p[k].y - dd < ymin) ymin = p[k].y - dd;
            if (p[k].y + dd > ymax) ymax = p[k].y + dd;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        xmin = fmin(xmin, __shfl_xor_sync(0xffffffffu, xmin, o));
        xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
        ymin = fmin(ymin, __shfl_xor_sync(0xffffffffu, ymin, o));
        ymax = fmax(ymax, __shfl_xor_sync(0xffffffffu, ymax, o));
    }
    nonfinite = __any_sync(0xffffffffu, nonfinite);
    if (lane == 0) {
        double invperiod = 1. / d.period;
        double f0 = floor((xmin - d.xmin) * invperiod), f1 = floor((xmax - d.xmin) * invperiod);
        // a box that is not finite, or that spans more periods than any body can, comes from a
        // diverged state; it is reported and left out of the neighbour search, whose shift loop
        // it would otherwise drive through billions of iterations
        bool finite = !nonfinite && isfinite(xmin) && isfinite(xmax) && isfinite(ymin) && isfinite(ymax);
        bool sane = finite && fabs(f0) < 1.e6 && fabs(f1) < 1.e6 && f1 - f0 <= MEL_MAX_SHIFT_SPAN;
        if (!sane) {
            atomicOr(&d.err[MEL_E_NAN], finite ? 2u : 1u);
            xmin = 1.e300; xmax = -1.e300; ymin = 1.e300; ymax = -1.e300; f0 = 0.; f1 = -1.;
        }
        aabb[4 * g] = xmin; aabb[4 * g + 1] = xmax; aabb[4 * g + 2] = ymin; aabb[4 * g + 3] = ymax;
        shmin[g] = (int)f0;
        shmax[g] = (int)f1;
    }
}

// the neighbour entries of border g1 (of body b1) against every active body, appended to out at
// `count` in the reference's order (body, border, shift ascending; Code/Proximity.h:112-169): an
// entry already listed for an earlier border of b1 (out[0..count_before)) is not repeated
__device__ __forceinline__ void nbr_scan_all(const mel_dev& d, const double* aabb, const int* shmin, const int* shmax,
                                             int* out, int cap, int b1, int g1, int count_before, int& count, int lane)
{
    const double xmin1 = aabb[4 * g1], xmax1 = aabb[4 * g1 + 1], ymin1 = aabb[4 * g1 + 2], ymax1 = aabb[4 * g1 + 3];
    const int smin1 = shmin[g1], smax1 = shmax[g1];
    const int first_border = (g1 == d.b_bd0[b1]);
    for (int base = 0; base < d.nb; base += 32) {
        int b2 = base + lane;
        bool ok = b2 < d.nb && b2 != b1 && d.b_status[b2] != MEL_STATUS_INACTIVE;
        int mine = 0;
        for (int pass = 0; pass < 2; pass++) {
            int k = 0;
            if (ok) {
                for (int g2 = d.b_bd0[b2]; g2 < d.b_bd0[b2 + 1]; g2++) {
                    double xmin2 = aabb[4 * g2], xmax2 = aabb[4 * g2 + 1], ymin2 = aabb[4 * g2 + 2], ymax2 = aabb[4 * g2 + 3];
                    if ((ymax2 < ymin1) || (ymax1 < ymin2)) continue;
                    int r2 = g2 - d.b_bd0[b2];
                    for (int s = smin1 - shmax[g2]; s <= smax1 - shmin[g2]; s++) {
                        if ((xmax2 + s * d.period > xmin1) && (xmin2 + s * d.period < xmax1)) {
                            bool dup = false;
                            if (!first_border) {
                                for (int q = 0; q < count_before && q < cap; q++)
                                    if (out[3 * q] == b2 && out[3 * q + 1] == r2 && out[3 * q + 2] == s) { dup = true; break; }
                            }
                            if (dup) continue;
                            if (pass == 1) {
                                int pos = mine + k;
                                if (pos < cap) { out[3 * pos] = b2; out[3 * pos + 1] = r2; out[3 * pos + 2] = s; }
                            }
                            k++;
                        }
                    }
                }
            }
            if (pass == 0) {
                // exclusive prefix of k across lanes
                int incl = k;
                for (int o = 1; o < 32; o <<= 1) {
                    int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                int total = __shfl_sync(0xffffffffu, incl, 31);
                mine = count + incl - k;
                count += total;
            }
        }
        __syncwarp();
    }
}

// neighbour lists by all pairs of bodies, one warp per body
__device__ __forceinline__ void neighbour_item(const mel_dev& d, const double* aabb, const int* shmin, const int* shmax,
                                               int* nbr, int* nbn, int cap, int b1, int lane)
{
    if (b1 >= d.nb) return;
    if (d.b_status[b1] == MEL_STATUS_INACTIVE) { if (lane == 0) nbn[b1] = 0; return; }
    int* out = nbr + (size_t)3 * cap * b1;
    int count = 0;
    for (int g1 = d.b_bd0[b1]; g1 < d.b_bd0[b1 + 1]; g1++) {
        const int count_before = count;   // entries of earlier border1 iterations (dedup scope)
        nbr_scan_all(d, aabb, shmin, shmax, out, cap, b1, g1, count_before, count, lane);
    }
    if (lane == 0) {
        nbn[b1] = count;
        if (count > cap) { atomicOr(&d.err[MEL_E_NBR_OVERFLOW], 1u); atomicMax(&d.err[MEL_E_NBR_NEED], (unsigned)count); }
    }
}

// ---------------------------------------------------------------------------------------------
// cell-list broad phase: the same neighbour lists from a hashed uniform grid.  Each border box is
// binned by its lower corner (x wrapped over the period, so that shifted copies share columns)
// into cells of side cl_h (the largest initial box, widened; columns cl_hx = period / cl_ncx), the
// borders are counting-sorted by bucket, and each border of a body gathers the borders whose
// lower corner lies in a cell that a box of the run's largest width and height overlapping it
// can occupy.  The gathered borders (hash collisions and repeated columns included) are sorted,
// made unique and emitted with the exact overlap and shift tests of the all-pairs pass, so the
// lists are entry for entry those of nbr_scan_all; a border whose cell range or candidate count
// is too large takes the all-pairs pass instead.  A big box is itself a query like any other: the
// borders it can meet have their corners in the cells its extent (widened by the binned boxes'
// largest width and height) covers, or are big themselves.
// ---------------------------------------------------------------------------------------------
#define PROX_THREADS_CL 256  // threads of the job kernels (PROX_THREADS below)
#define CL_CAND 256          // gathered candidates per border (beyond: all-pairs for that border)
#define CL_MAX_CELLS 4096    // cells one border's query visits (beyond: all-pairs)

__device__ __forceinline__ int cl_bucket(const mel_prox_job& j, double x, double y)
{
    // (a coordinate beyond the integer range saturates: such a box is only ever found by the
    // all-pairs pass of the borders that query it)
    long long cx = (long long)floor((x - j.d.xmin) / j.cl_hx);
    long long cw = cx % j.cl_ncx;
    if (cw < 0) cw += j.cl_ncx;
    const long long cy = (long long)floor(y / j.cl_h);
    const unsigned k = (unsigned)cw * 73856093u ^ (unsigned)cy * 19349663u;
    return (int)(k & (unsigned)(j.cl_T - 1));
}

__device__ __forceinline__ bool cl_box_ok(const mel_dev& d, const double* a, int g)
{
    return d.b_status[d.bd_body[g]] != MEL_STATUS_INACTIVE && a[4 * g] <= a[4 * g + 1] && a[4 * g + 2] <= a[4 * g + 3];
}

// a box wider or higher than a cell (a long wall, a plate) is kept out of the grid: every query
// tests it, and its own border takes the all-pairs pass
__device__ __forceinline__ bool cl_big(const mel_prox_job& j, const double* a)
{
    return a[1] - a[0] > j.cl_h || a[3] - a[2] > j.cl_h;
}

// bucket counts and the largest width and height of the binned boxes (non-negative doubles order
// as their bits); big boxes are listed at the end of cl_idx, counted in cl_cur[cl_T]
__device__ __forceinline__ void cl_count_item(const mel_prox_job& j, int g)
{
    const mel_dev& d = j.d;
    if (g >= d.nbd || !cl_box_ok(d, j.aabb, g)) return;
    const double* a = j.aabb + 4 * g;
    if (cl_big(j, a)) { j.cl_idx[d.nbd - 1 - atomicAdd(&j.cl_cur[j.cl_T], 1)] = g; return; }
    atomicMax(&j.cl_w[0], (unsigned long long)__double_as_longlong(a[1] - a[0]));
    atomicMax(&j.cl_w[1], (unsigned long long)__double_as_longlong(a[3] - a[2]));
    atomicAdd(&j.cl_cnt[cl_bucket(j, a[0], a[2])], 1);
}

__device__ __forceinline__ void cl_fill_item(const mel_prox_job& j, int g)
{
    const mel_dev& d = j.d;
    if (g >= d.nbd || !cl_box_ok(d, j.aabb, g)) return;
    const double* a = j.aabb + 4 * g;
    if (cl_big(j, a)) return;
    const int bk = cl_bucket(j, a[0], a[2]);
    j.cl_idx[j.cl_start[bk] + atomicAdd(&j.cl_cur[bk], 1)] = g;
}

__device__ __forceinline__ void cl_zero_item(const mel_prox_job& j, int i)
{
    if (i > j.cl_T) return;
    j.cl_cnt[i] = 0;
    j.cl_cur[i] = 0;
    if (i == 0) { j.cl_w[0] = 0ull; j.cl_w[1] = 0ull; }
}

__device__ __forceinline__ void cl_neighbour_item(const mel_prox_job& j, int b1, int lane)
{
    __shared__ int s_cl[PROX_THREADS_CL / 32][2 * CL_CAND];
    const mel_dev& d = j.d;
    if (b1 >= d.nb) return;
    if (d.b_status[b1] == MEL_STATUS_INACTIVE) { if (lane == 0) j.nbn[b1] = 0; return; }
    int* cand = s_cl[(threadIdx.x >> 5) % (PROX_THREADS_CL / 32)];
    int* srt = cand + CL_CAND;
    const double* aabb = j.aabb;
    const int cap = j.nbr_cap;
    int* out = j.nbr + (size_t)3 * cap * b1;
    const double W = __longlong_as_double((long long)j.cl_w[0]), H = __longlong_as_double((long long)j.cl_w[1]);
    int count = 0;
    for (int g1 = d.b_bd0[b1]; g1 < d.b_bd0[b1 + 1]; g1++) {
        const int count_before = count;
        const double xmin1 = aabb[4 * g1], xmax1 = aabb[4 * g1 + 1], ymin1 = aabb[4 * g1 + 2], ymax1 = aabb[4 * g1 + 3];
        // boxes left out and boxes too far out for integer cell indices: all pairs.  A big box (a
        // wall) queries the cells its own extent covers, which may be many
        bool all = !(xmin1 <= xmax1) || !(ymin1 <= ymax1) ||
                   !(fabs(ymin1 - H) < 1e12 * j.cl_h && fabs(ymax1) < 1e12 * j.cl_h &&
                     fabs(xmin1 - W - d.xmin) < 1e12 * j.cl_hx && fabs(xmax1 - d.xmin) < 1e12 * j.cl_hx);
        long long cx0 = 0, cx1 = -1, cy0 = 0, cy1 = -1;
        if (!all) {
            // a border g2 overlapping g1 (with some shift) has its lower corner in x within
            // [xmin1 - W, xmax1] modulo the period and in y within [ymin1 - H, ymax1]
            cx0 = (long long)floor((xmin1 - W - d.xmin) / j.cl_hx);
            cx1 = (long long)floor((xmax1 - d.xmin) / j.cl_hx);
            cy0 = (long long)floor((ymin1 - H) / j.cl_h);
            cy1 = (long long)floor(ymax1 / j.cl_h);
            // one more cell on every side: a corner's cell is computed from its unshifted position,
            // and rounding may put it across a cell edge from the shifted value tested here
            cx0--; cx1++; cy0--; cy1++;
            if (cx1 - cx0 + 1 > j.cl_ncx) cx1 = cx0 + j.cl_ncx - 1;      // every wrapped column once
            all = cx1 - cx0 + 1 > CL_MAX_CELLS || cy1 - cy0 + 1 > CL_MAX_CELLS ||
                  (cx1 - cx0 + 1) * (cy1 - cy0 + 1) > CL_MAX_CELLS;      // each factor bounded first: no overflow
        }
        int n = 0;
        if (!all) {
            // the cells' bucket ranges looked up by the lanes together (one cell per lane), then
            // their entries taken as one concatenated list, 32 at a time; the owner cell of list
            // item t is found by a search over the per-lane offsets kept in shared memory
            const int ncx = (int)(cx1 - cx0 + 1), ncell = ncx * (int)(cy1 - cy0 + 1);
            int* c_off = srt;                 // [33]: list offset of each lane's cell, then the total
            int* c_e0 = srt + 64;             // [32]: first entry of each lane's cell
            for (int cb = 0; cb < ncell; cb += 32) {
                const int c = cb + lane;
                int e0 = 0, len = 0;
                if (c < ncell) {
                    const long long cx = cx0 + c % ncx, cy = cy0 + c / ncx;
                    const double xc = d.xmin + ((double)cx + 0.5) * j.cl_hx, yc = ((double)cy + 0.5) * j.cl_h;
                    const int bk = cl_bucket(j, xc, yc);
                    e0 = j.cl_start[bk];
                    len = j.cl_start[bk + 1] - e0;
                }
                int incl = len;
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                c_off[lane] = incl - len;
                c_e0[lane] = e0;
                if (lane == 31) c_off[32] = total;
                __syncwarp();
                for (int tb = 0; tb < total; tb += 32) {
                    const int t = tb + lane;
                    bool ok = false;
                    int g2 = -1;
                    if (t < total) {
                        int lo = 0, hi = 32;          // last lane whose offset is <= t
                        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (c_off[mid] <= t) lo = mid; else hi = mid; }
                        g2 = j.cl_idx[c_e0[lo] + (t - c_off[lo])];
                        ok = d.bd_body[g2] != b1 && !((aabb[4 * g2 + 3] < ymin1) || (ymax1 < aabb[4 * g2 + 2]));
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, ok);
                    const int pos = n + __popc(m & ((1u << lane) - 1u));
                    if (ok && pos < CL_CAND) cand[pos] = g2;
                    n += __popc(m);
                }
                __syncwarp();
            }
            // the big boxes, outside the grid
            const int nbig = j.cl_cur[j.cl_T];
            for (int e = 0; e < nbig; e += 32) {
                bool ok = false;
                int g2 = -1;
                if (e + lane < nbig) {
                    g2 = j.cl_idx[d.nbd - 1 - (e + lane)];
                    ok = d.bd_body[g2] != b1 && !((aabb[4 * g2 + 3] < ymin1) || (ymax1 < aabb[4 * g2 + 2]));
                }
                const unsigned m = __ballot_sync(0xffffffffu, ok);
                const int pos = n + __popc(m & ((1u << lane) - 1u));
                if (ok && pos < CL_CAND) cand[pos] = g2;
                n += __popc(m);
            }
            all = n > CL_CAND;
        }
        __syncwarp();
        if (all) { nbr_scan_all(d, aabb, j.shmin, j.shmax, out, cap, b1, g1, count_before, count, lane); continue; }
        // stable rank sort of the gathered borders, then the first of each run of equal values
        for (int i = lane; i < n; i += 32) {
            const int v = cand[i];
            int r = 0;
            for (int k = 0; k < n; k++) r += (cand[k] < v) || (cand[k] == v && k < i);
            srt[r] = v;
        }
        __syncwarp();
        const int smin1 = j.shmin[g1], smax1 = j.shmax[g1];
        const int first_border = (g1 == d.b_bd0[b1]);
        for (int base = 0; base < n; base += 32) {
            const int i = base + lane;
            const bool valid = i < n && (i == 0 || srt[i] != srt[i - 1]);
            const int g2 = valid ? srt[i] : 0;
            const int b2 = valid ? d.bd_body[g2] : 0;
            const int r2 = g2 - (valid ? d.b_bd0[b2] : 0);
            int mine = 0;
            for (int pass = 0; pass < 2; pass++) {
                int k = 0;
                if (valid) {
                    const double xmin2 = aabb[4 * g2], xmax2 = aabb[4 * g2 + 1];
                    for (int s = smin1 - j.shmax[g2]; s <= smax1 - j.shmin[g2]; s++) {
                        if ((xmax2 + s * d.period > xmin1) && (xmin2 + s * d.period < xmax1)) {
                            bool dup = false;
                            if (!first_border)
                                for (int q = 0; q < count_before && q < cap; q++)
                                    if (out[3 * q] == b2 && out[3 * q + 1] == r2 && out[3 * q + 2] == s) { dup = true; break; }
                            if (dup) continue;
                            if (pass == 1) {
                                const int pos = mine + k;
                                if (pos < cap) { out[3 * pos] = b2; out[3 * pos + 1] = r2; out[3 * pos + 2] = s; }
                            }
                            k++;
                        }
                    }
                }
                if (pass == 0) {
                    int incl = k;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    const int total = __shfl_sync(0xffffffffu, incl, 31);
                    mine = count + incl - k;
                    count += total;
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
    if (lane == 0) {
        j.nbn[b1] = count;
        if (count > cap) { atomicOr(&d.err[MEL_E_NBR_OVERFLOW], 1u); atomicMax(&d.err[MEL_E_NBR_NEED], (unsigned)count); }
    }
}

// ---------------------------------------------------------------------------------------------
// segment blocks: bounding boxes of MEL_SEGB consecutive segments of a border (node1/node2 positions
// with the border's own period shifts).  Used only to skip segments that cannot pass
// Detect_Segment_Proximity; the boxes are widened by the detection distance plus a margin, so the
// accepted candidates and their order are unchanged.
// ---------------------------------------------------------------------------------------------
// Superblock boxes are unions of MEL_SEGB2 consecutive block boxes of one border.  One warp per
// superblock, a half-warp per block and a lane per segment.
static_assert(MEL_SEGB == 16 && MEL_SEGB2 == 16, "a half-warp serves a block of 16 segments, 16 blocks a superblock");
__device__ __forceinline__ void superblock_item(const mel_dev& d, int k, int lane)
{
    if (k >= d.nsblk) return;
    const int g = d.sblk_border[k];
    const int n0 = d.b_node0[d.bd_body[g]];
    const int e0 = d.bd_e0[g], nseg = d.bd_e0[g + 1] - e0 - 1;
    const int kb0 = (k - d.bd_sblk0[g]) * MEL_SEGB2, nb = min(MEL_SEGB2, d.bd_blk0[g + 1] - d.bd_blk0[g] - kb0);
    double ux0 = 1.e300, ux1 = -1.e300, uy0 = 1.e300, uy1 = -1.e300;
    for (int i = 0; i < nb; i += 8) {           // four blocks in flight a half-warp
        double2 p[8];
        double xs[8];
        bool on[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int kb = i + 2 * q + (lane >> 4), sg = (kb0 + kb) * MEL_SEGB + (lane & 15);
            on[q] = kb < nb && sg < nseg;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                // shifted (regular search) and unshifted (self search) abscissae both count
                const int e = 4 * (e0 + sg) + 1 + j;
                p[2 * q + j] = on[q] ? d.x[n0 + d.e_sn[e]] : make_double2(0., 0.);
                xs[2 * q + j] = on[q] ? p[2 * q + j].x + d.period * d.e_ss[e] : 0.;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            double x0 = 1.e300, x1 = -1.e300, y0 = 1.e300, y1 = -1.e300;
            if (on[q])
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const double2 v = p[2 * q + j];
                    x0 = fmin(x0, fmin(xs[2 * q + j], v.x)); x1 = fmax(x1, fmax(xs[2 * q + j], v.x));
                    y0 = fmin(y0, v.y); y1 = fmax(y1, v.y);
                }
            for (int o = 8; o > 0; o >>= 1) {
                x0 = fmin(x0, __shfl_xor_sync(0xffffffffu, x0, o)); x1 = fmax(x1, __shfl_xor_sync(0xffffffffu, x1, o));
                y0 = fmin(y0, __shfl_xor_sync(0xffffffffu, y0, o)); y1 = fmax(y1, __shfl_xor_sync(0xffffffffu, y1, o));
            }
            const int kb = i + 2 * q + (lane >> 4);
            if ((lane & 15) == 0 && kb < nb) d.seg_blk[d.bd_blk0[g] + kb0 + kb] = make_double4(x0, x1, y0, y1);
            ux0 = fmin(ux0, x0); ux1 = fmax(ux1, x1); uy0 = fmin(uy0, y0); uy1 = fmax(uy1, y1);
        }
    }
    ux0 = fmin(ux0, __shfl_xor_sync(0xffffffffu, ux0, 16)); ux1 = fmax(ux1, __shfl_xor_sync(0xffffffffu, ux1, 16));
    uy0 = fmin(uy0, __shfl_xor_sync(0xffffffffu, uy0, 16)); uy1 = fmax(uy1, __shfl_xor_sync(0xffffffffu, uy1, 16));
    if (lane == 0) d.seg_sblk[k] = make_double4(ux0, ux1, uy0, uy1);
}

__device__ __forceinline__ bool block_may_detect(const double4& bb, double xs, double ys, double m)
{
    return !(xs < bb.x - m || xs > bb.y + m || ys < bb.z - m || ys > bb.w + m);
}

// whether any block box of border g lies within `margin` of (x, y)
__device__ __forceinline__ bool any_near_block(const mel_dev& d, int g, double x, double y, double margin)
{
    const int blk0 = d.bd_blk0[g], blk1 = d.bd_blk0[g + 1];
    for (int ks = d.bd_sblk0[g]; ks < d.bd_sblk0[g + 1]; ks++) {
        if (!block_may_detect(d.seg_sblk[ks], x, y, margin)) continue;
        const int k0 = blk0 + (ks - d.bd_sblk0[g]) * MEL_SEGB2, k1 = min(k0 + MEL_SEGB2, blk1);
        for (int k = k0; k < k1; k += 4) {
            double4 bb[4];
#pragma unroll
            for (int q = 0; q < 4; q++) bb[q] = d.seg_blk[min(k + q, k1 - 1)];
#pragma unroll
            for (int q = 0; q < 4; q++) if (block_may_detect(bb[q], x, y, margin)) return true;
        }
    }
    return false;
}

// Calls test(seg) in all lanes for the segments of border g's blocks that lie within `margin` of (x, y),
// two blocks (32 segments, a lane each; seg -1: none) at a time in ascending order, and hit(accepted
// lanes) after each.  One warp.  A border of several superblocks has their boxes tested first, a lane
// each: without that the warp read every block's box (find_kernel for two blocks of 22,000 segments a
// border, B200: 705 us, so 128 us).  One superblock, as a grain's border has, goes straight to its blocks.
template <typename T, typename H>
__device__ __forceinline__ void for_near_segments(const mel_dev& d, int g, double x, double y, double margin, int lane, T&& test, H&& hit)
{
    const int blk0 = d.bd_blk0[g], nblk = d.bd_blk0[g + 1] - blk0, nseg = d.bd_e0[g + 1] - d.bd_e0[g] - 1;
    const int sb0 = d.bd_sblk0[g], nsb = d.bd_sblk0[g + 1] - sb0;
    for (int s0 = 0; s0 < nsb; s0 += 32) {
        unsigned sm = 1u;
        if (nsb > 1) sm = __ballot_sync(0xffffffffu, s0 + lane < nsb && block_may_detect(d.seg_sblk[sb0 + s0 + lane], x, y, margin));
        for (; sm; sm &= sm - 1) {
            const int k0 = (s0 + __ffs(sm) - 1) * MEL_SEGB2;
            const bool near = lane < 16 && k0 + lane < nblk && block_may_detect(d.seg_blk[blk0 + k0 + lane], x, y, margin);
            unsigned m = __ballot_sync(0xffffffffu, near);
            while (m) {
                const int a = __ffs(m) - 1;
                m &= m - 1;
                const int b = m ? __ffs(m) - 1 : -1;
                m &= m - 1;
                const int kb = lane < 16 ? a : b;
                int seg = kb >= 0 ? (k0 + kb) * MEL_SEGB + (lane & 15) : -1;
                if (seg >= nseg) seg = -1;
                const bool ok = seg >= 0 && test(seg);
                hit(__ballot_sync(0xffffffffu, ok), seg);
            }
        }
    }
}

// projection of slave node (xs, ys) onto segment e of a master body (nodes from mb, shifted by shM): the
// acceptance test of the regular search (Code/Proximity.h:221-270)
__device__ __forceinline__ bool project_regular(const mel_dev& d, double2 xs, int mb, int shM, int e, double dd, double cd, Proj& p)
{
    const int* sn = d.e_sn + 4 * e;
    const int* ss = d.e_ss + 4 * e;
    const double2 p1 = d.x[mb + sn[1]], p2 = d.x[mb + sn[2]];
    const double X1 = p1.x + d.period * (shM + ss[1]), Y1 = p1.y;
    const double X2 = p2.x + d.period * (shM + ss[2]), Y2 = p2.y;
    if (detect_proximity(xs.x, xs.y, X1, Y1, X2, Y2, dd) == 0) return false;
    const double2 p0 = d.x[mb + sn[0]], p3 = d.x[mb + sn[3]];
    const double X0 = p0.x + d.period * (shM + ss[0]), Y0 = p0.y;
    const double X3 = p3.x + d.period * (shM + ss[3]), Y3 = p3.y;
    p.gap = 0.; p.xsi = 0.; p.xn = p.yn = p.xt = p.yt = 0.; p.N[0] = p.N[1] = p.N[2] = p.N[3] = 0.; p.flag = 0;
    closest_linear(xs.x, xs.y, X0, Y0, X1, Y1, X2, Y2, X3, Y3, p);
    return (p.flag == -2 || p.flag == -1 || p.flag == 0) && (p.gap > -cd);
}

// the same against the body's own segment e (Code/Proximity.h:355-405); Closest_2_segment_self never
// yields flag 0, so those pairs are skipped
__device__ __forceinline__ bool project_self(const mel_dev& d, double2 xs, int NodeS, int n0, int e, double dd, double cd, Proj& p)
{
    const int* sn = d.e_sn + 4 * e;
    if (sn[1] == NodeS) return false;
    if (sn[2] == NodeS) return false;
    const double2 p1 = d.x[n0 + sn[1]], p2 = d.x[n0 + sn[2]];
    if (detect_proximity(xs.x, xs.y, p1.x, p1.y, p2.x, p2.y, dd) == 0) return false;
    if (sn[0] == NodeS || sn[3] == NodeS) return false;
    const double2 p0 = d.x[n0 + sn[0]], p3 = d.x[n0 + sn[3]];
    p.gap = 0.; p.xsi = 0.; p.xn = p.yn = p.xt = p.yt = 0.; p.N[0] = p.N[1] = p.N[2] = p.N[3] = 0.; p.flag = 0;
    closest_linear(xs.x, xs.y, p0.x, p0.y, p1.x, p1.y, p2.x, p2.y, p3.x, p3.y, p);
    return p.flag == 0 && (p.gap > -cd);
}

// margin of the box tests around (x, y): the detection distance, widened past rounding
__device__ __forceinline__ double near_margin(const mel_dev& d, double2 xs, double dd, int shM)
{
    return dd * 1.0001 + 1e-12 * (fabs(xs.x) + fabs(xs.y) + fabs(d.period * shM)) + 1e-15;
}

// ---------------------------------------------------------------------------------------------
// tasks and slots.  A body's tasks are contiguous: (border, neighbour) pairs in the reference's loop
// order (Code/Proximity.h:207-212), then self tasks per border (Code/Proximity.h:346-356); its
// slots likewise, a slot per slave border node of each task.  A pair, or a border with itself, is cut
// into pieces of TASK_NODES slave border nodes, a task each: a candidate finds its place by looking
// through all of its task (write_item), which over a border of thousands of nodes is quadratic.
// Measured on B200, two blocks of 10,000 contacts each: write_kernel 1,129 us with a task for the whole
// border, 596 with pieces.  A grain's
// border, 33 to 97 nodes, is one piece.
// ---------------------------------------------------------------------------------------------
#define TASK_NODES 128
__device__ __forceinline__ int task_pieces(int nS) { return (nS + TASK_NODES - 1) / TASK_NODES; }

__device__ __forceinline__ bool has_self(const mel_dev& d, int b)
{
    return d.self_contact && d.b_type[b] == MEL_BODY_DEFORMABLE && !d.b_per[b];
}

// a slot's slave body, slave border (global), neighbour (-1: self), slave border node and task
struct slot_ref { int b, g, q, kS, t; };
__device__ __forceinline__ slot_ref slot_of(const mel_prox_job& j, int s)
{
    const mel_dev& d = j.d;
    int lo = 0, hi = d.nb;                   // largest b with bslot0[b] <= s that has slots
    while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (j.bslot0[mid] <= s) lo = mid; else hi = mid; }
    slot_ref r;
    r.b = lo;
    int at = s - j.bslot0[lo];
    const int n = j.nbn[lo], g0 = d.b_bd0[lo], g1 = d.b_bd0[lo + 1];
    int g = g0, before = 0;                  // tasks before the border's (for the first of its neighbours)
    r.q = -1;
    for (; g < g1; g++) {                    // regular tasks
        const int nS = d.bd_e0[g + 1] - d.bd_e0[g];
        if (at < n * nS) { r.q = at / nS; at -= r.q * nS; before += r.q * task_pieces(nS); break; }
        at -= n * nS;
        before += n * task_pieces(nS);
    }
    if (g == g1)                             // self tasks
        for (g = g0; g < g1 - 1; g++) {
            const int nS = d.bd_e0[g + 1] - d.bd_e0[g];
            if (at < nS) break;
            at -= nS;
            before += task_pieces(nS);
        }
    r.g = g;
    r.kS = at;
    r.t = j.btask0[lo] + before + at / TASK_NODES;
    return r;
}

// A candidate: a = {task, slave border node, its number among the node's candidates, master entry},
// b = {slave body, slave border (global), neighbour or -1, master border (global)}
#define FIND_THREADS 128
__global__ void __launch_bounds__(FIND_THREADS) find_kernel(const mel_prox_job* J, const int* bpre, int nj, const __grid_constant__ mel_prox_job one)
{
    __shared__ mel_prox_job sj;
    __shared__ slot_ref s_near[FIND_THREADS];
    __shared__ int s_n;
    const int jj = J ? block_job(bpre, nj) : 0;
    {
        const int* src = reinterpret_cast<const int*>(J ? J + jj : &one);
        int* dst = reinterpret_cast<int*>(&sj);
        for (int k = threadIdx.x; k < (int)(sizeof(mel_prox_job) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
    }
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    grid_wait();
    grid_release();
    const mel_prox_job& j = sj;
    const mel_dev& d = sj.d;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = ((int)blockIdx.x - (J ? bpre[jj] : 0)) * FIND_THREADS + (int)threadIdx.x;
    // a thread per slot: is the slave node near any block of the master?
    if (s < j.nslot) {
        const slot_ref r = slot_of(j, s);
        const double2 xs = d.x[d.b_node0[r.b] + d.e_node[d.bd_e0[r.g] + r.kS]];
        const double dd = d.b_dist[3 * r.b + 1];
        bool near = false;
        if (r.q >= 0) {
            const int* nb = j.nbr + 3 * ((size_t)j.nbr_cap * r.b + r.q);
            near = any_near_block(d, d.b_bd0[nb[0]] + nb[1], xs.x - d.period * nb[2], xs.y, near_margin(d, xs, dd, nb[2]));
        } else
            for (int g = d.b_bd0[r.b]; g < d.b_bd0[r.b + 1] && !near; g++)
                near = any_near_block(d, g, xs.x, xs.y, near_margin(d, xs, dd, 0));
        if (near) s_near[atomicAdd(&s_n, 1)] = r;
    }
    __syncthreads();
    // a warp per near slot: its candidates, in segment order
    for (int i = warp; i < s_n; i += FIND_THREADS / 32) {
        const slot_ref r = s_near[i];
        const int n0 = d.b_node0[r.b], NodeS = d.e_node[d.bd_e0[r.g] + r.kS];
        const double2 xs = d.x[n0 + NodeS];
        const double dd = d.b_dist[3 * r.b + 1], cd = d.b_dist[3 * r.b + 2];
        int found = 0;
        auto list = [&](unsigned m, int e, int gM) {
            if (!m) return;
            int at = 0;
            if (lane == 0) at = atomicAdd(j.ncand, __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if ((m >> lane) & 1u) {
                const int k = __popc(m & ((1u << lane) - 1u));
                if (at + k < j.cand_cap) {
                    j.cand[2 * (size_t)(at + k)] = make_int4(r.t, r.kS, found + k, e);
                    j.cand[2 * (size_t)(at + k) + 1] = make_int4(r.b, r.g, r.q, gM);
                }
            }
            found += __popc(m);
        };
        Proj p;
        if (r.q >= 0) {
            const int* nb = j.nbr + 3 * ((size_t)j.nbr_cap * r.b + r.q);
            const int bM = nb[0], shM = nb[2], gM = d.b_bd0[bM] + nb[1], mb = d.b_node0[bM], eM0 = d.bd_e0[gM];
            for_near_segments(d, gM, xs.x - d.period * shM, xs.y, near_margin(d, xs, dd, shM), lane,
                [&](int seg) { return project_regular(d, xs, mb, shM, eM0 + seg, dd, cd, p); },
                [&](unsigned m, int seg) { list(m, eM0 + seg, gM); });
        } else
            for (int gM = d.b_bd0[r.b]; gM < d.b_bd0[r.b + 1]; gM++) {
                const int eM0 = d.bd_e0[gM];
                for_near_segments(d, gM, xs.x, xs.y, near_margin(d, xs, dd, 0), lane,
                    [&](int seg) { return project_self(d, xs, NodeS, n0, eM0 + seg, dd, cd, p); },
                    [&](unsigned m, int seg) { list(m, eM0 + seg, gM); });
            }
        if (lane == 0 && found) atomicAdd(&j.tcand[r.t], found);
    }
}

// candidate i into its task's bucket (any order); leaves tcand at zero
__device__ __forceinline__ void bucket_item(const mel_prox_job& j, int i)
{
    if (i >= j.ncont_new) return;
    const int t = j.cand[2 * (size_t)i].x;
    j.bucket[j.toff[t] + atomicSub(&j.tcand[t], 1) - 1] = i;
}

// ---------------------------------------------------------------------------------------------
// History.  A candidate inherits from the first old element, in list order, of its slave border node on
// the same master border within one segment.  A warp looks through the slave body's old elements, 32 at
// a time; those of a body with more than LONG_LIST are chained per border entry first (in any order: the
// first in the list is the smallest index), by the launch that makes the boxes.  A chain's head is
// valid when it carries the run's stamp.  Measured on B200, two blocks of n contacts each, an update
// looking through / chained: n 1,000 209 and 197 us, n 3,000 308 and 248 us, n 10,000 933 and 450 us; equal
// at 300.
// ---------------------------------------------------------------------------------------------
#define LONG_LIST 256
__device__ __forceinline__ int old_entry(const mel_dev& d, const mel_contact& o) { return d.bd_e0[d.b_bd0[o.bodyS] + o.borderS] + o.border_nodeS; }
__device__ __forceinline__ void link_item(const mel_prox_job& j, int c)
{
    const mel_dev& d = j.d;
    if (c >= d.ncont) return;
    const mel_contact& o = d.cont[c];
    if (j.b_cont0[o.bodyS + 1] - j.b_cont0[o.bodyS] <= LONG_LIST) return;
    const unsigned long long was = atomicExch(&j.e_head[old_entry(d, o)], (unsigned long long)j.stamp << 32 | (unsigned)c);
    j.c_next[c] = (unsigned)(was >> 32) == j.stamp ? (int)(unsigned)was : -1;
}

// index of the old element that a candidate of slave entry eS inherits from, or -1; one warp
__device__ __forceinline__ int old_element(const mel_prox_job& j, int bS, int rS, int kS, int eS, int bM, int rM, int seg, int lane)
{
    const mel_dev& d = j.d;
    const int o0 = j.b_cont0[bS], o1 = j.b_cont0[bS + 1];
    if (o1 - o0 > LONG_LIST) {
        const unsigned long long h = j.e_head[eS];
        int best = 0x7fffffff;
        for (int k = (unsigned)(h >> 32) == j.stamp ? (int)(unsigned)h : -1; k >= 0; k = j.c_next[k]) {
            const mel_contact& o = d.cont[k];
            if (o.bodyM == bM && o.borderM == rM && abs(o.segmentM - seg) <= 1 && k < best) best = k;
        }
        return best == 0x7fffffff ? -1 : best;
    }
    for (int k = o0; k < o1; k += 32) {
        bool match = false;
        if (k + lane < o1) {
            const mel_contact& o = d.cont[k + lane];
            match = o.border_nodeS == kS && o.borderS == rS && o.bodyM == bM && o.borderM == rM && abs(o.segmentM - seg) <= 1;
        }
        const unsigned m = __ballot_sync(0xffffffffu, match);
        if (m) return k + __ffs(m) - 1;
    }
    return -1;
}

// candidate i at its place in the new list; one warp
__device__ __forceinline__ void write_item(const mel_prox_job& j, int i, int lane)
{
    if (i >= j.ncont_new) return;
    const mel_dev& d = j.d;
    const int4 a = j.cand[2 * (size_t)i], c4 = j.cand[2 * (size_t)i + 1];
    const int t = a.x, kS = a.y, e = a.w, bS = c4.x, gS = c4.y, q = c4.z, gM = c4.w;
    const int t0 = j.toff[t], t1 = j.toff[t + 1];
    int rank = 0;
    for (int k = t0 + lane; k < t1; k += 32) {
        const int4 o = j.cand[2 * (size_t)j.bucket[k]];
        rank += o.y < kS || (o.y == kS && o.z < a.z);
    }
    for (int o = 16; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    const int pos = t0 + rank;
    const int rS = gS - d.b_bd0[bS], eS = d.bd_e0[gS] + kS, NodeS = d.e_node[eS], n0 = d.b_node0[bS];
    const int seg = e - d.bd_e0[gM];
    int bM = bS, shM = 0;
    if (q >= 0) {
        const int* nb = j.nbr + 3 * ((size_t)j.nbr_cap * bS + q);
        bM = nb[0];
        shM = nb[2];
    }
    const int rM = gM - d.b_bd0[bM];
    if (lane == 0) {
        if (rank == 0) { j.tkey[t] = bM; atomicAdd(&j.inc_cnt[bM], 1); }
        d.cont_w[pos] = 0.;
    }
    mel_contact* out = j.cont_new + pos;
    if (q >= 0 && j.have_old) {
        const int k = old_element(j, bS, rS, kS, eS, bM, rM, seg, lane);
        if (k >= 0) {
            const int* src = reinterpret_cast<const int*>(d.cont + k);
            int* dst = reinterpret_cast<int*>(out);
            for (int w = lane; w < (int)(sizeof(mel_contact) / sizeof(int)); w += 32) dst[w] = src[w];
            __syncwarp();
            if (lane == 0) { out->bodyS = bS; out->pad_ = 0; }
            return;
        }
    }
    if (lane) return;
    const double2 xs = d.x[n0 + NodeS];
    const double dd = d.b_dist[3 * bS + 1], cd = d.b_dist[3 * bS + 2];
    Proj p;
    const bool ok = q >= 0 ? project_regular(d, xs, d.b_node0[bM], shM, e, dd, cd, p) : project_self(d, xs, NodeS, n0, e, dd, cd, p);
    if (!ok) atomicOr(&d.err[MEL_E_BOUNDS], 4u);         // both passes read the same positions
    mel_contact c;
    c.bodyS = bS; c.borderS = rS; c.border_nodeS = kS; c.nodeS = NodeS;
    c.bodyM = bM; c.borderM = rM; c.shiftM = shM; c.segmentM = seg;
    for (int k = 0; k < 4; k++) { c.nodeM[k] = d.e_sn[4 * e + k]; c.shiftMk[k] = q >= 0 ? d.e_ss[4 * e + k] : 0; c.shapeM[k] = p.N[k]; }
    c.gapn = p.gap; c.vgapn = 0.; c.gapt = 0.; c.vgapt = 0.; c.xsi = p.xsi;
    c.xnorm = p.xn; c.ynorm = p.yn; c.xtan = p.xt; c.ytan = p.yt;
    if (q >= 0) {
        const double* rgM = d.rg + MEL_RIGID_NF * bM;
        const double* rgS = d.rg + MEL_RIGID_NF * bS;
        if (rgM[MEL_RG_MASS] == 0.) c.effective_mass = 0.;
        else if (rgS[MEL_RG_MASS] == 0.) c.effective_mass = 0.;
        else c.effective_mass = 1. / (rgM[MEL_RG_INV_MASS] + rgS[MEL_RG_INV_MASS]);
    } else c.effective_mass = d.rg[MEL_RIGID_NF * bS + MEL_RG_MASS];
    c.length = d.e_len[eS]; c.fx = 0.; c.fy = 0.;
    c.nb_internal = 0; c.internal[0] = 0.; c.internal[1] = 0.; c.internal[2] = 0.;
    c.pad_ = 1;                                          // new elements get vgapn/vgapt in the carry
    *out = c;
}

// ---------------------------------------------------------------------------------------------
// incoming (master-side) contact ranges of each body in send order.  Send_contact_forces runs over
// the sending bodies in index order (Code/Solver.h:61-62) and each sender over its contact list, so
// the incoming ranges of master body B are the tasks whose master is B, in ascending task order; tasks
// without contacts are left out.  Tasks are grouped by master with a counting pass and an atomic fill,
// then each group is put back in ascending order by a rank sort (task ids are unique).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void inc_fill_item(const mel_prox_job& j, int t)
{
    if (t >= j.ntask || j.toff[t + 1] == j.toff[t]) return;
    const int key = j.tkey[t];
    j.inc_task[j.b_inc0[key] + atomicSub(&j.inc_cnt[key], 1) - 1] = t;
}

// first index with bodyS >= b of a body-major list
__device__ __forceinline__ void body_range_item(const mel_contact* cont, int n, int nb, int* b_cont0, int b)
{
    if (b > nb) return;
    int lo = 0, hi = n;
    while (lo < hi) { int mid = (lo + hi) >> 1; if (cont[mid].bodyS < b) lo = mid + 1; else hi = mid; }
    b_cont0[b] = lo;
}

// Newly created elements leave vgapn/vgapt unassigned in the reference: they keep the values of the
// element pushed before them in the slave body's list (the reused new_contact variable,
// Code/Proximity.h:286-313); self contacts use a fresh variable (Code/Proximity.h:350).  One warp
// per body, 32 contacts at a time: a new element takes the values of the last inherited non-self
// element before it (found by ballot within the 32, else carried over from earlier ones).
__device__ __forceinline__ void carry_item(mel_contact* cont, int b, int c0, int c1, int lane)
{
    double vn = 0., vt = 0.;                 // carried value (equal in all lanes)
    for (int base = c0; base < c1; base += 32) {
        const int c = base + lane;
        const bool valid = c < c1;
        int bodyM = -1, pad = 0;
        double gn = 0., gt = 0.;
        if (valid) { bodyM = cont[c].bodyM; pad = cont[c].pad_; gn = cont[c].vgapn; gt = cont[c].vgapt; }
        const bool self = bodyM == b;
        const bool src = valid && !self && !pad;          // inherited non-self elements set the value
        const unsigned m = __ballot_sync(0xffffffffu, src);
        const unsigned lower = m & ((1u << lane) - 1u);
        const int from = lower ? 31 - __clz(lower) : 0;
        const double sn = __shfl_sync(0xffffffffu, gn, from), st = __shfl_sync(0xffffffffu, gt, from);
        if (valid && pad) {
            if (self) { cont[c].vgapn = 0.; cont[c].vgapt = 0.; }
            else if (lower) { cont[c].vgapn = sn; cont[c].vgapt = st; }
            else { cont[c].vgapn = vn; cont[c].vgapt = vt; }
            cont[c].pad_ = 0;
        } else if (valid && self) {
            cont[c].pad_ = 0;
        }
        if (m) {
            const int last = 31 - __clz(m);
            vn = __shfl_sync(0xffffffffu, gn, last);
            vt = __shfl_sync(0xffffffffu, gt, last);
        }
    }
}

// body b of the new list (one warp): its incoming ranges, its contact range and the carry
__device__ __forceinline__ void body_item(const mel_prox_job& j, int b, int lane)
{
    const mel_dev& d = j.d;
    if (b >= d.nb) return;
    const int i0 = j.b_inc0[b], n = j.b_inc0[b + 1] - i0;
    for (int i = lane; i < n; i += 32) {
        const int t = j.inc_task[i0 + i];
        int r = 0;
        for (int k = 0; k < n; k++) r += j.inc_task[i0 + k] < t;
        j.inc_rng[i0 + r] = make_int2(j.toff[t], j.toff[t + 1]);
    }
    const int c0 = j.toff[j.btask0[b]], c1 = j.toff[j.btask0[b + 1]];
    if (lane == 0) {
        j.b_cont0[b] = c0;
        if (b == d.nb - 1) j.b_cont0[d.nb] = c1;
    }
    carry_item(d.cont, b, c0, c1, lane);
}

// ---------------------------------------------------------------------------------------------
// job-table launches: blocks [bpre[j], bpre[j+1]) serve member j.  The block copies the member's
// job into shared memory; item `it` of the member is handled by TPI consecutive threads (TPI 32:
// one warp per item, TPI 1: one thread).
// ---------------------------------------------------------------------------------------------
#define PROX_THREADS 256
static_assert(PROX_THREADS == PROX_THREADS_CL, "cell-list scratch is sized for the job kernels' block");
#define JOB_KERNEL(name, TPI, ...)                                                                  \
    __global__ void __launch_bounds__(PROX_THREADS) name(const mel_prox_job* J, const int* bpre, int nj, \
                                                         const __grid_constant__ mel_prox_job one)  \
    {                                                                                               \
        __shared__ mel_prox_job sj;                                                                 \
        const int jj = J ? block_job(bpre, nj) : 0;                                                         \
        {                                                                                           \
            const int* src = reinterpret_cast<const int*>(J ? J + jj : &one);                                  \
            int* dst = reinterpret_cast<int*>(&sj);                                                 \
            for (int k = threadIdx.x; k < (int)(sizeof(mel_prox_job) / sizeof(int)); k += blockDim.x) dst[k] = src[k]; \
        }                                                                                           \
        __syncthreads();                                                                            \
        grid_wait();                                                                                \
        grid_release();                                                                             \
        const int it = ((int)blockIdx.x - (J ? bpre[jj] : 0)) * (PROX_THREADS / (TPI)) + (int)threadIdx.x / (TPI); \
        const int lane = threadIdx.x & 31;                                                          \
        (void)lane;                                                                                 \
        const mel_prox_job& j = sj;                                                                 \
        const mel_dev& d = sj.d;                                                                    \
        (void)j; (void)d;                                                                           \
        __VA_ARGS__;                                                                                \
    }

// the boxes, the chains of old elements, and what the first neighbour attempt starts from: cleared
// overflow words and buckets
JOB_KERNEL(boxes_kernel, 32,
    const int nz = j.cl_on ? j.cl_T / 32 + 1 : 0;
    if (it < d.nbd) aabb_item(d, j.aabb, j.shmin, j.shmax, it, lane);
    else if (it < d.nbd + d.nsblk) superblock_item(d, it - d.nbd, lane);
    else if (it < d.nbd + d.nsblk + nz) cl_zero_item(j, 32 * (it - d.nbd - d.nsblk) + lane);
    else if (j.link) link_item(j, 32 * (it - d.nbd - d.nsblk - nz) + lane);
    if (it == 0 && lane == 0) { d.err[MEL_E_NBR_OVERFLOW] = 0u; d.err[MEL_E_NBR_NEED] = 0u; })
JOB_KERNEL(neighbour_kernel, 32, neighbour_item(d, j.aabb, j.shmin, j.shmax, j.nbr, j.nbn, j.nbr_cap, it, lane))
JOB_KERNEL(cl_zero_kernel, 1, cl_zero_item(j, it))
JOB_KERNEL(cl_count_kernel, 1, cl_count_item(j, it))
JOB_KERNEL(cl_fill_kernel, 1, cl_fill_item(j, it))
JOB_KERNEL(cl_neighbour_kernel, 32, cl_neighbour_item(j, it, lane))
// (a run leaves these at zero; cleared for new buffers and after a run that stopped half way)
JOB_KERNEL(clear_kernel, 1,
    if (it < j.tcand_n) j.tcand[it] = 0;
    if (it <= d.nb) j.inc_cnt[it] = 0;
    if (it == 0) *j.ncand = 0)
JOB_KERNEL(bucket_kernel, 1, bucket_item(j, it))
JOB_KERNEL(write_kernel, 32, write_item(j, it, lane))
JOB_KERNEL(inc_fill_kernel, 1, inc_fill_item(j, it))
JOB_KERNEL(bodies_kernel, 32, body_item(j, it, lane); if (it == 0 && lane == 0) *j.ncand = 0)
JOB_KERNEL(body_range_kernel, 1, body_range_item(d.cont, d.ncont, d.nb, j.b_cont0, it))

// one block per member: tasks and slots of every body, their offsets (btask0, bslot0), and the words
// the host needs after the neighbour stage (0-4)
__global__ void __launch_bounds__(1024) tasks_kernel(const mel_prox_job* J, int nj, const __grid_constant__ mel_prox_job one)
{
    __shared__ int s[32];
    grid_wait();
    grid_release();
    const mel_prox_job& j = J ? J[blockIdx.x] : one;
    const mel_dev& d = j.d;
    int t0 = 0, s0 = 0;
    for (int base = 0; base < d.nb; base += 1024) {
        const int b = base + (int)threadIdx.x;
        int tc = 0, sc = 0;
        if (b < d.nb) {
            const int g0 = d.b_bd0[b], g1 = d.b_bd0[b + 1], per = j.nbn[b] + (has_self(d, b) ? 1 : 0);
            for (int g = g0; g < g1; g++) tc += task_pieces(d.bd_e0[g + 1] - d.bd_e0[g]);
            tc *= per;
            sc = (d.bd_e0[g1] - d.bd_e0[g0]) * per;
        }
        int tt, st;
        const int ta = block_scan(tc, s, tt), sa = block_scan(sc, s, st);
        if (b < d.nb) { j.btask0[b] = t0 + ta; j.bslot0[b] = s0 + sa; }
        t0 += tt;
        s0 += st;
    }
    if (threadIdx.x == 0) {
        j.btask0[d.nb] = t0;
        j.bslot0[d.nb] = s0;
        int* r = j.readback;
        r[0] = (int)d.err[MEL_E_NAN];
        r[1] = (int)d.err[MEL_E_NBR_OVERFLOW];
        r[2] = (int)d.err[MEL_E_NBR_NEED];
        r[3] = t0;
        r[4] = s0;
    }
}

// one thread per member: clear the neighbour-overflow words before another attempt
__global__ void nbr_clear_kernel(const mel_prox_job* J, int nj, const __grid_constant__ mel_prox_job one)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nj) return;
    const mel_dev& d = J ? J[k].d : one.d;
    d.err[MEL_E_NBR_OVERFLOW] = 0u;
    d.err[MEL_E_NBR_NEED] = 0u;
}
} // namespace mel

// =============================================================================================
// host driver
// =============================================================================================
static int ensure_impl(void** p, size_t* cap_bytes, size_t need, const char* what)
{
    if (need <= *cap_bytes && *p) return 0;
    size_t nc = 2 * need + 4096;            // doubling: few reallocations (each free synchronises the device)
    void* np = nullptr;
    cudaError_t e = cudaMalloc(&np, nc);
    if (e != cudaSuccess) {
        mel_set_error("allocation of %zu bytes for %s failed: %s", nc, what, cudaGetErrorString(e));
        return 1;
    }
    if (*p) cudaFree(*p);
    *p = np;
    *cap_bytes = nc;
    return 0;
}
#define ensure(p, cap, need) ensure_impl(p, cap, need, #p)

// launch errors and stream failures of the pipeline, reported with their CUDA error and line
static int launch_status(int line)
{
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return MEL_OK;
    mel_set_cuda_error(e, "proximity kernel launch", __FILE__, line);
    return MEL_ERR_CUDA;
}
static bool sync_failed(cudaStream_t s, int line)
{
    cudaError_t e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) return false;
    mel_set_cuda_error(e, "proximity stream", __FILE__, line);
    return true;
}

// Staging of a run: job tables, block prefixes and scan jobs are written to pinned host memory and
// copied to the same offsets of a device buffer on the run's stream; the space is reused after
// each synchronisation of the stream.  The read-back words of the members live apart.
struct mel_prox_stage {
    char* h = nullptr; char* dv = nullptr; size_t cap = 0, used = 0;
    int* rb = nullptr; int rb_cap = 0;       // 8 words per member, pinned host memory the kernels write to
    std::vector<std::pair<char*, char*>> retired;               // outgrown buffers, freed after a sync
};

static void stage_release_retired(mel_prox_stage& S)
{
    for (auto& b : S.retired) { cudaFreeHost(b.first); cudaFree(b.second); }
    S.retired.clear();
}

void mel_prox_stage_free(mel_prox_stage* S)
{
    if (!S) return;
    stage_release_retired(*S);
    if (S->h) cudaFreeHost(S->h);
    if (S->dv) cudaFree(S->dv);
    if (S->rb) cudaFreeHost(S->rb);
    delete S;
}

// copies `bytes` from src to the device side of the stage (stream ordered); nullptr on failure
static void* stage_upload(mel_prox_stage& S, const void* src, size_t bytes, cudaStream_t s)
{
    const size_t off = (S.used + 15) & ~(size_t)15;
    if (off + bytes > S.cap) {
        // grow: data already staged may still be read by work on the stream, so the old buffers
        // are kept until the next synchronisation
        size_t nc = 2 * (off + bytes) + (1 << 16);
        char *nh = nullptr, *nd = nullptr;
        if (cudaMallocHost(&nh, nc) != cudaSuccess) return nullptr;
        if (cudaMalloc(&nd, nc) != cudaSuccess) { cudaFreeHost(nh); return nullptr; }
        if (S.h) S.retired.push_back({ S.h, S.dv });
        S.h = nh; S.dv = nd; S.cap = nc;
        S.used = 0;
        return stage_upload(S, src, bytes, s);
    }
    memcpy(S.h + off, src, bytes);
    if (cudaMemcpyAsync(S.dv + off, S.h + off, bytes, cudaMemcpyHostToDevice, s) != cudaSuccess) return nullptr;
    S.used = off + bytes;
    return S.dv + off;
}

namespace {

typedef void (*job_kernel_t)(const mel_prox_job*, const int*, int, const mel_prox_job);

// members of a launch: a table on the device, or the one member as the kernels' argument
struct job_table { const mel_prox_job* J; mel_prox_job one; };

struct run_ctx {
    mel_prox_stage& S;
    cudaStream_t s;
    int launches;
};

// scratch ints of an exclusive scan of n entries (block totals of every level)
size_t scan_scratch_ints(int n)
{
    size_t t = 0;
    while (true) {
        int nblk = (n + SCAN_ITEMS) / SCAN_ITEMS;
        t += (size_t)nblk + 1 + nblk + 2;
        if (nblk <= 1) break;
        n = nblk;
    }
    return t;
}

// kernel k over items[j] items of member j of the job table T (TPI threads per item)
int launch_jobs(run_ctx& C, job_kernel_t k, const job_table& T, const std::vector<int>& items, int tpi, int threads = PROX_THREADS)
{
    const int nj = (int)items.size();
    const int per_block = threads / tpi;
    std::vector<int> bpre(nj + 1, 0);
    for (int j = 0; j < nj; j++) bpre[j + 1] = bpre[j] + (items[j] + per_block - 1) / per_block;
    if (bpre[nj] == 0) return MEL_OK;
    const int* dp = T.J ? (const int*)stage_upload(C.S, bpre.data(), sizeof(int) * (nj + 1), C.s) : nullptr;
    if (T.J && !dp) { mel_set_error("proximity staging upload failed"); return MEL_ERR_CUDA; }
    launch_dependent(k, bpre[nj], threads, 0, C.s, T.J, dp, nj, T.one);
    C.launches++;
    return MEL_OK;
}

// exclusive scans: req[j] scans in[0..n) into out[0..n] using the scratch ws (scan_scratch_ints(n))
struct scan_req { const int* in; int* out; int n; int* ws; int* total = nullptr; };
// the jobs and block prefixes of a scan launch, as its argument or on the device
bool scan_pack(run_ctx& C, const std::vector<mel_scan_job>& jobs, const std::vector<int>& bpre, mel::scan_args& A)
{
    memset(&A, 0, sizeof A);
    A.nj = (int)jobs.size();
    if (A.nj <= SCAN_INLINE) {
        for (int j = 0; j < A.nj; j++) A.job[j] = jobs[j];
        for (int j = 0; j <= A.nj; j++) A.pre[j] = bpre[j];
        return true;
    }
    A.J = (const mel_scan_job*)stage_upload(C.S, jobs.data(), sizeof(mel_scan_job) * jobs.size(), C.s);
    A.bpre = (const int*)stage_upload(C.S, bpre.data(), sizeof(int) * bpre.size(), C.s);
    if (A.J && A.bpre) return true;
    mel_set_error("proximity staging upload failed");
    return false;
}
int scan_many(run_ctx& C, const std::vector<scan_req>& req)
{
    if (req.empty()) return MEL_OK;
    const int nj = (int)req.size();
    std::vector<mel_scan_job> jobs(nj), adds;
    std::vector<int> bpre(nj + 1, 0), apre(1, 0);
    std::vector<scan_req> next;
    for (int j = 0; j < nj; j++) {
        const int nblk = (req[j].n + SCAN_ITEMS) / SCAN_ITEMS;      // covers index n as well
        jobs[j] = { req[j].in, req[j].out, req[j].n, req[j].ws, nblk > 1 ? nullptr : req[j].total };
        bpre[j + 1] = bpre[j] + nblk;
        if (nblk > 1) {                                              // block totals scanned the same way
            int* soff = req[j].ws + nblk + 1;
            next.push_back({ req[j].ws, soff, nblk, soff + nblk + 2, req[j].total });
            adds.push_back({ soff, req[j].out, req[j].n + 1, nullptr, nullptr });
            apre.push_back(apre.back() + nblk);
        }
    }
    mel::scan_args A;
    if (!scan_pack(C, jobs, bpre, A)) return MEL_ERR_CUDA;
    launch_dependent(mel::scan_block_kernel, bpre[nj], SCAN_BLOCK, 0, C.s, A);
    C.launches++;
    if (next.empty()) return MEL_OK;
    if (int rc = scan_many(C, next)) return rc;
    if (!scan_pack(C, adds, apre, A)) return MEL_ERR_CUDA;
    launch_dependent(mel::scan_add_kernel, apre.back(), SCAN_BLOCK, 0, C.s, A);
    C.launches++;
    return MEL_OK;
}

mel_prox_job make_job(const mel_prox_member& m, int* readback)
{
    mel_prox_job j;
    memset(&j, 0, sizeof j);
    const mel_prox_state& P = *m.P;
    j.d = *m.d;
    j.aabb = P.aabb; j.shmin = P.shmin; j.shmax = P.shmax;
    j.nbr = P.nbr; j.nbn = P.nbn; j.nbr_cap = P.nbr_cap;
    j.ntask = P.ntask; j.nslot = P.nslot; j.have_old = m.d->ncont > 0 ? 1 : 0;
    j.btask0 = P.btask0; j.bslot0 = P.bslot0;
    j.cand = (int4*)P.cand; j.cand_cap = P.cand_cap; j.ncand = P.ncand; j.ncont_new = P.ncont_new;
    j.tcand = P.tcand; j.tcand_n = (int)(P.tcand_bytes / sizeof(int)); j.toff = P.toff; j.bucket = P.bucket; j.tkey = P.tkey;
    j.inc_task = P.inc_task; j.inc_cnt = P.inc_cnt;
    j.inc_rng = P.inc_rng; j.b_inc0 = P.b_inc0; j.b_cont0 = P.b_cont0;
    j.cont_new = P.cont_alt;
    j.e_head = P.e_head; j.c_next = P.c_next; j.stamp = P.stamp; j.link = m.d->ncont > LONG_LIST ? 1 : 0;
    j.readback = readback;
    j.cl_on = P.cl_on; j.cl_T = P.cl_T; j.cl_ncx = P.cl_ncx; j.cl_h = P.cl_h; j.cl_hx = P.cl_hx;
    j.cl_cnt = P.cl_cnt; j.cl_cur = P.cl_cur; j.cl_start = P.cl_start; j.cl_idx = P.cl_idx; j.cl_w = P.cl_w;
    return j;
}

// job table of the members idx (read-back words by member index)
bool make_jobs(run_ctx& C, mel_prox_member* m, const std::vector<int>& idx, std::vector<mel_prox_job>& hj, job_table& T)
{
    hj.clear();
    for (int i : idx) hj.push_back(make_job(m[i], C.S.rb + 8 * i));
    T.J = nullptr;
    T.one = hj[0];
    if (hj.size() == 1) return true;
    T.J = (const mel_prox_job*)stage_upload(C.S, hj.data(), sizeof(mel_prox_job) * hj.size(), C.s);
    if (!T.J) mel_set_error("proximity staging upload failed");
    return T.J != nullptr;
}

template <typename F>
std::vector<int> items_of(const std::vector<mel_prox_job>& hj, F&& f)
{
    std::vector<int> v;
    for (const mel_prox_job& j : hj) v.push_back(f(j));
    return v;
}

bool stage_ready(mel_prox_stage*& stage, int n)
{
    if (!stage) stage = new mel_prox_stage();
    mel_prox_stage& S = *stage;
    if (S.rb_cap >= n) return true;
    if (S.rb) { cudaFreeHost(S.rb); S.rb = nullptr; }
    S.rb_cap = 0;
    const int cap = std::max(n, 16);
    if (cudaMallocHost(&S.rb, sizeof(int) * 8 * (size_t)cap) != cudaSuccess) return false;
    memset(S.rb, 0, sizeof(int) * 8 * (size_t)cap);
    S.rb_cap = cap;
    return true;
}

// waits until the members' read-back words are there; the stage space is free again afterwards
bool read_back(run_ctx& C)
{
    if (sync_failed(C.s, __LINE__)) return false;
    C.S.used = 0;
    stage_release_retired(C.S);
    return true;
}

}  // namespace

int mel_run_proximity_many(mel_prox_member* m, int n, mel_prox_stage*& stage, int& launches, cudaStream_t s)
{
    using namespace mel;
    if (n <= 0) return MEL_OK;
    if (!stage_ready(stage, n)) { mel_set_error("proximity read-back buffers could not be allocated"); return MEL_ERR_OOM; }
    run_ctx C{ *stage, s, 0 };
    std::vector<mel_prox_job> hj;
    std::vector<int> act;
    job_table T;
    int rc;
    for (int i = 0; i < n; i++) {
        m[i].rc = MEL_OK;
        m[i].msg.clear();
        mel_prox_state& P = *m[i].P;
        if (ensure((void**)&P.scan_ws, &P.scan_ws_bytes, sizeof(int) * scan_scratch_ints(std::max(m[i].d->nb, P.cl_T)))) return MEL_ERR_OOM;
        if (m[i].d->ncont > LONG_LIST && ensure((void**)&P.c_next, &P.c_next_bytes, sizeof(int) * (size_t)m[i].d->ncont)) return MEL_ERR_OOM;
        if (++P.stamp == 0) {                            // stamps begin again: no head may carry an old one
            cudaMemsetAsync(P.e_head, 0, sizeof(unsigned long long) * (size_t)m[i].d->ne, s);
            P.stamp = 1;
        }
        act.push_back(i);
    }
    // 1. border boxes, segment-block boxes and the chains of old elements
    if (!make_jobs(C, m, act, hj, T)) return MEL_ERR_CUDA;
    if ((rc = launch_jobs(C, boxes_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.d.nbd + j.d.nsblk + (j.cl_on ? j.cl_T / 32 + 1 : 0) + (j.link ? (j.d.ncont + 31) / 32 : 0); }), 32))) return rc;
    // 2. neighbours and the task counts; a member whose neighbour lists overflow grows them and
    //    repeats this stage (up to 4 attempts)
    std::vector<int> pend = act;
    for (int attempt = 0; attempt < 4 && !pend.empty(); attempt++) {
        const int np = (int)pend.size();
        // members with the cell list: bucket the border boxes (counting sort), then query; the
        // others: all pairs of bodies
        bool any_cl = false, any_ap = false;
        if (attempt > 0) {
            if (!make_jobs(C, m, pend, hj, T)) return MEL_ERR_CUDA;
            nbr_clear_kernel<<<(np + 127) / 128, 128, 0, s>>>(T.J, np, T.one); C.launches++;
            if ((rc = launch_jobs(C, cl_zero_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.cl_on ? j.cl_T + 1 : 0; }), 1))) return rc;
        }
        for (const mel_prox_job& jj : hj) { any_cl = any_cl || jj.cl_on; any_ap = any_ap || !jj.cl_on; }
        if (any_cl) {
            if ((rc = launch_jobs(C, cl_count_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.cl_on ? j.d.nbd : 0; }), 1))) return rc;
            std::vector<scan_req> sc;
            for (int i : pend) if (m[i].P->cl_on) sc.push_back({ m[i].P->cl_cnt, m[i].P->cl_start, m[i].P->cl_T, m[i].P->scan_ws });
            if ((rc = scan_many(C, sc))) return rc;
            if ((rc = launch_jobs(C, cl_fill_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.cl_on ? j.d.nbd : 0; }), 1))) return rc;
            if ((rc = launch_jobs(C, cl_neighbour_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.cl_on ? j.d.nb : 0; }), 32))) return rc;
        }
        if (any_ap)
            if ((rc = launch_jobs(C, neighbour_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.cl_on ? 0 : j.d.nb; }), 32))) return rc;
        launch_dependent(tasks_kernel, np, 1024, 0, s, T.J, np, T.one); C.launches++;
        if ((rc = launch_status(__LINE__))) return rc;
        if (!read_back(C)) return MEL_ERR_CUDA;
        std::vector<int> retry;
        for (int i : pend) {
            const int* r = C.S.rb + 8 * i;
            mel_prox_state& P = *m[i].P;
            if (r[0]) {
                m[i].rc = MEL_ERR_NAN;
                char buf[160];
                if (r[0] & 1) snprintf(buf, sizeof buf, "non-finite node positions at the proximity update");
                else snprintf(buf, sizeof buf, "a border box spans more than %d periods: diverged positions", MEL_MAX_SHIFT_SPAN);
                m[i].msg = buf;
                continue;
            }
            if (r[1]) {
                const int need = r[2] + 16;
                cudaFree(P.nbr); P.nbr = nullptr;
                if (cudaMalloc(&P.nbr, sizeof(int) * 3 * (size_t)need * m[i].d->nb) != cudaSuccess) {
                    mel_set_error("allocation of neighbour lists (%d per body) failed", need);
                    return MEL_ERR_OOM;
                }
                P.nbr_cap = need;
                retry.push_back(i);
                continue;
            }
            P.ntask = r[3];
            P.nslot = r[4];
        }
        pend = retry;
    }
    for (int i : pend) { m[i].rc = MEL_ERR_BOUNDS; m[i].msg = "neighbour lists still over capacity after 4 attempts"; }
    act.clear();
    for (int i = 0; i < n; i++) if (m[i].rc == MEL_OK) act.push_back(i);
    if (act.empty()) { launches += C.launches; return launch_status(__LINE__); }
    // 3. the candidates and the tasks' offsets in the new list; members whose candidates outgrow their
    //    list grow it and repeat this stage
    pend = act;
    while (!pend.empty()) {
        for (int i : pend) {
            mel_prox_state& P = *m[i].P;
            const size_t nt = (size_t)P.ntask + 2;
            const size_t had = P.tcand_bytes;
            if (ensure((void**)&P.tcand, &P.tcand_bytes, sizeof(int) * nt)) return MEL_ERR_OOM;
            if (P.tcand_bytes != had) P.clear = true;
            if (ensure((void**)&P.toff, &P.toff_bytes, sizeof(int) * nt)) return MEL_ERR_OOM;
            if (ensure((void**)&P.tkey, &P.tkey_bytes, sizeof(int) * nt)) return MEL_ERR_OOM;
            if (ensure((void**)&P.cand, &P.cand_bytes, sizeof(int4) * 2 * 1024)) return MEL_ERR_OOM;
            P.cand_cap = (int)std::min<size_t>(P.cand_bytes / (2 * sizeof(int4)), 0x7fffffff);
            if (ensure((void**)&P.scan_ws, &P.scan_ws_bytes, sizeof(int) * scan_scratch_ints(std::max(std::max(m[i].d->nb, P.ntask), P.cl_T)))) return MEL_ERR_OOM;
        }
        if (!make_jobs(C, m, pend, hj, T)) return MEL_ERR_CUDA;
        bool any_clear = false;
        std::vector<int> clear;
        for (int i : pend) {
            mel_prox_state& P = *m[i].P;
            any_clear = any_clear || P.clear;
            clear.push_back(P.clear ? std::max((int)(P.tcand_bytes / sizeof(int)) - 1, m[i].d->nb) + 1 : 0);
            P.clear = true;                              // until the run is through
        }
        if (any_clear && (rc = launch_jobs(C, clear_kernel, T, clear, 1))) return rc;
        if ((rc = launch_jobs(C, find_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.ntask > 0 ? j.nslot : 0; }), 1, FIND_THREADS))) return rc;
        std::vector<scan_req> sc;
        for (int i : pend) sc.push_back({ m[i].P->tcand, m[i].P->toff, m[i].P->ntask, m[i].P->scan_ws, C.S.rb + 8 * i + 5 });
        if ((rc = scan_many(C, sc))) return rc;
        if ((rc = launch_status(__LINE__))) return rc;
        if (!read_back(C)) return MEL_ERR_CUDA;
        std::vector<int> retry;
        for (int i : pend) {
            mel_prox_state& P = *m[i].P;
            P.ncont_new = C.S.rb[8 * i + 5];
            if (P.ncont_new <= P.cand_cap) continue;
            if (ensure((void**)&P.cand, &P.cand_bytes, sizeof(int4) * 2 * (size_t)P.ncont_new)) return MEL_ERR_OOM;
            retry.push_back(i);
        }
        pend = retry;
    }
    // 4. the new list, written into the spare buffer with history inherited from the current one
    for (int i : act) {
        mel_prox_state& P = *m[i].P;
        const size_t total = (size_t)P.ncont_new;
        if (ensure((void**)&P.cont_alt, &P.cont_alt_bytes, sizeof(mel_contact) * (total + 1))) return MEL_ERR_OOM;
        if (ensure((void**)&P.cont_w, &P.cont_w_bytes, sizeof(double) * (total + 1))) return MEL_ERR_OOM;
        if (ensure((void**)&P.cont_rt, &P.cont_rt_bytes, 6 * sizeof(double) * (total + 1))) return MEL_ERR_OOM;
        if (ensure((void**)&P.inc_rng, &P.inc_rng_bytes, sizeof(int2) * (total + 1))) return MEL_ERR_OOM;
        if (ensure((void**)&P.inc_task, &P.inc_task_bytes, sizeof(int) * (total + 1))) return MEL_ERR_OOM;
        if (ensure((void**)&P.bucket, &P.bucket_bytes, sizeof(int) * (total + 1))) return MEL_ERR_OOM;
        m[i].d->cont_w = P.cont_w;
        m[i].d->cont_rt = P.cont_rt;
        m[i].d->inc_rng = P.inc_rng;
        m[i].d->b_inc0 = P.b_inc0;
        m[i].d->b_cont0 = P.b_cont0;
    }
    if (!make_jobs(C, m, act, hj, T)) return MEL_ERR_CUDA;
    if ((rc = launch_jobs(C, bucket_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.ncont_new; }), 1))) return rc;
    if ((rc = launch_jobs(C, write_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.ncont_new; }), 32))) return rc;
    // 5. incoming ranges in send order, contact ranges, vgapn/vgapt carry of new elements
    {
        std::vector<scan_req> sc;
        for (int i : act) sc.push_back({ m[i].P->inc_cnt, m[i].P->b_inc0, m[i].d->nb, m[i].P->scan_ws });
        if ((rc = scan_many(C, sc))) return rc;
    }
    if ((rc = launch_jobs(C, inc_fill_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.ncont_new > 0 ? j.ntask : 0; }), 1))) return rc;
    for (int i : act) {
        mel_dev& d = *m[i].d;
        mel_prox_state& P = *m[i].P;
        std::swap(d.cont, P.cont_alt);
        std::swap(P.cont_bytes, P.cont_alt_bytes);
        d.ncont = P.ncont_new;
        P.clear = false;                                 // bucket, inc_fill and bodies leave zeros
    }
    if (!make_jobs(C, m, act, hj, T)) return MEL_ERR_CUDA;
    if ((rc = launch_jobs(C, bodies_kernel, T, items_of(hj, [](const mel_prox_job& j) { return j.d.nb; }), 32))) return rc;
    launches += C.launches;
    return launch_status(__LINE__);
}

int mel_run_proximity(mel_dev& d, mel_prox_state& P, const mel_prox_host& H, cudaStream_t s)
{
    (void)H;
    mel_prox_member m;
    m.d = &d;
    m.P = &P;
    int launches = 0;
    const int rc = mel_run_proximity_many(&m, 1, P.stage, launches, s);
    P.launches += launches;
    if (rc) return rc;
    if (m.rc) { mel_set_error("%s", m.msg.c_str()); return m.rc; }
    return MEL_OK;
}

// Index structures for a list supplied by the caller (mel_set_contacts): incoming ranges are built
// on the host from the list itself (contacts grouped by master body, in list order).
int mel_index_external(mel_dev& d, mel_prox_state& P, const mel_contact* host_list, int n, cudaStream_t s)
{
    int nb = d.nb;
    std::vector<int> cnt(nb + 1, 0);
    std::vector<int2> rng;
    std::vector<std::vector<int2>> per(nb);
    for (int i = 0; i < n; ) {
        int j = i;
        while (j < n && host_list[j].bodyS == host_list[i].bodyS && host_list[j].bodyM == host_list[i].bodyM) j++;
        per[host_list[i].bodyM].push_back(make_int2(i, j));
        i = j;
    }
    for (int b = 0; b < nb; b++) { cnt[b + 1] = cnt[b] + (int)per[b].size(); for (auto& r : per[b]) rng.push_back(r); }
    if (ensure((void**)&P.inc_rng, &P.inc_rng_bytes, sizeof(int2) * (rng.size() + 1))) return MEL_ERR_OOM;
    if (!rng.empty()) cudaMemcpyAsync(P.inc_rng, rng.data(), sizeof(int2) * rng.size(), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(P.b_inc0, cnt.data(), sizeof(int) * (nb + 1), cudaMemcpyHostToDevice, s);
    d.inc_rng = P.inc_rng;
    d.b_inc0 = P.b_inc0;
    d.b_cont0 = P.b_cont0;
    if (!stage_ready(P.stage, 1)) { mel_set_error("proximity read-back buffers could not be allocated"); return MEL_ERR_OOM; }
    mel_prox_member m;
    m.d = &d;
    m.P = &P;
    run_ctx C{ *P.stage, s, 0 };
    std::vector<mel_prox_job> hj;
    job_table T;
    if (!make_jobs(C, &m, std::vector<int>{ 0 }, hj, T)) return MEL_ERR_CUDA;
    int rc = launch_jobs(C, mel::body_range_kernel, T, std::vector<int>{ d.nb + 1 }, 1);
    P.launches += C.launches;
    if (rc) return rc;
    if (sync_failed(s, __LINE__)) return MEL_ERR_CUDA;
    C.S.used = 0;
    stage_release_retired(C.S);
    return launch_status(__LINE__);
}
