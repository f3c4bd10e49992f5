// Block ILU(0) in block multicolour order.
//
// The level-scheduled ILU(0) in mesh order needs one launch per dependency
// level in the factorisation and in each triangular solve; on a banded
// (RCM-like) numbering of an n^3 mesh that is O(n) levels of a few thousand
// rows each, so the solves are bound by launch latency, not by HBM.  Here the
// rows are grouped in patches of kMcRows (32) consecutive rows and the
// patch graph (two patches adjacent when a matrix block couples them) is
// coloured by DSATUR.  The factorisation order is: colours in increasing
// order, rows of a colour in increasing index.  Two patches of one colour are
// never coupled, so every patch of a colour is factored (or solved) by its own
// warp or CTA in one launch per colour.  This is ILU(0) of P A P^T
// for the permutation P of that order (the ordering idea is the algebraic block
// multicolour ordering of Iwashita, Nakashima and Takahashi, IPDPS 2012).
//
// Storage: `slot` lists each row's CRS slots as [lower, in factorisation
// order | diagonal | upper, in factorisation order]; `loc` is the place of
// entry u of row i (at IA[i] + u) in M: L (unit diagonal) for the lower
// entries, inv(U_ii) for the diagonal, U for the upper entries.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <memory>
#include <set>
#include <tuple>
#include <vector>

#include "ctx.cuh"
#include "kernels.cuh"
#include "ilu_mc.cuh"
#include "host_par.h"

namespace cfd {

namespace {

// Rows per patch of the ordering (five solve threads per row).
constexpr int kMcRows = 32;

template <typename T>
__device__ __forceinline__ double ld(const T *p);
template <>
__device__ __forceinline__ double ld<double>(const double *p) { return *p; }
template <>
__device__ __forceinline__ double ld<float>(const float *p) { return (double)*p; }
template <>
__device__ __forceinline__ double ld<uint16_t>(const uint16_t *p) { return load_low(p); }

template <typename T>
__device__ __forceinline__ void st(T *p, double v);
template <>
__device__ __forceinline__ void st<double>(double *p, double v) { *p = v; }
template <>
__device__ __forceinline__ void st<float>(float *p, double v) { *p = (float)v; }

// 5x5 inverse by Gauss-Jordan with partial pivoting across a warp: lane
// r*5+c (r, c < 5) holds entry (r,c) of the matrix (a) and of the inverse
// being formed (v); lanes 25-31 carry zeros.  The pivot of column k is the
// first row >= k of largest magnitude, as in the sequential elimination, and
// every entry sees the same operations in the same order.  Returns false
// (on every lane) when a pivot is zero.
__device__ __forceinline__ bool warp_inverse5(double &a, double &v, int lane) {
    const int r = lane / 5, c = lane - 5 * (lane / 5);
    const bool on = lane < 25;
    v = (on && r == c) ? 1.0 : 0.0;
    if (!on) a = 0.0;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        // column k, on every lane; pivot: its largest magnitude at or below
        // row k, lowest row on ties.  Every lane inverts its own entry
        // meanwhile: the pivot's is among them.
        const double inv_own = 1.0 / a;
        double col[5];
#pragma unroll
        for (int t = 0; t < 5; t++) col[t] = __shfl_sync(0xffffffffu, a, t * 5 + k);
        int p = k;
        double pv = col[k];
#pragma unroll
        for (int t = k + 1; t < 5; t++)
            if (fabs(col[t]) > fabs(pv)) { pv = col[t]; p = t; }
        if (!(fabs(pv) > 0.0)) ok = false;
        // rows k and p change places; row k is scaled by 1 / pivot and
        // eliminated from the others
        const double d = __shfl_sync(0xffffffffu, inv_own, p * 5 + k);
        const double ak = __shfl_sync(0xffffffffu, a, p * 5 + (on ? c : 0)) * d;
        const double vk = __shfl_sync(0xffffffffu, v, p * 5 + (on ? c : 0)) * d;
        const double a0 = __shfl_sync(0xffffffffu, a, k * 5 + (on ? c : 0));
        const double v0 = __shfl_sync(0xffffffffu, v, k * 5 + (on ? c : 0));
        double f = 0.0;
#pragma unroll
        for (int t = 0; t < 5; t++)
            if (t == r) f = col[t];
        if (r == p) { f = col[k]; a = a0; v = v0; }
        if (on) {
            a = r == k ? ak : a - f * ak;
            v = r == k ? vk : v - f * vk;
        }
    }
    return ok;
}

// Triangular solves: six warps per patch, six groups of five lanes per warp
// (lanes 30 and 31 idle), a group per row.
constexpr int kMcWarps = 6, kMcGroups = 6 * kMcWarps, kMcSolveThreads = 32 * kMcWarps;
static_assert(kMcGroups >= kMcRows, "a group per row");

// Storage of the factors in M.  A patch's lower blocks are one region, its
// inverted diagonal and upper blocks another, so that one triangular solve of
// a patch reads one contiguous run.  A region holds [diagonal blocks, by row
// | blocks inside the patch, by row | slots of off-patch blocks]: slot t of
// warp w holds the t-th off-patch block of each of the warp's six rows.
// Rows are given to groups by decreasing number of off-patch blocks, so a
// warp's six rows have nearly equal numbers and few places stay empty (8 % of
// M on the tet cubes; they hold zeros).  Element 30 k + 5 g + c of a slot is
// entry (row (k + c) mod 5, column c) of group g's block: lane c of a group
// reads column c of its block with five loads, each of 30 consecutive values
// per warp.  The other blocks are row-major.  A block's place is its first
// element / 5, with kMcSlotBit for one in a slot.  Regions start at multiples
// of 20 elements (16 bytes in FP32 and FP64).
constexpr unsigned kMcSlotBit = 0x80000000u;
constexpr int kMcSlot = 150, kMcUnit = 20;

// Element (r, c) of the block at place p.
__device__ __forceinline__ int64_t mc_element(unsigned p, int r, int c) {
    const int k = (p & kMcSlotBit) ? 30 * (r >= c ? r - c : r - c + 5) : 5 * r;
    return (int64_t)(p & ~kMcSlotBit) * 5 + k + c;
}

// One step of a row's elimination by a warp: L_ip = A_ip inv(U_pp) in block tk
// of w, then A_ij -= L_ip U_pj over the step's cnt pairs, target(t) the block
// of pair t, inv(k) / U(t, k) entry k of the factor blocks.  Lane 5 r + c owns
// entry (r, c) of every block; four pairs are in flight (no two have the same
// target).
template <typename FT, typename FI, typename FU>
__device__ __forceinline__ void mc_eliminate(double *w, int tk, int cnt, FT target, FI inv, FU U, int lane) {
    const int r = min(lane / 5, 4), c = lane - 5 * (lane / 5);
    const bool on = lane < 25;
    double *row = w + tk * 25 + 5 * r;
    double L[5], Lrc = 0.0;
#pragma unroll
    for (int k = 0; k < 5; k++) Lrc = fma(row[k], inv(5 * k + c), Lrc);
    __syncwarp();
    if (on) row[c] = Lrc;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 5; k++) L[k] = row[k];
    for (int t0 = 0; t0 < cnt; t0 += 4) {
        double *d[4], v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int t = min(t0 + j, cnt - 1);
            d[j] = w + target(t) * 25 + (on ? lane : 0);
            v[j] = *d[j];
#pragma unroll
            for (int k = 0; k < 5; k++) v[j] = fma(-L[k], U(t, 5 * k + c), v[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (on && t0 + j < cnt) *d[j] = v[j];
    }
    __syncwarp();
}

// Shared-memory bytes of one warp of k_mc_factor (factor blocks staged in
// their storage type TM), rounded up to 16.
template <typename TM>
__host__ __device__ inline size_t mc_factor_warp_bytes(int maxrow, int maxstage) {
    const size_t b = (size_t)maxrow * sizeof(int4) + (size_t)maxrow * 25 * sizeof(double) +
                     (size_t)maxstage * 25 * sizeof(TM) + (size_t)(2 * maxstage + maxrow) * sizeof(int);
    return (b + 15) & ~(size_t)15;
}

// Factorisation of the patches of one colour, one warp per patch: the warp
// factors the patch's rows in increasing order (a row's lower blocks inside
// the patch belong to earlier rows of the same warp; the others to earlier
// colours), so no CTA-wide barrier is needed.  Row i's
// blocks are staged in shared memory in FP64 (CRS slot order) together with
// every factor block the row needs from earlier rows: inv(U_pp) for each lower
// block (i,p) and U_pj for each pair (p,j) with j in row i, listed per row at
// setup.  All those loads are issued together, then the elimination runs from
// shared memory: for each lower block, in factorisation order,
// L_ip = A_ip inv(U_pp) and A_ij -= L_ip U_pj over the row's pairs of p.
// The factors are stored by patch, as the triangular solves stage them:
// loc[k] is the place of CRS block k, meta[i].w = level of row i in its patch |
// pairs of its off-patch blocks << 8.
// hdr[IA[i]+u] = (place of inv(U_pp), pairs, CRS-local slot of (i,p), 0);
// pairs are (place of U_pj, CRS-local slot of (i,j)).  Where the CTA-per-patch
// kernel can run too (by_cta), the places of blocks of p in row i's own patch
// are CRS positions in the patch instead, and hdr.w is p's level.
template <typename TA, typename TM>
__global__ void k_mc_factor(const int *__restrict__ patches, int npatch, int n, int maxrow, int maxstage, int by_cta,
                            const int *__restrict__ IA, const int *__restrict__ slot, const int4 *__restrict__ meta,
                            const int4 *__restrict__ hdr, const unsigned *__restrict__ loc,
                            const int64_t *__restrict__ pair_ptr, const int2 *__restrict__ pairs,
                            const TA *__restrict__ A, TM *__restrict__ M, int *__restrict__ err) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int nwarp = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // per-warp region (a multiple of 16 bytes): headers first, so they stay
    // 16-byte aligned, then the FP64 blocks, then the integer lists
    unsigned char *reg = smraw + (size_t)wid * mc_factor_warp_bytes<TM>(maxrow, maxstage);
    int4 *hd = reinterpret_cast<int4 *>(reg);                                     // [maxrow]
    double *w = reinterpret_cast<double *>(reg + (size_t)maxrow * sizeof(int4));  // [maxrow][25] row blocks
    TM *stg = reinterpret_cast<TM *>(w + (size_t)maxrow * 25);       // [maxstage][25] staged factor blocks
    int *pm = reinterpret_cast<int *>(stg + (size_t)maxstage * 25);  // [maxstage] CRS-local slot of each pair
    int *src = pm + maxstage;                                         // [maxstage] place of staged blocks in M
    int *sl = src + maxstage;                                         // [maxrow] CRS-local slot of list entry u
    const int pidx = blockIdx.x * nwarp + wid;
    if (pidx >= npatch) return;  // whole warp; no CTA barrier follows
    const int P = patches[pidx];
    const int p0 = P * kMcRows, nr = min(kMcRows, n - p0), base0 = IA[p0];
    const int a = lane / 5, b = lane - 5 * (lane / 5);
    {
        for (int q = 0; q < nr; q++) {
            const int i = p0 + q;
            const int4 mt = meta[i];
            const int base = IA[i], len = IA[i + 1] - base, nlo = mt.y;
            const int64_t pp = pair_ptr[i];
            const int npair = (int)(pair_ptr[i + 1] - pp), next_pairs = mt.w >> 8;
            for (int e = lane; e < nlo; e += 32) {
                const int4 h = hdr[base + e];
                hd[e] = h;
                src[e] = !by_cta || e < mt.x ? h.x : (int)loc[base0 + h.x];
            }
            for (int e = lane; e < npair; e += 32) {
                const int2 pr = pairs[pp + e];
                pm[e] = pr.y;
                src[nlo + e] = !by_cta || e < next_pairs ? pr.x : (int)loc[base0 + pr.x];
            }
            for (int e = lane; e < len; e += 32) sl[e] = slot[base + e] - base;
            // one block per lane, its 25 loads in flight together
            for (int t = lane; t < len; t += 32) {
                const TA *ab = A + (int64_t)(base + t) * 25;
#pragma unroll
                for (int k = 0; k < 25; k++) w[t * 25 + k] = ld<TA>(ab + k);
            }
            __syncwarp();
            const int nst = nlo + npair;
            // a block per step, an entry per lane, eight steps in flight
            for (int t8 = 0; t8 < nst; t8 += 8) {
                TM v[8];
#pragma unroll
                for (int k = 0; k < 8; k++)
                    v[k] = M[mc_element((unsigned)src[min(t8 + k, nst - 1)], min(a, 4), b)];
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (t8 + k < nst && lane < 25) stg[(t8 + k) * 25 + lane] = v[k];
            }
            __syncwarp();
            int t0 = 0;
            for (int u = 0; u < nlo; u++) {
                const int4 h = hd[u];
                const int tk = h.z;
                // L_ip = A_ip inv(U_pp)
                double Lab = 0.0;
                if (lane < 25) {
#pragma unroll
                    for (int c = 0; c < 5; c++) Lab = fma(w[tk * 25 + a * 5 + c], (double)stg[u * 25 + c * 5 + b], Lab);
                }
                __syncwarp();
                if (lane < 25) w[tk * 25 + lane] = Lab;
                __syncwarp();
                // A_ij -= L_ip U_pj, the pairs' 25 entries spread over the lanes
                for (int e = lane; e < h.y * 25; e += 32) {
                    const int t = e / 25, ab = e - 25 * t, ea = ab / 5, eb = ab - 5 * ea;
                    const int mj = pm[t0 + t];
                    const TM *U = stg + (size_t)(nlo + t0 + t) * 25;
                    double s = w[mj * 25 + ab];
#pragma unroll
                    for (int c = 0; c < 5; c++) s = fma(-w[tk * 25 + ea * 5 + c], (double)U[c * 5 + eb], s);
                    w[mj * 25 + ab] = s;
                }
                __syncwarp();
                t0 += h.y;
            }
            const int td = sl[nlo];  // the diagonal follows the lower entries
            {
                double av = lane < 25 ? w[td * 25 + lane] : 0.0, iv;
                const bool ok = warp_inverse5(av, iv, lane);
                if (!ok && lane == 0) atomicOr(err, ERR_NAN);
                __syncwarp();
                if (lane < 25) w[td * 25 + lane] = iv;
            }
            __syncwarp();
            // a block per step, an entry per lane, the places of eight blocks in flight
            for (int t8 = 0; t8 < len; t8 += 8) {
                unsigned to[8];
#pragma unroll
                for (int k = 0; k < 8; k++) to[k] = loc[base + min(t8 + k, len - 1)];
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (t8 + k < len && lane < 25) st<TM>(M + mc_element(to[k], a, b), w[(t8 + k) * 25 + lane]);
            }
            __syncwarp();
        }
    }
}

// Factorisation of the patches of one colour, one CTA of 16 warps per patch:
// the same operations as the warp-per-patch kernel, for meshes whose patches'
// blocks fit in shared memory in FP64 (and see mc_factor_by_cta).  The patch's
// blocks and lists are loaded once.  Blocks that couple to other patches come
// first in every row's order and depend on nothing inside the patch, so the
// warps, two rows each, eliminate them at once, staging the factor blocks of
// the other patches.  Then, level by level, the rows of a level invert their
// diagonal blocks, and every row eliminates its blocks in their columns.
// Bound by the chain of a patch's levels, some 9 inversions and eliminations
// behind each other (up to 32 on a mesh numbered along its lines), where the
// warp-per-patch kernel takes 32 rows one after the other.  A cfd_gmres call of
// one iteration (factorisation, two applies) with a CTA / a warp per patch, FP32
// factors: tets in blocked RCM order 24^3 0.77 / 3.8 ms, 64^3 3.7 / 6.2, 96^3
// 10.7 / 11.3, 112^3 16.8 / 14.4; in natural order 40^3 1.7 / 2.9, 64^3 5.6 /
// 4.0; hexahedra in blocked RCM order 64^3 2.3 / 2.5, 96^3 6.6 / 4.5, in natural
// order 40^3 1.16 / 0.86, 96^3 13.0 / 4.0.  FP64: tets 96^3 11.7 / 13.6, in
// natural order 17.9 / 13.5, hexahedra 6.8 / 5.2.  By the rule: 10.7 and 13.5 ms
// for the tets of 96^3 and 112^3 in FP32, 4.2 for the hexahedra of 96^3.
constexpr int kMcFactorWarps = 16, kMcFactorRows = kMcRows / kMcFactorWarps;
static_assert(kMcFactorRows == 2, "two rows per warp");
constexpr size_t kMcFactorBytes = 222u << 10;  // its shared memory at most
__host__ __device__ inline size_t mc_factor_cta_bytes(int maxblk, int maxpairs) {
    return ((size_t)maxblk * (25 * sizeof(double) + sizeof(int4) + 2 * sizeof(int)) + (size_t)maxpairs * sizeof(int2) + 15) &
           ~(size_t)15;
}

template <typename TA, typename TM>
__global__ void __launch_bounds__(32 * kMcFactorWarps, 1) k_mc_factor_cta(
    const int *__restrict__ patches, int n, int maxblk, int maxpairs, int stage, const int *__restrict__ IA,
    const int *__restrict__ slot, const int4 *__restrict__ meta, const int4 *__restrict__ hdr,
    const unsigned *__restrict__ loc, const int64_t *__restrict__ pair_ptr, const int2 *__restrict__ pairs,
    const TA *__restrict__ A, TM *__restrict__ M, int *__restrict__ err) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ int4 mts[kMcRows];                          // the rows' meta
    __shared__ int first[kMcRows + 1], pfirst[kMcRows + 1];  // first block / pair of each row in the patch
    int4 *hd = reinterpret_cast<int4 *>(smraw);                          // [maxblk]
    double *w = reinterpret_cast<double *>(hd + maxblk);                 // [maxblk][25], CRS slot order
    int2 *pr = reinterpret_cast<int2 *>(w + (size_t)maxblk * 25);        // [maxpairs]
    int *sl = reinterpret_cast<int *>(pr + maxpairs);                    // [maxblk] CRS position of list entry u
    unsigned *at = reinterpret_cast<unsigned *>(sl + maxblk);            // [maxblk] place in M of CRS position k
    constexpr int NT = 32 * kMcFactorWarps;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    TM *stg = reinterpret_cast<TM *>(smraw + mc_factor_cta_bytes(maxblk, maxpairs)) + (size_t)wid * stage * 25;
    const int p0 = patches[blockIdx.x] * kMcRows, nr = min(kMcRows, n - p0);
    const int base = IA[p0], nblk = IA[p0 + nr] - base;
    const int64_t pbase = pair_ptr[p0];
    const int npair = (int)(pair_ptr[p0 + nr] - pbase);
    const TA *Ap = A + (int64_t)base * 25;
    for (int e0 = tid; e0 < nblk * 25; e0 += 8 * NT) {
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = ld<TA>(Ap + min(e0 + k * NT, nblk * 25 - 1));
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (e0 + k * NT < nblk * 25) w[e0 + k * NT] = v[k];
    }
    for (int e = tid; e <= nr; e += NT) {
        first[e] = IA[p0 + e] - base;
        pfirst[e] = (int)(pair_ptr[p0 + e] - pbase);
        if (e < nr) mts[e] = meta[p0 + e];
    }
    for (int e = tid; e < nblk; e += NT) {
        hd[e] = hdr[base + e];
        sl[e] = slot[base + e] - base;
        at[e] = loc[base + e];
    }
    for (int e = tid; e < npair; e += NT) pr[e] = pairs[pbase + e];
    __syncthreads();
    const int a = min(lane / 5, 4), b = lane - 5 * (lane / 5);
    // rows to warps in order of their levels, so that a level's rows have
    // different warps
    const int mylev = lane < nr ? mts[lane].w & 255 : -1;
    int last = 0, rank = 0, before = 0;
    for (int l = 0; before < nr && l < kMcRows; l++) {
        const unsigned m = __ballot_sync(0xffffffffu, mylev == l);
        if (mylev == l) rank = before + __popc(m & ((1u << lane) - 1u));
        before += __popc(m);
        last = l;
    }
    int rows[kMcFactorRows];  // the warp's rows, nr: none
#pragma unroll
    for (int k = 0; k < kMcFactorRows; k++) {
        const unsigned m = __ballot_sync(0xffffffffu, lane < nr && rank == wid + k * kMcFactorWarps);
        rows[k] = m ? __ffs(m) - 1 : nr;
    }
    // blocks that couple to other patches: as many at a time as the staging holds
#pragma unroll 1
    for (int k = 0; k < kMcFactorRows; k++) {
        const int q = k == 0 ? rows[0] : rows[1];
        if (q >= nr) continue;
        const int row0 = first[q], next = mts[q].x;
        const int2 *q0 = pr + pfirst[q];
        for (int u0 = 0; u0 < next;) {
            int u1 = u0, np = 0;
            for (; u1 < next; u1++) {
                const int y = hd[row0 + u1].y;
                if (u1 > u0 && u1 + 1 - u0 + np + y > stage) break;
                np += y;
            }
            const int m = u1 - u0 + np;
            // a block per step, an entry per lane, eight steps in flight
            for (int t8 = 0; t8 < m; t8 += 8) {
                TM v[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int t = min(t8 + k, m - 1);
                    const unsigned p = (unsigned)(t < u1 - u0 ? hd[row0 + u0 + t].x : q0[t - (u1 - u0)].x);
                    v[k] = M[mc_element(p, a, b)];
                }
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (t8 + k < m && lane < 25) stg[(t8 + k) * 25 + lane] = v[k];
            }
            __syncwarp();
            const TM *Up = stg + (u1 - u0) * 25;
            for (int u = u0; u < u1; u++) {
                const int4 h = hd[row0 + u];
                const TM *iv = stg + (u - u0) * 25;
                mc_eliminate(w, row0 + h.z, h.y, [&](int t) { return row0 + q0[t].y; },
                             [&](int k) { return (double)iv[k]; }, [&](int t, int k) { return (double)Up[t * 25 + k]; },
                             lane);
                q0 += h.y;
                Up += h.y * 25;
            }
            u0 = u1;
        }
    }
    // the headers of the warp's rows' intra-patch blocks, one per lane, with
    // the place of their pairs (a row has at most 31 of them)
    int4 mine[kMcFactorRows];
    int pairs_at[kMcFactorRows], lev[kMcFactorRows], nin[kMcFactorRows];
#pragma unroll
    for (int k = 0; k < kMcFactorRows; k++) {
        const int q = rows[k];
        lev[k] = -1;
        nin[k] = 0;
        mine[k] = make_int4(0, 0, 0, -1);
        if (q < nr) {
            lev[k] = mts[q].w & 255;
            nin[k] = mts[q].y - mts[q].x;
            if (lane < nin[k]) mine[k] = hd[first[q] + mts[q].x + lane];
        }
        int sum = mine[k].y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        pairs_at[k] = sum - mine[k].y + (q < nr ? pfirst[q] + (mts[q].w >> 8) : 0);
    }
    for (int l = 0; l <= last; l++) {
#pragma unroll
        for (int k = 0; k < kMcFactorRows; k++) {
            if (lev[k] != l) continue;
            const int q = rows[k];
            double *dg = w + sl[first[q] + mts[q].y] * 25;  // the diagonal follows the lower entries
            double av = lane < 25 ? dg[lane] : 0.0, iv;
            const bool ok = warp_inverse5(av, iv, lane);
            if (!ok && lane == 0) atomicOr(err, ERR_NAN);
            __syncwarp();
            if (lane < 25) dg[lane] = iv;
            __syncwarp();
            // the other rows see the factors as stored
            if (sizeof(TM) < sizeof(double)) {
                const int end = first[q + 1] * 25;
                for (int e0 = first[q] * 25 + lane; e0 < end; e0 += 256) {
                    double v[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) v[j] = (double)(TM)w[min(e0 + 32 * j, end - 1)];
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        if (e0 + 32 * j < end) w[e0 + 32 * j] = v[j];
                }
            }
        }
        if (l == last) break;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kMcFactorRows; k++) {
            unsigned todo = __ballot_sync(0xffffffffu, lane < nin[k] && mine[k].w == l);
            const int row0 = first[rows[k]];
            for (; todo; todo &= todo - 1) {
                const int s = __ffs(todo) - 1;
                const int x = __shfl_sync(0xffffffffu, mine[k].x, s), cnt = __shfl_sync(0xffffffffu, mine[k].y, s);
                const int z = __shfl_sync(0xffffffffu, mine[k].z, s), pa = __shfl_sync(0xffffffffu, pairs_at[k], s);
                const int2 *q = pr + pa;
                const double *iv = w + x * 25;
                mc_eliminate(w, row0 + z, cnt, [&](int t) { return row0 + q[t].y; }, [&](int j) { return iv[j]; },
                             [&](int t, int j) { return w[q[t].x * 25 + j]; }, lane);
            }
        }
    }
    __syncthreads();
    // a block per warp and step, an entry per lane
#pragma unroll 4
    for (int k = wid; k < nblk; k += kMcFactorWarps)
        if (lane < 25) st<TM>(M + mc_element(at[k], a, b), w[k * 25 + lane]);
}

// Programmatic dependent launch (sm_90+): the solve of one colour lets the
// next colour's launch begin as soon as all of its own CTAs are resident
// (launch_dependents), and that launch stages its constant factor blocks
// before waiting (wait) for the vectors the earlier launches write.  Every
// CTA of the earlier grid is resident before a dependent CTA can start, so
// the earlier grid always completes.  Both are no-ops in a plain launch.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// 16-byte asynchronous copy global -> shared (LDGSTS), and the wait for all of
// the thread's copies.
__device__ __forceinline__ void copy16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
// Starts fetching [gmem, gmem + bytes) from DRAM into L2 (bytes > 0, multiples of 16).
__device__ __forceinline__ void prefetch_l2(const void *gmem, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A group's row in its patch (255 none) and its off-patch blocks.
struct McGroup {
    unsigned short row, next;
};
static_assert(sizeof(McGroup) == 4, "packed in the patch lists");
// Byte offsets of a patch's lists: int4 {off-patch columns, steps, rows, first
// row}, int4 {first element of the slots in the region, slots, 0, 0}, per
// warp {first slot, slots}, the groups; then the distinct off-patch columns,
// the steps (six operations each, see mc_op) and, 16 bits per slot and group,
// its column's index among those columns (their number for an empty place).
constexpr int kMcWarpAt = 32, kMcGroupAt = kMcWarpAt + 4 * kMcWarps, kMcColAt = kMcGroupAt + 4 * kMcGroups;

// An operation of a step, on values v_r of the patch's rows: v_row -= block *
// v_col for an intra-patch block or, diag, v_row = block * v_row with the
// inverted diagonal block.  block counts from the region's start (diagonal
// blocks first).  row = col = 32 for an idle group.
__host__ __device__ inline unsigned mc_op(int block, int col, int row, bool diag) {
    return (unsigned)block | ((unsigned)col << 10) | ((unsigned)row << 16) | (diag ? 0x80000000u : 0u);
}

// Largest part of a region staged in shared memory, in units of kMcUnit
// elements (the slots past it are read from global memory).  A colour whose
// patches are all resident at once stages whole regions, for the shortest
// patch (48^3, 340 patches per colour, FP64: 181 us per apply, 228 with 176
// units); a larger one stages less, for more CTAs per SM (96^3, 2600 patches
// per colour: FP64 795 us, 1005 with 640 units; FP32 521 and 568).
constexpr int kMcStageUnits = 640;
template <typename TM>
struct McStageMany {
    static constexpr int units = sizeof(TM) == 8 ? 200 : 400;
};
// Largest lists and gathered values beside it; colours that need more (rows
// with hundreds of blocks) run unstaged.
constexpr size_t kMcListBytes = 64u << 10;
// Patches ahead of a CTA's own whose data it starts fetching into L2, about
// one wave of the larger colours (96^3, FP32: 603 -> 571 us per apply).
constexpr int kMcAheadPatches = 592;

// Sum over the five lanes of a group: lane c ends with entry c of the product
// whose part for entry (k + c) mod 5 lane c holds in p[k].
__device__ __forceinline__ double group_sum(const double p[5], int g, int c) {
    double v[5];
#pragma unroll
    for (int k = 0; k < 5; k++) v[k] = __shfl_sync(0xffffffffu, p[k], g < 6 ? 5 * g + (c >= k ? c - k : c - k + 5) : 31);
    return ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
}

// One triangular solve over the patches of one colour, one CTA per patch:
// forward y = L^-1 r (OUT = y) or, BWD, backward z = U^-1 y (R = y, OUT = z).
// Off-patch blocks couple to colours that earlier launches finished; the blocks
// inside the patch follow its dependency levels.
//  1. Everything constant is copied to shared memory while the previous
//     colour still runs: the patch's lists and its region of M.
//  2. After the dependency wait, one round trip fetches the values of the
//     patch's distinct off-patch columns (59 on average for 140 blocks on the
//     tet cubes) into shared memory.
//  3. Each row subtracts its off-patch blocks.  Lane c multiplies column c, so
//     a block costs a lane one value and five independent multiply-adds (one
//     output per lane would load five values and chain the five
//     multiply-adds, which bound the solve at 75-130 cycles per block).
//  4. One warp works off the blocks inside the patch: six operations per step,
//     on different rows and on values that earlier steps finished (scheduled
//     at setup; about 15 steps forward, 22 backward).  The next step's blocks
//     are already in registers, so that a step waits for one shared-memory read
//     and five multiply-adds (some 140 cycles), never for a CTA barrier or for
//     global memory.
// What bounds it: latency.  A patch takes one global round trip for its
// off-patch values and the chain of step 4, about 6,000 cycles, and three to
// five patches share an SM.  One apply (all colours, both solves) on the tet
// cubes, FP32 / FP64 factors: 24^3 68 / 73 us, 48^3 106 / 156 us, 96^3 521 /
// 795 us (2.6 / 3.1 TB/s).  The row-per-five-threads form it replaces, which
// walked the levels behind CTA barriers and read off-patch columns in chains
// of two round trips: 173 / 202, 285 / 353 and 896 / 1178 us.
// Slower here: one warp per patch's level walk with a row's blocks chained
// (96^3 1130 us, FP32); all six warps walking the levels (768 us); persistent
// CTAs with three buffers and a separate solving warp (813 us; fewer patches
// per SM).
template <typename TM, bool BWD, bool STAGED>
__global__ void __launch_bounds__(kMcSolveThreads, 5) k_mc_solve(const int4 *__restrict__ desc,
                                                              const uint4 *__restrict__ lists,
                                                              const TM *__restrict__ M, const double *__restrict__ R,
                                                              double *OUT, int list16, int units) {
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ double own[(kMcRows + 1) * 5];  // values of the patch's rows, and of idle groups
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane / 5, c = lane - 5 * g;
    // {first 16-byte word of the lists, words, first unit of the region, units}
    const int4 d = desc[blockIdx.x];
    // the next colour's launch may start staging its own patches now
    pdl_trigger();
    const TM *G = M + (int64_t)d.z * kMcUnit;
    const unsigned char *L = STAGED ? sm : reinterpret_cast<const unsigned char *>(lists + d.x);
    TM *S = reinterpret_cast<TM *>(sm + (size_t)list16 * 16);
    double *xs = reinterpret_cast<double *>(S + (size_t)units * kMcUnit);  // off-patch values
    const int staged = STAGED ? min(d.w, units) : 0;
    if (STAGED) {
        uint4 *sl = reinterpret_cast<uint4 *>(sm);
        for (int k = tid; k < d.y; k += kMcSolveThreads) copy16(sl + k, lists + d.x + k);
        const int words = staged * (kMcUnit * (int)sizeof(TM) / 16);
        for (int k = tid; k < words; k += kMcSolveThreads)
            copy16(reinterpret_cast<uint4 *>(S) + k, reinterpret_cast<const uint4 *>(G) + k);
        // a patch that a later wave of this grid takes
        if (tid == 0 && blockIdx.x + kMcAheadPatches < gridDim.x) {
            const int4 f = desc[blockIdx.x + kMcAheadPatches];
            // a patch without lower blocks has an empty region, which may begin at the end of M
            if (f.w > 0) prefetch_l2(M + (int64_t)f.z * kMcUnit, (unsigned)(f.w * kMcUnit * sizeof(TM)));
            prefetch_l2(lists + f.x, (unsigned)f.y * 16u);
        }
        copy_wait();
        __syncthreads();
    }
    const int4 h = reinterpret_cast<const int4 *>(L)[0], h1 = reinterpret_cast<const int4 *>(L)[1];
    const ushort2 ws = reinterpret_cast<const ushort2 *>(L + kMcWarpAt)[w];
    const int *cols = reinterpret_cast<const int *>(L + kMcColAt);
    const unsigned *ops = reinterpret_cast<const unsigned *>(cols + h.x);
    const unsigned short *sidx = reinterpret_cast<const unsigned short *>(ops + 6 * h.y);
    McGroup gr = {255, 0};
    if (lane < 30) gr = reinterpret_cast<const McGroup *>(L + kMcGroupAt)[6 * w + g];
    const bool act = gr.row != 255;
    const int64_t at = ((int64_t)h.w + gr.row) * 5 + c;  // the row's entry c in R
    if (tid < 5) own[kMcRows * 5 + tid] = 0.0;
    double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    // r is complete before the first forward launch starts
    if (!BWD && act) acc[0] = R[at];
    // this thread's values of the off-patch columns: the first kGather places
    // are read before the wait, so that their loads go out together after it
    constexpr int kGather = 4;
    int64_t from[kGather];
#pragma unroll
    for (int u = 0; u < kGather; u++) {
        const int k = tid + u * kMcSolveThreads, j = k / 5;
        from[u] = STAGED && k < 5 * h.x ? (int64_t)cols[j] * 5 + (k - 5 * j) : -1;
    }
    pdl_wait();  // the earlier launches' values are complete from here on
    if (BWD && act) acc[0] = __ldcg(R + at);
    if (STAGED) {
        double v[kGather];
#pragma unroll
        for (int u = 0; u < kGather; u++) v[u] = from[u] >= 0 ? __ldcg(OUT + from[u]) : 0.0;
#pragma unroll
        for (int u = 0; u < kGather; u++)
            if (tid + u * kMcSolveThreads < 5 * (h.x + 1)) xs[tid + u * kMcSolveThreads] = v[u];
        for (int k = tid + kGather * kMcSolveThreads; k < 5 * (h.x + 1); k += kMcSolveThreads) {
            const int j = k / 5;
            xs[k] = j < h.x ? __ldcg(OUT + (int64_t)cols[j] * 5 + (k - 5 * j)) : 0.0;
        }
        __syncthreads();
    }
    const TM *in = STAGED ? S : G;  // the diagonal and intra-patch blocks are always staged
    {
        // slots whose elements are all staged, then the others
        const int ns = STAGED ? max(0, staged * kMcUnit - h1.x) / kMcSlot : 0;
        const int first = ws.x, n = ws.y;
        const int m = min(n, max(0, ns - first));
        int t = 0;
        // empty places hold zeros and the index of a zero after the gathered
        // values, so that the loops take no branch per row
        const unsigned short *si = sidx + 6 * first + min(g, 5);
        const int sl = min(lane, 29);
        if (STAGED) {
            const TM *a = S + h1.x + (size_t)first * kMcSlot + sl;
#pragma unroll 4
            for (; t < m; t++) {
                const double x = xs[si[6 * t] * 5 + c];
#pragma unroll
                for (int k = 0; k < 5; k++) acc[k] = fma(-(double)a[t * kMcSlot + 30 * k], x, acc[k]);
            }
        }
        const TM *a = G + h1.x + (size_t)first * kMcSlot + sl;
#pragma unroll 4
        for (; t < n; t++) {
            const int j = si[6 * t];
            const double x = STAGED ? xs[j * 5 + c] : j < h.x ? __ldcg(OUT + (int64_t)cols[j] * 5 + c) : 0.0;
#pragma unroll
            for (int k = 0; k < 5; k++) acc[k] = fma(-(double)a[t * kMcSlot + 30 * k], x, acc[k]);
        }
    }
    const double s = group_sum(acc, g, c);  // entry c of the row
    if (act) own[gr.row * 5 + c] = s;
    __syncthreads();
    if (w == 0) {
        const int gg = min(g, 5);
        const unsigned *op = ops + gg;
        const TM *ib = in + 5 * c;
        const int n = h.y;
        // this step's block and the next step's operation wait in registers
        unsigned e0 = n > 0 ? op[0] : 0u, e1 = n > 1 ? op[6] : e0;
        TM a0[5];
        if (n > 0) {
#pragma unroll
            for (int k = 0; k < 5; k++) a0[k] = ib[(e0 & 1023u) * 25 + k];
        }
        for (int t = 0; t < n; t++) {
            const double *x = own + 5 * ((e0 >> 10) & 63u);
            double *y = own + 5 * ((e0 >> 16) & 63u) + c;
            double xv[5];
#pragma unroll
            for (int k = 0; k < 5; k++) xv[k] = x[k];
            const double yv = *y;
            TM a1[5];
#pragma unroll
            for (int k = 0; k < 5; k++) a1[k] = ib[(e1 & 1023u) * 25 + k];
            const unsigned e2 = op[6 * min(t + 2, n - 1)];
            double p = (double)a0[0] * xv[0];
#pragma unroll
            for (int k = 1; k < 5; k++) p = fma((double)a0[k], xv[k], p);
            __syncwarp();
            if (lane < 30) *y = BWD && (e0 >> 31) ? p : yv - p;
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 5; k++) a0[k] = a1[k];
            e0 = e1;
            e1 = e2;
        }
    }
    __syncthreads();
    if (tid < 5 * h.z) OUT[(int64_t)h.w * 5 + tid] = own[tid];
}

}  // namespace

namespace {

// The steps of a patch's solve (see mc_op): up to six operations each, on
// different rows, an operation after those it depends on: v_row -= L v_col
// after column col is finished; in a backward solve the diagonal operation of
// a row after all its blocks.  Greedy, rows with the longest chain of
// operations behind them first.
struct McSchedule {
    struct Op {
        int block, row, col;  // col = row: the diagonal
    };
    int nr = 0;
    bool bwd = false;
    std::vector<Op> todo, byheight;
    int left[kMcRows], height[kMcRows];
    void reset(int rows, bool backward) {
        nr = rows;
        bwd = backward;
        todo.clear();
        for (int q = 0; q < nr; q++) left[q] = 0;
    }
    // rows in increasing order
    void block(int b, int row, int col) {
        todo.push_back({b, row, col});
        left[row]++;
    }
    void run(std::vector<unsigned> &out) {
        out.clear();
        // height of a row: the longest chain of rows from its value on (at most
        // nr).  Forward, a row's columns precede it; backward, they follow it
        for (int q = 0; q < nr; q++) height[q] = 1;
        const int m = (int)todo.size();
        for (int t = 0; t < m; t++) {
            const Op &o = todo[bwd ? t : m - 1 - t];  // rows solved last first
            height[o.col] = std::max(height[o.col], height[o.row] + 1);
        }
        if (bwd)
            for (int q = 0; q < nr; q++) todo.push_back({q, q, q});
        // highest first, otherwise as listed
        int at[kMcRows + 2] = {};
        for (const Op &o : todo) at[kMcRows - height[o.row] + 1]++;
        for (int k = 0; k <= kMcRows; k++) at[k + 1] += at[k];
        byheight.resize(todo.size());
        for (const Op &o : todo) byheight[at[kMcRows - height[o.row]]++] = o;
        unsigned solved = 0;  // rows whose values are final
        for (int q = 0; q < nr; q++)
            if (!bwd && left[q] == 0) solved |= 1u << q;
        while (!byheight.empty()) {
            unsigned used = 0;
            size_t kept = 0;
            int k = 0;
            Op taken[6];
            for (size_t t = 0; t < byheight.size(); t++) {
                const Op o = byheight[t];
                const bool ready = o.row == o.col ? left[o.row] == 0 : (solved >> o.col) & 1u;
                if (k < 6 && ready && !((used >> o.row) & 1u)) {
                    used |= 1u << o.row;
                    taken[k++] = o;
                } else {
                    byheight[kept++] = o;
                }
            }
            byheight.resize(kept);
            for (int g = 0; g < 6; g++) {
                if (g >= k) {
                    out.push_back(mc_op(0, kMcRows, kMcRows, false));
                    continue;
                }
                const int q = taken[g].row;
                const bool diag = taken[g].col == q;
                out.push_back(mc_op(taken[g].block, taken[g].col, q, diag));
                if (!diag) left[q]--;
                if (bwd ? diag : left[q] == 0) solved |= 1u << q;
            }
        }
    }
};

}  // namespace

// Ordering, slot lists, the solves' plans and the factorisation's update lists
// (host, once per mesh).
int mc_build(cfd_ctx *c) {
    Abmc &mc = c->mc;
    if (mc.built) return CFD_OK;
    const int n = c->nnode;
    const std::vector<int> &IA = c->h_IA, &JA = c->h_JA, &IAU = c->h_IAU;
    const int np = (n + kMcRows - 1) / kMcRows;
    // ranges of patches or rows, on as many threads as their rows are worth (a
    // row's lists cost some microseconds, an item of a plain loop nanoseconds)
    constexpr int kRowWeight = 16;
    auto parallel_patches = [&](auto fn) {
        const int64_t items = kRowWeight * (int64_t)n;
        parallel_ranges(items, [&](int t, int64_t i0, int64_t i1) { fn(t, i0 * np / items, i1 * np / items); });
    };
    auto parallel_rows = [&](auto fn) {
        const int64_t items = kRowWeight * (int64_t)n;
        parallel_ranges(items, [&](int, int64_t i0, int64_t i1) { fn((int)(i0 / kRowWeight), (int)(i1 / kRowWeight)); });
    };
    // DSATUR colouring of the patch graph (Brelaz 1979): repeatedly colour the
    // uncoloured patch with the most distinct colours among its neighbours
    // (ties: most neighbours, then lowest index) with the lowest colour free
    // there.  On the tet cubes and channels it needs 10-11 colours where the
    // greedy colouring in patch order needs 13-14, i.e. fewer launches per
    // factorisation and per triangular solve.
    std::vector<std::vector<int>> adj(np);
    parallel_patches([&](int, int64_t p0, int64_t p1) {
        for (int P = (int)p0; P < (int)p1; P++) {
            const int r0 = P * kMcRows, r1 = std::min(n, r0 + kMcRows);
            for (int i = r0; i < r1; i++)
                for (int k = IA[i]; k < IA[i + 1]; k++) {
                    const int Q = JA[k] / kMcRows;
                    if (Q != P) adj[P].push_back(Q);
                }
            std::sort(adj[P].begin(), adj[P].end());
            adj[P].erase(std::unique(adj[P].begin(), adj[P].end()), adj[P].end());
        }
    });
    std::vector<int> color(np, -1);
    std::vector<uint64_t> seen(np, 0);  // colours among a patch's neighbours
    std::set<std::tuple<int, int, int>> open;  // (-saturation, -degree, patch)
    for (int P = 0; P < np; P++) open.insert({0, -(int)adj[P].size(), P});
    int ncolor = 0;
    while (!open.empty()) {
        const int P = std::get<2>(*open.begin());
        open.erase(open.begin());
        const uint64_t m = seen[P];
        int col = 0;
        while (col < 64 && ((m >> col) & 1u)) col++;
        if (col >= 64) {
            set_error("ILU(0) multicolour: the patch graph needs more than 64 colours");
            return CFD_ERR_RANGE;
        }
        color[P] = col;
        ncolor = std::max(ncolor, col + 1);
        for (int Q : adj[P]) {
            if (color[Q] >= 0 || ((seen[Q] >> col) & 1u)) continue;
            const int sat = __builtin_popcountll(seen[Q]);
            open.erase({-sat, -(int)adj[Q].size(), Q});
            seen[Q] |= 1ull << col;
            open.insert({-(sat + 1), -(int)adj[Q].size(), Q});
        }
    }
    mc.ncolor = ncolor;
    mc.h_pcolor = color;
    mc.cptr.assign(ncolor + 1, 0);
    for (int P = 0; P < np; P++) mc.cptr[color[P] + 1]++;
    for (int k = 0; k < ncolor; k++) mc.cptr[k + 1] += mc.cptr[k];
    std::vector<int> patches(np), fill(mc.cptr.begin(), mc.cptr.end() - 1);
    for (int P = 0; P < np; P++) patches[fill[color[P]]++] = P;
    // position key of a row in the factorisation order
    auto key = [&](int j) { return (int64_t)color[j / kMcRows] * n + j; };
    std::vector<int> slot(c->nnzb), scol(c->nnzb);
    std::vector<int4> meta(n);
    std::vector<int> maxrow_in(range_count(n), 0);
    parallel_ranges(n, [&](int rt, int64_t i0, int64_t i1) {
    std::vector<std::pair<int64_t, int>> lo, up;
    int &maxrow = maxrow_in[rt];
    for (int i = (int)i0; i < (int)i1; i++) {
        lo.clear();
        up.clear();
        const int64_t ki = key(i);
        const int Pi = i / kMcRows;
        int next = 0, nint = 0;
        for (int k = IA[i]; k < IA[i + 1]; k++) {
            if (k == IAU[i]) continue;
            const int64_t kj = key(JA[k]);
            if (kj < ki) lo.push_back({kj, k});
            else up.push_back({kj, k});
        }
        std::sort(lo.begin(), lo.end());
        std::sort(up.begin(), up.end());
        int w = IA[i];
        for (auto &e : lo) {
            slot[w++] = e.second;
            if (JA[e.second] / kMcRows != Pi) next++;
        }
        slot[w++] = IAU[i];
        for (auto &e : up) {
            slot[w++] = e.second;
            if (JA[e.second] / kMcRows == Pi) nint++;
        }
        // external lower blocks come first in key order (smaller colours),
        // intra-patch upper blocks first among the upper ones
        meta[i] = make_int4(next, (int)lo.size(), nint, 0);
        maxrow = std::max(maxrow, IA[i + 1] - IA[i]);
    }
    });
    const int maxrow = *std::max_element(maxrow_in.begin(), maxrow_in.end());
    parallel_ranges(c->nnzb, [&](int, int64_t u0, int64_t u1) {
        for (int64_t u = u0; u < u1; u++) scol[u] = JA[slot[u]];
    });
    // A row's level in its patch: the longest chain of intra-patch lower blocks
    // before it (meta.w, for the factorisation)
    parallel_patches([&](int, int64_t q0, int64_t q1) {
        for (int i = (int)q0 * kMcRows; i < std::min<int64_t>(n, q1 * kMcRows); i++) {
            int l = 0;
            for (int u = IA[i] + meta[i].x; u < IA[i] + meta[i].y; u++) l = std::max(l, meta[scol[u]].w + 1);
            meta[i].w = l;
        }
    });
    int64_t levels = 0;
    for (int P = 0; P < np; P++) {
        int l = 0;
        for (int i = P * kMcRows; i < std::min(n, (P + 1) * kMcRows); i++) l = std::max(l, meta[i].w);
        levels += l + 1;
    }
    mc.levels = (double)levels / np;
    int maxblk = 0;
    for (int P = 0; P < np; P++) maxblk = std::max(maxblk, IA[std::min(n, (P + 1) * kMcRows)] - IA[P * kMcRows]);
    // The solves' plan of each patch and direction (0 forward, 1 backward):
    // rows to groups, the region's size, and the lists (layout at kMcWarpAt);
    // then the regions' places in M, in launch order, and every block's place.
    std::vector<int4> desc[2];
    std::vector<std::vector<unsigned char>> lists[2];
    std::vector<unsigned> loc(c->nnzb);  // first the place in the region
    std::vector<int> ucount[2];
    for (int dir = 0; dir < 2; dir++) {
        desc[dir].assign(np, make_int4(0, 0, 0, 0));
        lists[dir].resize(np);
        ucount[dir].assign(np, 0);
    }
    std::atomic<bool> too_long{false};
    parallel_patches([&](int, int64_t q0, int64_t q1) {
        std::vector<int> cols, index_of(n, -1);  // column -> its index among the patch's, -1 outside the loop below
        int order[kMcRows];
        std::vector<unsigned short> sidx;
        std::vector<unsigned> ops;
        McSchedule plan;
        for (int pos = (int)q0; pos < (int)q1; pos++)
            for (int dir = 0; dir < 2; dir++) {
                const int r0 = patches[pos] * kMcRows, r1 = std::min(n, r0 + kMcRows), nr = r1 - r0;
                // list entries of row i: intra-patch and off-patch blocks of this solve
                auto in_at = [&](int i) { return dir ? IA[i] + meta[i].y + 1 : IA[i] + meta[i].x; };
                auto in_n = [&](int i) { return dir ? meta[i].z : meta[i].y - meta[i].x; };
                auto ext_at = [&](int i) { return dir ? IA[i] + meta[i].y + 1 + meta[i].z : IA[i]; };
                auto ext_n = [&](int i) { return dir ? IA[i + 1] - ext_at(i) : meta[i].x; };
                cols.clear();
                int nin = 0;
                for (int i = r0; i < r1; i++) {
                    for (int t = 0; t < ext_n(i); t++) {
                        const int j = scol[ext_at(i) + t];
                        if (index_of[j] >= 0) continue;
                        index_of[j] = 0;
                        cols.push_back(j);
                    }
                    nin += in_n(i);
                }
                std::sort(cols.begin(), cols.end());
                for (size_t k = 0; k < cols.size(); k++) index_of[cols[k]] = (int)k;
                // rows by decreasing number of off-patch blocks (insertion sort)
                for (int q = 0; q < nr; q++) {
                    int k = q;
                    for (; k > 0 && ext_n(r0 + order[k - 1]) < ext_n(r0 + q); k--) order[k] = order[k - 1];
                    order[k] = q;
                }
                const int diag = dir ? nr : 0;
                int slots = 0;
                ushort2 ws[kMcWarps];
                for (int w = 0; w < kMcWarps; w++) {
                    const int t = 6 * w < nr ? ext_n(r0 + order[6 * w]) : 0;
                    ws[w] = make_ushort2((unsigned short)slots, (unsigned short)t);
                    slots += t;
                }
                const int64_t size = (int64_t)(diag + nin) * 25 + (int64_t)slots * kMcSlot;
                if (slots > 65535 || cols.size() > 65534) {
                    too_long = true;
                    return;
                }
                McGroup gr[kMcGroups];
                sidx.assign((size_t)6 * slots, (unsigned short)cols.size());
                plan.reset(nr, dir == 1);
                int at = 0;
                for (int k = 0; k < kMcGroups; k++) gr[k] = {255, 0};
                for (int k = 0; k < nr; k++) {
                    const int q = order[k], i = r0 + q;
                    gr[k] = {(unsigned short)q, (unsigned short)ext_n(i)};
                    for (int t = 0; t < ext_n(i); t++) {
                        const int u = ext_at(i) + t, at_slot = ws[k / 6].x + t;
                        sidx[6 * at_slot + k % 6] = (unsigned short)index_of[scol[u]];
                        loc[u] = (unsigned)(5 * (diag + nin) + (kMcSlot / 5) * at_slot + k % 6) | kMcSlotBit;
                    }
                }
                for (int i = r0; i < r1; i++) {
                    if (dir) loc[IA[i] + meta[i].y] = (unsigned)(5 * (i - r0));
                    for (int t = 0; t < in_n(i); t++) {
                        const int u = in_at(i) + t;
                        loc[u] = (unsigned)(5 * (diag + at));
                        plan.block(diag + at, i - r0, scol[u] - r0);
                        at++;
                    }
                }
                plan.run(ops);
                for (int j : cols) index_of[j] = -1;
                const size_t nu = cols.size(), bytes = kMcColAt + 4 * nu + 4 * ops.size() + 12 * (size_t)slots;
                std::vector<unsigned char> &out = lists[dir][pos];
                out.assign((bytes + 15) / 16 * 16, 0);
                int4 *hd = reinterpret_cast<int4 *>(out.data());
                hd[0] = make_int4((int)nu, (int)(ops.size() / 6), nr, r0);
                hd[1] = make_int4((diag + nin) * 25, slots, 0, 0);
                std::memcpy(out.data() + kMcWarpAt, ws, sizeof ws);
                std::memcpy(out.data() + kMcGroupAt, gr, sizeof gr);
                unsigned char *o = out.data() + kMcColAt;
                auto put = [&](const void *p, size_t b) {
                    if (b) std::memcpy(o, p, b);
                    o += b;
                };
                put(cols.data(), 4 * nu);
                put(ops.data(), 4 * ops.size());
                put(sidx.data(), 2 * sidx.size());
                desc[dir][pos].w = (int)((size + kMcUnit - 1) / kMcUnit);
                ucount[dir][pos] = (int)nu;
            }
    });
    int64_t units = 0;
    for (int pos = 0; pos < np; pos++)
        for (int dir = 0; dir < 2; dir++) {
            desc[dir][pos].z = (int)units;
            units += desc[dir][pos].w;
        }
    if (too_long || units * (kMcUnit / 5) >= (int64_t)kMcSlotBit) {
        set_error("ILU(0) multicolour: too many blocks");
        return CFD_ERR_RANGE;
    }
    mc.nelem = units * kMcUnit;
    parallel_patches([&](int, int64_t q0, int64_t q1) {
        for (int pos = (int)q0; pos < (int)q1; pos++) {
            const int r0 = patches[pos] * kMcRows, r1 = std::min(n, r0 + kMcRows);
            for (int i = r0; i < r1; i++)
                for (int u = IA[i]; u < IA[i + 1]; u++)
                    loc[u] += (unsigned)desc[u < IA[i] + meta[i].y ? 0 : 1][pos].z * (kMcUnit / 5);
        }
    });
    for (int dir = 0; dir < 2; dir++) {
        mc.shape[dir].assign(ncolor, make_int4(0, 0, 0, 0));
        size_t words = 0;
        for (int pos = 0; pos < np; pos++) {
            const int w16 = (int)(lists[dir][pos].size() / 16);
            desc[dir][pos].x = (int)words;
            desc[dir][pos].y = w16;
            words += w16;
            int4 &sh = mc.shape[dir][color[patches[pos]]];
            sh.x = std::max(sh.x, w16);
            sh.y = std::max(sh.y, desc[dir][pos].w);
            sh.z = std::max(sh.z, ucount[dir][pos]);
            sh.w = std::max(sh.w, reinterpret_cast<const int4 *>(lists[dir][pos].data())[1].x);
        }
        if (words > (size_t)INT32_MAX) {
            set_error("ILU(0) multicolour: patch lists too long");
            return CFD_ERR_RANGE;
        }
        std::unique_ptr<unsigned char[]> all(new unsigned char[words * 16]);  // every byte written below
        parallel_patches([&](int, int64_t q0, int64_t q1) {
            for (int pos = (int)q0; pos < (int)q1; pos++)
                std::memcpy(all.get() + (size_t)desc[dir][pos].x * 16, lists[dir][pos].data(), lists[dir][pos].size());
        });
        CFD_CUDA(mc.desc[dir].upload(desc[dir].data(), desc[dir].size(), c->stream));
        CFD_CUDA(mc.lists[dir].upload(reinterpret_cast<const uint4 *>(all.get()), words, c->stream));
        CFD_CUDA(stream_wait(c->stream));
    }
    // update lists of the factorisation: for lower block (i,p), the upper
    // blocks (p,j) of row p whose column j row i also holds
    // Row i's pairs in order: for each lower block u, the upper entries v of
    // row p = JA[slot[base+u]] whose column row i holds, with its CRS-local slot.
    // Counted, then written, per row.  local[j] = that slot of column j, -1 outside
    // the call (searching the row for each column took three times as long).
    // hdr and pairs are written whole by the rows' threads (zeroing 500 MB each at
    // 128^3 on one thread took longer than the lists themselves)
    std::unique_ptr<int4[]> hdr(new int4[c->nnzb]);
    std::vector<int> ext_pairs(n, 0);  // pairs of each row's off-patch blocks
    std::vector<int> ext_most(n, 0);   // and the most of one such block
    std::vector<int64_t> pair_ptr(n + 1, 0);
    // returns the row's pair count; writes the pairs and headers when out != nullptr
    auto row_pairs = [&](int i, int2 *out, std::vector<int> &local) {
        const int base = IA[i], end = IA[i + 1];
        const int nlo = meta[i].y;
        for (int k = end - 1; k >= base; k--) local[JA[k]] = k - base;
        int total = 0, next_pairs = 0;
        for (int u = 0; u < nlo; u++) {
            const int kk = slot[base + u], p = JA[kk];
            // see k_mc_factor: blocks of the patch's own rows are named by their CRS position in the patch
            const bool own = u >= meta[i].x, named = own && mc.by_cta;
            const int patch0 = IA[i / kMcRows * kMcRows];
            int cnt = 0;
            for (int v = IA[p] + meta[p].y + 1; v < IA[p + 1]; v++) {
                const int l = local[scol[v]];
                if (l < 0) continue;
                if (out) out[total + cnt] = make_int2(named ? slot[v] - patch0 : (int)loc[v], l);
                cnt++;
            }
            if (out) {
                const int dg = IA[p] + meta[p].y;  // the diagonal's list entry
                hdr[base + u] = make_int4(named ? slot[dg] - patch0 : (int)loc[dg], cnt, kk - base,
                                          own ? meta[p].w & 255 : 0);
                if (!own) next_pairs += cnt;
            }
            if (!out && !own) ext_most[i] = std::max(ext_most[i], cnt);
            total += cnt;
        }
        for (int k = base; k < end; k++) local[JA[k]] = -1;
        if (out) std::fill(hdr.get() + base + nlo, hdr.get() + end, make_int4(0, 0, 0, 0));
        // other threads read the level meanwhile: the counts go in afterwards
        if (out) ext_pairs[i] = next_pairs;
        return total;
    };
    parallel_rows([&](int i0, int i1) {
        std::vector<int> local(n, -1);
        for (int i = i0; i < i1; i++) pair_ptr[i + 1] = row_pairs(i, nullptr, local);
    });
    int maxstage = 1;
    for (int i = 0; i < n; i++) {
        maxstage = std::max<int64_t>(maxstage, meta[i].y + pair_ptr[i + 1]);
        pair_ptr[i + 1] += pair_ptr[i];
    }
    int64_t maxpairs = 1;
    for (int P = 0; P < np; P++)
        maxpairs = std::max(maxpairs, pair_ptr[std::min(n, (P + 1) * kMcRows)] - pair_ptr[P * kMcRows]);
    // the CTA-per-patch factorisation, when its patches fit in either precision
    mc.maxblk = maxblk;
    mc.maxpairs = (int)std::min<int64_t>(maxpairs, 1 << 24);
    mc.stage = std::max(24, 1 + *std::max_element(ext_most.begin(), ext_most.end()));
    mc.by_cta = mc_factor_cta_bytes(mc.maxblk, mc.maxpairs) + (size_t)kMcFactorWarps * mc.stage * 25 * sizeof(double) <=
                kMcFactorBytes;
    std::unique_ptr<int2[]> pairs(new int2[std::max<int64_t>(pair_ptr[n], 1)]);
    parallel_rows([&](int i0, int i1) {
        std::vector<int> local(n, -1);
        for (int i = i0; i < i1; i++) row_pairs(i, pairs.get() + pair_ptr[i], local);
    });
    for (int i = 0; i < n; i++) meta[i].w |= ext_pairs[i] << 8;
    mc.maxrow = maxrow;
    mc.maxstage = maxstage;
    CFD_CUDA(mc.patches.upload(patches.data(), patches.size(), c->stream));
    CFD_CUDA(mc.slot.upload(slot.data(), slot.size(), c->stream));
    CFD_CUDA(mc.meta.upload(meta.data(), meta.size(), c->stream));
    std::vector<unsigned> place(c->nnzb);  // by CRS position
    parallel_ranges(c->nnzb, [&](int, int64_t u0, int64_t u1) {
        for (int64_t u = u0; u < u1; u++) place[slot[u]] = loc[u];
    });
    CFD_CUDA(mc.loc.upload(place.data(), place.size(), c->stream));
    CFD_CUDA(mc.hdr.upload(hdr.get(), (size_t)c->nnzb, c->stream));
    CFD_CUDA(mc.pair_ptr.upload(pair_ptr.data(), pair_ptr.size(), c->stream));
    CFD_CUDA(mc.pairs.upload(pairs.get(), (size_t)pair_ptr[n], c->stream));
    CFD_CUDA(stream_wait(c->stream));  // host vectors go out of scope
    mc.built = true;
    return CFD_OK;
}

// Whether a colour of cnt patches is factored by a CTA per patch, from measured
// costs per colour (microseconds; p patches per SM, b blocks per row, l levels
// per patch): p (2.3 b + 1.7 l) with a CTA per patch, whose levels follow one
// another; with a warp per patch 26-30 b for its 32 rows, whatever p, and from
// some 15 patches per SM, when its twenty warps are busy, 3.2 b p with FP32 and
// 4.1 b p with FP64 factors (fewer warps fit).
static bool mc_factor_by_cta(const cfd_ctx *c, int cnt, size_t elem) {
    const Abmc &mc = c->mc;
    const double b = (double)c->nnzb / c->nnode, p = (double)cnt / c->nsm;
    return mc.by_cta && (p * (b + 1.7 * mc.levels) <= 30.0 * b || (elem == 8 && 1.7 * mc.levels <= 1.3 * b));
}

template <typename TA, typename TM>
int mc_factor(cfd_ctx *c, const TA *A, TM *M) {
    Abmc &mc = c->mc;
    int st = mc_build(c);
    if (st) return st;
    CFD_CUDA(allow_max_dynamic_smem(k_mc_solve<TM, false, true>, c->device, nullptr));
    CFD_CUDA(allow_max_dynamic_smem(k_mc_solve<TM, true, true>, c->device, nullptr));
    // the slots' empty places read as zeros
    CFD_CUDA(cudaMemsetAsync(M, 0, (size_t)mc.nelem * sizeof(TM), c->stream));
    // four warps (patches) per CTA, fewer when their staging does not fit in
    // 200 KB; several CTAs share an SM so every SM gets patches
    const size_t per_warp = mc_factor_warp_bytes<TM>(mc.maxrow, mc.maxstage);
    const int nwarp = (int)std::max<size_t>(1, std::min<size_t>(4, (200u << 10) / per_warp));
    if (per_warp > (200u << 10)) {
        set_error("ILU(0) multicolour: a row needs %d staged blocks, more than fit in shared memory",
                  mc.maxrow + mc.maxstage);
        return CFD_ERR_RANGE;
    }
    const size_t smem = per_warp * nwarp;
    const size_t smem_cta = mc_factor_cta_bytes(mc.maxblk, mc.maxpairs) + (size_t)kMcFactorWarps * mc.stage * 25 * sizeof(TM);
    int smax = 0;
    CFD_CUDA(allow_max_dynamic_smem(k_mc_factor<TA, TM>, c->device, &smax));
    if (smem > (size_t)smax) {
        set_error("ILU(0) multicolour: %zu bytes of shared memory needed, %d available", smem, smax);
        return CFD_ERR_RANGE;
    }
    CFD_CUDA(allow_max_dynamic_smem(k_mc_factor_cta<TA, TM>, c->device, &smax));
    for (int k = 0; k < mc.ncolor; k++) {
        const int cnt = mc.cptr[k + 1] - mc.cptr[k];
        if (smem_cta <= (size_t)smax && mc_factor_by_cta(c, cnt, sizeof(TM)))
            k_mc_factor_cta<TA, TM><<<cnt, 32 * kMcFactorWarps, smem_cta, c->stream>>>(
                mc.patches.p + mc.cptr[k], c->nnode, mc.maxblk, mc.maxpairs, mc.stage, c->IA.p, mc.slot.p, mc.meta.p,
                mc.hdr.p, mc.loc.p, mc.pair_ptr.p, mc.pairs.p, A, M, c->err.p);
        else
            k_mc_factor<TA, TM><<<grid_for(cnt, nwarp), 32 * nwarp, smem, c->stream>>>(
                mc.patches.p + mc.cptr[k], cnt, c->nnode, mc.maxrow, mc.maxstage, mc.by_cta, c->IA.p, mc.slot.p, mc.meta.p,
                mc.hdr.p, mc.loc.p, mc.pair_ptr.p, mc.pairs.p, A, M, c->err.p);
    }
    CFD_LAUNCH_CHECK();
    return CFD_OK;
}

template <typename TM, bool BWD>
static int mc_solve_launch(cfd_ctx *c, int k, bool dependent, const TM *M, const double *r, double *out) {
    const Abmc &mc = c->mc;
    const int4 sh = mc.shape[BWD][k];
    const int npatch = mc.cptr[k + 1] - mc.cptr[k];
    const size_t lists = (size_t)sh.x * 16 + ((size_t)sh.z + 1) * 40;
    // the diagonal and intra-patch blocks are staged whole or not at all
    const bool staged = lists <= kMcListBytes && sh.w <= kMcStageUnits * kMcUnit;
    auto bytes = [&](int units) { return lists + (size_t)units * kMcUnit * sizeof(TM); };
    int units = std::min(sh.y, kMcStageUnits);
    if ((size_t)npatch > (size_t)c->nsm * ((220u << 10) / (bytes(units) + 3072)))
        units = std::min(units, std::max(McStageMany<TM>::units, (sh.w + kMcUnit - 1) / kMcUnit));
    if (!staged) units = 0;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(npatch);
    lc.blockDim = dim3(kMcSolveThreads);
    lc.dynamicSmemBytes = staged ? bytes(units) : 0;
    lc.stream = c->stream;
    lc.attrs = at;
    lc.numAttrs = dependent ? 1 : 0;
    auto kern = staged ? k_mc_solve<TM, BWD, true> : k_mc_solve<TM, BWD, false>;
    CFD_CUDA(cudaLaunchKernelEx(&lc, kern, (const int4 *)(mc.desc[BWD].p + mc.cptr[k]), (const uint4 *)mc.lists[BWD].p,
                                M, r, out, sh.x, units));
    return CFD_OK;
}

template <typename TM>
static int mc_apply_launch(cfd_ctx *c, const TM *M, const double *r, double *tmp, double *z) {
    const Abmc &mc = c->mc;
    int st;
    // the first colour starts after the stream's earlier work has completed
    // (no early start), so r is complete in every colour's launch
    for (int k = 0; k < mc.ncolor; k++)
        if ((st = mc_solve_launch<TM, false>(c, k, k > 0, M, r, tmp))) return st;
    for (int k = mc.ncolor - 1; k >= 0; k--)
        if ((st = mc_solve_launch<TM, true>(c, k, true, M, tmp, z))) return st;
    CFD_LAUNCH_CHECK();
    return CFD_OK;
}

// The 2 x ncolor launches of an apply, replayed as one captured CUDA graph
// when the context has its own stream (the legacy stream cannot be
// captured): the host then issues one launch instead of 2 x ncolor, which is
// what bounds small systems.  Graphs are cached per factor type and pointer set.
template <typename TM>
int mc_apply(cfd_ctx *c, const TM *M, const double *r, double *tmp, double *z) {
    Abmc &mc = c->mc;
    if (!c->stream) return mc_apply_launch<TM>(c, M, r, tmp, z);
    for (const auto &g : mc.graphs)
        if (g.elem == sizeof(TM) && g.M == M && g.r == r && g.tmp == tmp && g.z == z) {
            CFD_CUDA(cudaGraphLaunch(g.exec, c->stream));
            return CFD_OK;
        }
    if (mc.graphs.size() >= 64) mc.clear_graphs();
    cudaGraph_t graph = nullptr;
    CFD_CUDA(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    const int st = mc_apply_launch<TM>(c, M, r, tmp, z);
    const cudaError_t e = cudaStreamEndCapture(c->stream, &graph);
    if (st) {
        if (graph) cudaGraphDestroy(graph);
        return st;
    }
    CFD_CUDA(e);
    cudaGraphExec_t exec = nullptr;
    const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    CFD_CUDA(ei);
    mc.graphs.push_back({sizeof(TM), M, r, tmp, z, exec});
    CFD_CUDA(cudaGraphLaunch(exec, c->stream));
    return CFD_OK;
}

template int mc_factor<double, double>(cfd_ctx *, const double *, double *);
template int mc_factor<double, float>(cfd_ctx *, const double *, float *);
template int mc_factor<float, float>(cfd_ctx *, const float *, float *);
template int mc_factor<uint16_t, float>(cfd_ctx *, const uint16_t *, float *);
template int mc_apply<double>(cfd_ctx *, const double *, const double *, double *, double *);
template int mc_apply<float>(cfd_ctx *, const float *, const double *, double *, double *);

}  // namespace cfd

using namespace cfd;

extern "C" int cfd_ilu_mc_order(cfd_ctx *c, int *order, int *ncolor) {
    if (!c || !c->has_mesh) { cfd::set_error("cfd_ilu_mc_order: no mesh"); return CFD_ERR_STATE; }
    CFD_CUDA(cudaSetDevice(c->device));
    int st = mc_build(c);
    if (st) return st;
    const Abmc &mc = c->mc;
    if (ncolor) *ncolor = mc.ncolor;
    if (order) {
        const int n = c->nnode;
        int k = 0;
        for (int col = 0; col < mc.ncolor; col++)
            for (int P = 0; P * kMcRows < n; P++)
                if (mc.h_pcolor[P] == col)
                    for (int i = P * kMcRows; i < std::min(n, (P + 1) * kMcRows); i++) order[k++] = i;
    }
    return CFD_OK;
}
