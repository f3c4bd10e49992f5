// Core of the B200 edge-based finite-volume path: context lifecycle, mesh
// upload and device layout, boundary conditions, flux residual, local time
// step, residual RMS, approximate Roe Jacobian assembly, level-scheduled block
// Gauss-Seidel, solution update, and the C ABI around them.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

#include "ctx.cuh"
#include "host_par.h"
#include "kernels.cuh"

namespace cfd {

static thread_local char g_err[512] = "";

void set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

static inline double bitsd(unsigned long long u) {
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}

// ----------------------------------------------------------------- kernels

// Characteristic ghost states, one thread per boundary edge
// (Apply_Characteristic_Boundary_Condition, Euler3D/src/BC.cpp:1440-1487).
// list: the boundary edges to update (nullptr: edges 0 .. nbedge-1)
__global__ void k_apply_bc(int nbedge, int64_t ldq, double *__restrict__ Q, const int2 *__restrict__ bn,
                           const double4 *__restrict__ bg, const int *__restrict__ btype, Flow f,
                           int *__restrict__ err, const int *__restrict__ list) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nbedge) return;
    const int b = list ? list[t] : t;
    int2 nd = bn[b];
    double4 g = bg[b];
    double qI[5], qG[5], qB[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        qI[k] = Q[k * ldq + nd.x];
        qG[k] = Q[k * ldq + nd.y];
    }
    const int st = f.flux == CFD_FLUX_ROE_PRECOND ? precond_characteristic_bc(qI, qG, g.x, g.y, g.z, btype[b], f, qB)
                                                  : characteristic_bc(qI, qG, g.x, g.y, g.z, btype[b], f, qB);
    if (st) atomicOr(err, st == 1 ? ERR_BC_NEG_PRESSURE : ERR_BC_UNCLASSIFIED);
#pragma unroll
    for (int k = 0; k < 5; k++) Q[k * ldq + nd.y] = qB[k];
}

__device__ __forceinline__ void warp_minmax(double &mn, double &mx) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
}

// Block-wide min/max of 3 (min,max) pairs folded into the global extrema
// words with ordered-bit atomics (values are >= 0, so the IEEE bit pattern
// orders like the value; min/max are order independent, hence deterministic).
__device__ __forceinline__ void block_extrema3(double mn[3], double mx[3], unsigned long long *ext) {
    __shared__ double s_mn[3][32], s_mx[3][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        warp_minmax(mn[j], mx[j]);
        if (lane == 0) { s_mn[j][wid] = mn[j]; s_mx[j][wid] = mx[j]; }
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double a = lane < nw ? s_mn[j][lane] : DBL_MAX;
            double b = lane < nw ? s_mx[j][lane] : 0.0;
            warp_minmax(a, b);
            if (lane == 0) {
                atomicMin(&ext[2 * j], (unsigned long long)__double_as_longlong(a));
                atomicMax(&ext[2 * j + 1], (unsigned long long)__double_as_longlong(b));
            }
        }
    }
}

// Second-order face state (Compute_SecondOrderReconstructQ,
// Euler3D/src/HigherOrderReconstructQ.cpp:21-72) for the side `s` of an edge
// towards `o`: q = Q_s + phi_s*(frac*(Q_o - Q_s) + (1-frac)*grad_s . r),
// r = 0.5 (x_o - x_s).
__device__ __forceinline__ void reconstruct(const double qs[5], const double qo[5], int s, double rx, double ry,
                                            double rz, const double *__restrict__ grad, const double *__restrict__ phi,
                                            int nnode, bool limited, double frac, double out[5]) {
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const double gx = grad[(3 * k) * (int64_t)nnode + s];
        const double gy = grad[(3 * k + 1) * (int64_t)nnode + s];
        const double gz = grad[(3 * k + 2) * (int64_t)nnode + s];
        const double ph = limited ? phi[k * (int64_t)nnode + s] : 1.0;
        out[k] = qs[k] + ph * (frac * (qo[k] - qs[k]) + (1.0 - frac) * (gx * rx + gy * ry + gz * rz));
    }
}

// Flux residual, node-gather form: one thread per node walks its incident
// interior edges in a fixed order (neighbour id) and accumulates +flux (the node
// is node_L) or -flux (node_R); no atomics touch the residual, so every node's
// sum has a deterministic order.  The flux of edge (L,R) is always evaluated in
// the reference's orientation (Q_L, Q_R, n_{L->R}), so both endpoints see
// bit-identical values (Compute_Residual_Roe_New, FluxTest.cpp:7968-8100).
// Incidence is stored sliced-ELL (slices of 32 nodes, slot k of a slice's
// lanes contiguous): neighbour id (~id when the node is node_R) and the edge's
// unit normal + area per slot, so the per-edge loads of a warp are coalesced;
// the node's own state, gradients, limiters and coordinates stay in registers.
// KAPPA0: second order with frac = 0 (the default LIMITER_ORDER), where the
// reconstruction frac (Q_o - Q_s) + (1 - frac) grad_s.r rounds to grad_s.r
// exactly (up to the sign of an exact zero), so those terms are not formed.
#define GATHER_PARAMS                                                                                        \
    int nnode, int64_t ldq, const double *__restrict__ Q, const double *__restrict__ grad,                    \
        const double *__restrict__ phi, const double *__restrict__ xyz, const int64_t *__restrict__ sell_ptr, \
        const int *__restrict__ sell_nbr, const double4 *__restrict__ sell_geo, const int *__restrict__ deg,   \
        Flow f, int add_time, int checks, int *__restrict__ roeflag, int *__restrict__ fixcount,                 \
        double *__restrict__ res, double *__restrict__ resd, double *__restrict__ dtsum, const double *__restrict__ lgrad
#define GATHER_ARGS \
    nnode, ldq, Q, grad, phi, xyz, sell_ptr, sell_nbr, sell_geo, deg, f, add_time, checks, roeflag, fixcount, res, resd, \
        dtsum, lgrad

template <int FLUX, bool SECOND, bool KAPPA0, bool LG, bool RUP>
__device__ __forceinline__ void residual_gather_node_v(int i, GATHER_PARAMS, double mn[3], double mx[3]) {
    {
        const bool limited = f.limiter != CFD_LIMITER_NONE;
        double qo[5], go[15], po[5], xo[3];
#pragma unroll
        for (int v = 0; v < 5; v++) qo[v] = Q[v * ldq + i];
        if (SECOND) {
#pragma unroll
            for (int k = 0; k < 15; k++) go[k] = LG ? lgrad[k * (int64_t)nnode + i] : grad[k * (int64_t)nnode + i];
#pragma unroll
            for (int v = 0; v < 5; v++) po[v] = limited ? phi[v * (int64_t)nnode + i] : 1.0;
#pragma unroll
            for (int d = 0; d < 3; d++) xo[d] = xyz[d * (int64_t)nnode + i];
        }
        double ac[5] = {0, 0, 0, 0, 0}, ad[5] = {0, 0, 0, 0, 0}, adt = 0.0;
        int bad = 0;  // bit 0: Roe-average pressure < 0, bit 1: own reconstructed pressure < 0
        const int64_t base = sell_ptr[i >> 5] + (i & 31);
        const int d = deg[i];
        // the next slot's neighbour id is loaded one edge ahead, so the
        // neighbour gathers of an edge do not wait for their index load
        int sn_next = d > 0 ? sell_nbr[base] : 0;
        for (int k = 0; k < d; k++) {
            const int sn = sn_next;
            if (k + 1 < d) sn_next = sell_nbr[base + 32 * (k + 1)];
            const double4 g = sell_geo[base + 32 * k];
            const bool own_is_L = sn >= 0;
            const int j = own_is_L ? sn : ~sn;
            double qn[5], fo[5], fn[5];
#pragma unroll
            for (int v = 0; v < 5; v++) qn[v] = Q[v * ldq + j];
            if (SECOND) {
                const double rx = 0.5 * (xyz[j] - xo[0]);
                const double ry = 0.5 * (xyz[nnode + j] - xo[1]);
                const double rz = 0.5 * (xyz[2 * (int64_t)nnode + j] - xo[2]);
#pragma unroll
                for (int v = 0; v < 5; v++) {
                    const double gno = go[3 * v] * rx + go[3 * v + 1] * ry + go[3 * v + 2] * rz;
                    if (LG) {
                        const double gnn = -(lgrad[(3 * v) * (int64_t)nnode + j] * rx +
                                             lgrad[(3 * v + 1) * (int64_t)nnode + j] * ry +
                                             lgrad[(3 * v + 2) * (int64_t)nnode + j] * rz);
                        fo[v] = qo[v] + gno;
                        fn[v] = qn[v] + gnn;
                        continue;
                    }
                    const double gnn = -(grad[(3 * v) * (int64_t)nnode + j] * rx +
                                         grad[(3 * v + 1) * (int64_t)nnode + j] * ry +
                                         grad[(3 * v + 2) * (int64_t)nnode + j] * rz);
                    const double pn = limited ? phi[v * (int64_t)nnode + j] : 1.0;
                    if (KAPPA0) {
                        fo[v] = qo[v] + po[v] * gno;
                        fn[v] = qn[v] + pn * gnn;
                    } else {
                        fo[v] = qo[v] + po[v] * (f.frac * (qn[v] - qo[v]) + (1.0 - f.frac) * gno);
                        fn[v] = qn[v] + pn * (f.frac * (qo[v] - qn[v]) + (1.0 - f.frac) * gnn);
                    }
                }
                // the limiter's reconstructed-pressure correction (Limiters.cpp:273-304)
                // tests exactly this node's own face states
                if ((checks & 2) && recon_pressure_negative<RUP ? 1 : 0>(fo, f)) bad |= 2;
            } else {
#pragma unroll
                for (int v = 0; v < 5; v++) { fo[v] = qo[v]; fn[v] = qn[v]; }
            }
            double qL[5], qR[5];
#pragma unroll
            for (int v = 0; v < 5; v++) {
                qL[v] = own_is_L ? fo[v] : fn[v];
                qR[v] = own_is_L ? fn[v] : fo[v];
            }
            if (SECOND && !roe_c2_of<FLUX>() && (checks & 1) && roe_avg_pressure<RUP ? 1 : 0>(qL, qR, f) < 0.0)
                bad |= 1;
            double cf[5], df[5], lam[3], c2 = 1.0;
            const double lmax = edge_flux<FLUX, RUP ? 1 : 0>(qL, qR, g.x, g.y, g.z, g.w, f, cf, df, lam,
                                                SECOND && roe_c2_of<FLUX>() ? &c2 : nullptr);
            if (SECOND && roe_c2_of<FLUX>() && (checks & 1) && c2 < 0.0) bad |= 1;
            const double sg = own_is_L ? 1.0 : -1.0;
#pragma unroll
            for (int v = 0; v < 5; v++) {
                ac[v] += sg * cf[v];
                ad[v] += sg * df[v];
            }
            adt += g.w * lmax;
#pragma unroll
            for (int m = 0; m < 3; m++) { mn[m] = fmin(mn[m], lam[m]); mx[m] = fmax(mx[m], lam[m]); }
        }
        if (bad) {
            roeflag[i] = bad;
            if (bad & 1) atomicAdd(&fixcount[0], 1);
            if (bad & 2) atomicAdd(&fixcount[1], 1);
        }
#pragma unroll
        for (int v = 0; v < 5; v++) {
            res[v * (int64_t)nnode + i] = ac[v];
            resd[v * (int64_t)nnode + i] = ad[v];
        }
        if (add_time) dtsum[i] = adt;
    }
}

// The variable set is a compile-time constant of each kernel (RUP; every
// launch passes a Flow whose rup matches): the conservative kernels hold no
// reference to f.rup and carry no RUP branches.
template <int FLUX, bool SECOND, bool KAPPA0, bool LG = false, bool RUP = false>
__device__ __forceinline__ void residual_gather_node(int i, GATHER_PARAMS, double mn[3], double mx[3]) {
    residual_gather_node_v<FLUX, SECOND, KAPPA0, LG, RUP>(i, GATHER_ARGS, mn, mx);
}

template <int FLUX, bool SECOND, bool KAPPA0 = false, bool LG = false, bool RUP = false>
// Nodes [lo, hi) (lo a multiple of the block size; the whole mesh is 0, nnode).
__global__ void __launch_bounds__(128, 3) k_residual_gather(GATHER_PARAMS, unsigned long long *__restrict__ ext,
                                                            int lo, int hi) {
    const int i = lo + blockIdx.x * blockDim.x + threadIdx.x;
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {0.0, 0.0, 0.0};
    if (i < hi) residual_gather_node<FLUX, SECOND, KAPPA0, LG, RUP>(i, GATHER_ARGS, mn, mx);
    if (add_time) block_extrema3(mn, mx, ext);
}

// The gated re-evaluation after a limiter fix (gate = the fix counters): a
// grid of a few CTAs per SM strides over the nodes, so that the usual case,
// no node failed, costs one short wave instead of the full grid's.
template <int FLUX, bool SECOND, bool KAPPA0 = false, bool RUP = false>
__global__ void __launch_bounds__(128, 3) k_residual_gather_rerun(GATHER_PARAMS, const int *__restrict__ gate,
                                                                  unsigned long long *__restrict__ ext) {
    if (gate[0] == 0 && gate[1] == 0) return;
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {0.0, 0.0, 0.0};
    for (int b = blockIdx.x * blockDim.x; b < nnode; b += gridDim.x * blockDim.x) {
        const int i = b + threadIdx.x;
        if (i < nnode) residual_gather_node<FLUX, SECOND, KAPPA0, false, RUP>(i, GATHER_ARGS, mn, mx);
    }
    if (add_time) block_extrema3(mn, mx, ext);
}

// One launch of the gather residual over several contexts (a request table):
// block b belongs to the job whose [block_begin, block_begin + ceil(nnode/128))
// range holds it, and its threads run exactly the per-node code of
// k_residual_gather on that job's arrays and parameters, so every node's
// residual is the job's own launch's to round-off.  The serving loop uses it
// to fuse the interior residuals of the requests it runs side by side
// (conservative states only; RUP requests launch on their own).
template <int FLUX, bool SECOND, bool KAPPA0, bool LG>
__global__ void __launch_bounds__(128, 3) k_residual_gather_batch(const __grid_constant__ GatherBatch B) {
    int j = 0;
    while (j + 1 < B.njobs && (int)blockIdx.x >= B.job[j + 1].block_begin) j++;
    const GatherJob &J = B.job[j];
    const int i = ((int)blockIdx.x - J.block_begin) * blockDim.x + threadIdx.x;
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {0.0, 0.0, 0.0};
    if (i < J.nnode)
        residual_gather_node<FLUX, SECOND, KAPPA0, LG>(i, J.nnode, J.ldq, J.Q, J.grad, J.phi, J.xyz, J.sell_ptr,
                                                        J.sell_nbr, J.sell_geo, J.deg, J.f, J.add_time, J.checks,
                                                        J.roeflag, J.fixcount, J.res, J.resd, J.dtsum, J.lgrad, mn,
                                                        mx);
    if (J.add_time) block_extrema3(mn, mx, J.ext);
}

template <int FLUX>
static int launch_gather_batch_flux(int key, const GatherBatch &b, cudaStream_t s) {
    int blocks = 0;
    for (int k = 0; k < b.njobs; k++) blocks += grid_for(b.job[k].nnode, 128);
    if (blocks == 0) return CFD_OK;
    switch (key & 7) {
        case 0: k_residual_gather_batch<FLUX, false, false, false><<<blocks, 128, 0, s>>>(b); break;
        case 4: k_residual_gather_batch<FLUX, true, false, false><<<blocks, 128, 0, s>>>(b); break;
        case 6: k_residual_gather_batch<FLUX, true, true, false><<<blocks, 128, 0, s>>>(b); break;
        case 7: k_residual_gather_batch<FLUX, true, true, true><<<blocks, 128, 0, s>>>(b); break;
        default: return CFD_ERR_UNSUPPORTED;
    }
    CFD_LAUNCH_CHECK();
    return CFD_OK;
}

int launch_gather_batch(int key, const GatherBatch &b, cudaStream_t s) {
    switch (key >> 3) {
        case CFD_FLUX_ROE: return launch_gather_batch_flux<CFD_FLUX_ROE>(key, b, s);
        case CFD_FLUX_HLLC: return launch_gather_batch_flux<CFD_FLUX_HLLC>(key, b, s);
        case CFD_FLUX_AUSM: return launch_gather_batch_flux<CFD_FLUX_AUSM>(key, b, s);
        default: return CFD_ERR_UNSUPPORTED;
    }
}

// Boundary edges of the gather residual: first order, flux into node_L only
// (FluxTest.cpp:8044-8098).  One thread per node that has boundary edges
// (`bnode`, increasing), launched after k_residual_gather: it continues the
// node's interior sums with its boundary edges in increasing order, the
// order one loop over both would take, so every sum is the same bit for bit.
// Kept out of the interior kernel because the ~5 % of nodes that carry
// boundary edges sit in ~20 % of its warps, whose other lanes would idle
// through them.
template <int FLUX>
__global__ void __launch_bounds__(128) k_residual_bnd(
    int nbnode, const int *__restrict__ bnode, int nnode, int64_t ldq, const double *__restrict__ Q,
    const int *__restrict__ n2b_ptr, const int *__restrict__ n2b, const int2 *__restrict__ bn,
    const double4 *__restrict__ bg, Flow f, int add_time, const int *__restrict__ gate, double *__restrict__ res,
    double *__restrict__ resd, double *__restrict__ dtsum, unsigned long long *__restrict__ ext) {
    if (gate && gate[0] == 0 && gate[1] == 0) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {0.0, 0.0, 0.0};
    if (t < nbnode) {
        const int i = bnode[t];
        double qo[5], ac[5], ad[5];
#pragma unroll
        for (int v = 0; v < 5; v++) {
            qo[v] = Q[v * ldq + i];
            ac[v] = res[v * (int64_t)nnode + i];
            ad[v] = resd[v * (int64_t)nnode + i];
        }
        double adt = add_time ? dtsum[i] : 0.0;
        for (int k = n2b_ptr[i]; k < n2b_ptr[i + 1]; k++) {
            const int b = n2b[k];
            const int2 nd = bn[b];
            const double4 g = bg[b];
            double qR[5];
#pragma unroll
            for (int v = 0; v < 5; v++) qR[v] = Q[v * ldq + nd.y];
            double cf[5], df[5], lam[3];
            const double lmax = edge_flux<FLUX>(qo, qR, g.x, g.y, g.z, g.w, f, cf, df, lam);
#pragma unroll
            for (int v = 0; v < 5; v++) {
                ac[v] += cf[v];
                ad[v] += df[v];
            }
            adt += g.w * lmax;
#pragma unroll
            for (int m = 0; m < 3; m++) { mn[m] = fmin(mn[m], lam[m]); mx[m] = fmax(mx[m], lam[m]); }
        }
#pragma unroll
        for (int v = 0; v < 5; v++) {
            res[v * (int64_t)nnode + i] = ac[v];
            resd[v * (int64_t)nnode + i] = ad[v];
        }
        if (add_time) dtsum[i] = adt;
    }
    if (add_time) block_extrema3(mn, mx, ext);
}

// Flux residual, patch form: one CTA per patch of CFD_PATCH_NODES consecutive
// nodes.  Phase 0 stages the node data of the patch and of its halo into
// shared memory with coalesced loads (SoA, one row per variable).  The edges
// of the patch (each interior edge touching the patch; edges cut by the patch
// boundary are evaluated by both patches) are then processed in chunks of
// PATCH_CHUNK: every thread evaluates one edge flux from shared memory into a
// chunk buffer, and each owned node adds the contributions of the chunk in
// increasing local edge order (+ when it is node_L, - when it is node_R).  No
// atomics on the residual, deterministic summation order, one flux evaluation
// per edge per patch instead of one per edge end, and the L1 cache stays free
// for the few global loads left (ghost states of boundary edges).
// `gate`: when non-null and both fix counters are zero the launch does nothing
// (conditional re-evaluation after the limiter's pressure fixes).
template <int FLUX, bool SECOND>
__global__ void __launch_bounds__(PATCH_CHUNK, 2) k_residual_patch(
    int nnode, int64_t ldq, const double *__restrict__ Q, const double *__restrict__ grad,
    const double *__restrict__ phi, const double *__restrict__ xyz, const int *__restrict__ pe_ptr,
    const int *__restrict__ pe_loc, const double4 *__restrict__ pe_geo, const int *__restrict__ ph_ptr,
    const int *__restrict__ halo, const int *__restrict__ inc_ptr, const int *__restrict__ inc,
    const int *__restrict__ n2b_ptr, const int *__restrict__ n2b, const int2 *__restrict__ bn,
    const double4 *__restrict__ bg, Flow f, int add_time, int nlm, int check_roe, int *__restrict__ roeflag,
    int *__restrict__ fixcount, const int *__restrict__ gate, double *__restrict__ res, double *__restrict__ resd,
    double *__restrict__ dtsum, unsigned long long *__restrict__ ext) {
    if (gate && gate[0] == 0 && gate[1] == 0) return;
    constexpr int NV = SECOND ? PATCH_NV2 : 5;
    extern __shared__ double sm[];
    double *nv = sm;                       // [NV][nlm]: Q 0-4 | grad 5-19 | phi 20-24 | xyz 25-27
    double *cb = sm + (size_t)NV * nlm;    // [11][PATCH_CHUNK]
    const int p = blockIdx.x, tid = threadIdx.x;
    const int n0 = p * CFD_PATCH_NODES;
    const int nown = min(CFD_PATCH_NODES, nnode - n0);
    const int h0 = ph_ptr[p], nloc = nown + ph_ptr[p + 1] - h0;
    const bool limited = f.limiter != CFD_LIMITER_NONE;
    // phase 0: stage owned + halo node data
    for (int l = tid; l < nloc; l += PATCH_CHUNK) {
        const int g = l < nown ? n0 + l : halo[h0 + l - nown];
#pragma unroll
        for (int v = 0; v < 5; v++) nv[v * nlm + l] = Q[v * ldq + g];
        if (SECOND) {
#pragma unroll
            for (int k = 0; k < 15; k++) nv[(5 + k) * nlm + l] = grad[k * (int64_t)nnode + g];
#pragma unroll
            for (int v = 0; v < 5; v++) nv[(20 + v) * nlm + l] = limited ? phi[v * (int64_t)nnode + g] : 1.0;
#pragma unroll
            for (int d = 0; d < 3; d++) nv[(25 + d) * nlm + l] = xyz[d * (int64_t)nnode + g];
        }
    }
    __syncthreads();
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {0.0, 0.0, 0.0};
    double ac[5] = {0, 0, 0, 0, 0}, ad[5] = {0, 0, 0, 0, 0}, adt = 0.0;
    int q = 0, qe = 0;
    if (tid < nown) {
        q = inc_ptr[n0 + tid];
        qe = inc_ptr[n0 + tid + 1];
    }
    const int e0 = pe_ptr[p], ne = pe_ptr[p + 1] - e0;
    for (int c0 = 0; c0 < ne; c0 += PATCH_CHUNK) {
        const int k = c0 + tid;
        if (k < ne) {
            const int lp = pe_loc[e0 + k];
            const int a = lp & 0xffff, b = lp >> 16;
            const double4 g = pe_geo[e0 + k];
            double qL[5], qR[5];
#pragma unroll
            for (int v = 0; v < 5; v++) {
                qL[v] = nv[v * nlm + a];
                qR[v] = nv[v * nlm + b];
            }
            if (SECOND) {
                const double rx = 0.5 * (nv[25 * nlm + b] - nv[25 * nlm + a]);
                const double ry = 0.5 * (nv[26 * nlm + b] - nv[26 * nlm + a]);
                const double rz = 0.5 * (nv[27 * nlm + b] - nv[27 * nlm + a]);
                double rL[5], rR[5];
#pragma unroll
                for (int v = 0; v < 5; v++) {
                    const double gL = nv[(5 + 3 * v) * nlm + a] * rx + nv[(6 + 3 * v) * nlm + a] * ry +
                                      nv[(7 + 3 * v) * nlm + a] * rz;
                    const double gR = -(nv[(5 + 3 * v) * nlm + b] * rx + nv[(6 + 3 * v) * nlm + b] * ry +
                                        nv[(7 + 3 * v) * nlm + b] * rz);
                    rL[v] = qL[v] + nv[(20 + v) * nlm + a] * (f.frac * (qR[v] - qL[v]) + (1.0 - f.frac) * gL);
                    rR[v] = qR[v] + nv[(20 + v) * nlm + b] * (f.frac * (qL[v] - qR[v]) + (1.0 - f.frac) * gR);
                }
#pragma unroll
                for (int v = 0; v < 5; v++) { qL[v] = rL[v]; qR[v] = rR[v]; }
                if (check_roe && roe_avg_pressure(qL, qR, f) < 0.0) {
                    roeflag[a < nown ? n0 + a : halo[h0 + a - nown]] = 1;
                    roeflag[b < nown ? n0 + b : halo[h0 + b - nown]] = 1;
                    atomicAdd(&fixcount[0], 1);
                }
            }
            double cf[5], df[5], lam[3];
            const double lmax = edge_flux<FLUX>(qL, qR, g.x, g.y, g.z, g.w, f, cf, df, lam);
#pragma unroll
            for (int v = 0; v < 5; v++) {
                cb[v * PATCH_CHUNK + tid] = cf[v];
                cb[(5 + v) * PATCH_CHUNK + tid] = df[v];
            }
            cb[10 * PATCH_CHUNK + tid] = g.w * lmax;
#pragma unroll
            for (int j = 0; j < 3; j++) { mn[j] = fmin(mn[j], lam[j]); mx[j] = fmax(mx[j], lam[j]); }
        }
        __syncthreads();
        const int cend = c0 + PATCH_CHUNK;
        for (; q < qe; q++) {
            const int t = inc[q];
            const int kk = (t >> 1);
            if (kk >= cend) break;
            const int s = kk - c0;
            const double sg = (t & 1) ? -1.0 : 1.0;
#pragma unroll
            for (int v = 0; v < 5; v++) {
                ac[v] += sg * cb[v * PATCH_CHUNK + s];
                ad[v] += sg * cb[(5 + v) * PATCH_CHUNK + s];
            }
            adt += cb[10 * PATCH_CHUNK + s];
        }
        __syncthreads();
    }
    if (tid < nown) {
        const int i = n0 + tid;
        for (int k = n2b_ptr[i]; k < n2b_ptr[i + 1]; k++) {
            const int b = n2b[k];
            const int2 nd = bn[b];
            const double4 g = bg[b];
            double qL[5], qR[5];
#pragma unroll
            for (int v = 0; v < 5; v++) {
                qL[v] = nv[v * nlm + tid];
                qR[v] = Q[v * ldq + nd.y];
            }
            double cf[5], df[5], lam[3];
            const double lmax = edge_flux<FLUX>(qL, qR, g.x, g.y, g.z, g.w, f, cf, df, lam);
#pragma unroll
            for (int v = 0; v < 5; v++) {
                ac[v] += cf[v];
                ad[v] += df[v];
            }
            adt += g.w * lmax;
#pragma unroll
            for (int m = 0; m < 3; m++) { mn[m] = fmin(mn[m], lam[m]); mx[m] = fmax(mx[m], lam[m]); }
        }
#pragma unroll
        for (int v = 0; v < 5; v++) {
            res[v * (int64_t)nnode + i] = ac[v];
            resd[v * (int64_t)nnode + i] = ad[v];
        }
        if (add_time) dtsum[i] = adt;
    }
    if (add_time) block_extrema3(mn, mx, ext);
}

// Limiter fixes selected by the residual's checks (count = fixcount, flag =
// per-node bits).  When no reconstructed pressure failed (count[1] == 0) the
// Roe check saw the final limiters and its flagged nodes (bit 0) drop to
// first order.  Otherwise the correction (bit 1) is applied first, as the
// reference orders the two (Limiters.cpp:61-110 after :273-304), and, when
// `redo_roe`, the corrected limiters are also copied to `work` for a full
// k_roe_pressure_fix pass.  No-op when both counts are zero.
__global__ void k_limiter_fix_apply(int nnode, const int *__restrict__ count, const int *__restrict__ flag,
                                    int redo_roe, double *__restrict__ phi, double *__restrict__ work) {
    const int nroe = count[0], npc = count[1];
    if (nroe == 0 && npc == 0) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnode; i += gridDim.x * blockDim.x) {
        const int fl = flag[i];
        if (npc == 0) {
            if (fl & 1) {
#pragma unroll
                for (int v = 0; v < 5; v++) phi[v * (int64_t)nnode + i] = 0.0;
            }
            continue;
        }
#pragma unroll
        for (int v = 0; v < 5; v++) {
            const double ph = (fl & 2) ? 0.0 : phi[v * (int64_t)nnode + i];
            if (fl & 2) phi[v * (int64_t)nnode + i] = 0.0;
            if (redo_roe) work[v * (int64_t)nnode + i] = ph;
        }
    }
}

// dt_i = V_i * CFL / sum_i (Compute_DeltaT, Euler3D/src/Time_Step.cpp:23-51).
__global__ void k_deltat(int nnode, const double *__restrict__ vol, double cfl, double *__restrict__ dt,
                         unsigned long long *__restrict__ ext) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {0.0, 0.0, 0.0};
    if (i < nnode) {
        const double d = vol[i] * cfl / dt[i];
        dt[i] = d;
        mn[0] = d;
        mx[0] = d;
    }
    __shared__ double s_mn[32], s_mx[32];
    warp_minmax(mn[0], mx[0]);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) { s_mn[wid] = mn[0]; s_mx[wid] = mx[0]; }
    __syncthreads();
    if (wid == 0) {
        double a = lane < nw ? s_mn[lane] : DBL_MAX, b = lane < nw ? s_mx[lane] : 0.0;
        warp_minmax(a, b);
        if (lane == 0) {
            atomicMin(&ext[6], (unsigned long long)__double_as_longlong(a));
            atomicMax(&ext[7], (unsigned long long)__double_as_longlong(b));
        }
    }
}

__global__ void k_fill_global_dt(int nnode, const unsigned long long *__restrict__ ext, double *__restrict__ dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nnode) dt[i] = __longlong_as_double((long long)ext[6]);
}

// Deterministic sum of squares of nvec strided vectors: stage 1 per block.
__global__ void k_sumsq_partial(const double *__restrict__ x, int64_t n, int64_t stride, int nvec,
                                double *__restrict__ part) {
    extern __shared__ double sh[];
    for (int v = 0; v < nvec; v++) {
        double s = 0.0;
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
            const double a = x[v * stride + i];
            s += a * a;
        }
        sh[threadIdx.x] = s;
        __syncthreads();
        for (int o = blockDim.x >> 1; o > 0; o >>= 1) {
            if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) part[blockIdx.x * nvec + v] = sh[0];
        __syncthreads();
    }
}

__global__ void k_sum_final(const double *__restrict__ part, int nblk, int nvec, double *__restrict__ out) {
    extern __shared__ double sh[];
    for (int v = 0; v < nvec; v++) {
        double s = 0.0;
        for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += part[b * nvec + v];
        sh[threadIdx.x] = s;
        __syncthreads();
        for (int o = blockDim.x >> 1; o > 0; o >>= 1) {
            if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) out[v] = sh[0];
        __syncthreads();
    }
}

__global__ void k_add_diss(int64_t n, const double *__restrict__ a, const double *__restrict__ b,
                           double *__restrict__ o) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) o[i] = a[i] + b[i];
}

// ---- approximate Roe Jacobian (Compute_Jacobian_Approximate_Roe,
//      Euler3D/src/Roe_Jacobian.cpp:29-228)

// Blocks of an interior edge (L,R): A[L,R] = 0.5 (J(Q_R) - |A|) area,
// A[R,L] = -0.5 (J(Q_L) + |A|) area; the rows' diagonal blocks and right-hand
// sides:
//   A[i,i] = V_i/dt_i I - sum_j A[j,i] + sum_b 0.5 (J(Q_i) + |A|)_b area_b
//   B_i    = -(Res_i [+ Res_Diss_i])
// LANES threads per row (see kJacLanesRows) walk its edges (the sliced-ELL
// incidence, whose order is that of the row's blocks) and form both blocks of
// each: its own, stored, and the transposed one, added to the diagonal block in
// registers.  Every edge is evaluated from both ends, in the same orientation
// and so to the same bits, and no block is read back: the two passes this
// replaces (edges, then rows that gathered the transposed blocks) moved the
// blocks three times, half of it in partial sectors.  Measured on the 96^3
// cube, FP32 / FP64 blocks: 1067 / 1268 us (before: 1430 / 1632), 24^3 34 / 33
// us (58 / 61).  Bound by latency at three CTAs per SM (168 registers).  The
// lanes stage their blocks in shared memory and the warp stores them one after
// the other, 100 or 200 contiguous bytes each; a row's next block follows in
// the next step, so the sectors they share fill in L2.  BF16 blocks and
// Thornber's form take this loop unrolled eight times (66^3 cube, BF16: Thornber
// 531 -> 492 us, Roe 409 -> 394; 16 times 515 and 406), the others as the compiler
// does (FP32 Roe 386 us; eight times 408, four 422, rolled 495); two matrices are
// stored by all 32 lanes (617 us, 642 with a block per step).
// The low-precision-only system sums the diagonal from the rounded blocks.
// MODE: 0 Roe, 1 preconditioned Roe (CFD_FLUX_ROE_PRECOND), 2 Thornber (|A| of
// the modified states).  RUP: the state's variables (f.rup).  HIGH / LOW: an
// FP64 / a low-precision matrix is stored.
constexpr int JAC_WARPS = 4;  // warps per CTA
// Rows up to which four lanes share a row, every fourth edge each, and add their
// parts of the diagonal block at the end.  A thread per row leaves most SMs'
// warp slots empty up to 148 SMs x 12 warps x 32 lanes / 4, and each thread then
// works off its edges one behind the other: 8^3 cube (729 rows), Roe FP64 39.5 /
// 14.9 us with 1 / 4 lanes, preconditioned Roe 78.9 / 29.2, 24^3 (15,625 rows)
// 41.4 / 33.2 and 80.4 / 64.2; 64^3 FP32 347 / 377, preconditioned 724 / 865.
// With two matrices stored, FP64 and a low-precision one, it is four lanes up to
// the same limit and two above (Roe, FP64 and FP32, 4 / 2 lanes: tets 20^3 25.2 /
// 32.8 us, 26^3 53.7 / 46.8, 48^3 255 / 271, 66^3 617 / 627, preconditioned 1063 /
// 887; hexahedra, whose rows have six edges, 16^3 12.7 / 16.7, 32^3 38.3 / 35.4,
// 96^3 977 / 844; a thread per row: tets 24^3 70, 48^3 346).
constexpr int kJacLanesRows = 16000;

template <typename TA>
__device__ __forceinline__ double round_low(double v) {
    TA t;
    store_low(&t, v);
    return load_low(&t);
}

template <typename TA, int MODE, bool RUP, bool HIGH, bool LOW, int LANES>
__global__ void __launch_bounds__(32 * JAC_WARPS, MODE == 1 ? 2 : 3) k_jacobian(
    int nnode, int64_t ldq, const double *__restrict__ Q, const int *__restrict__ IA, const int *__restrict__ IAU,
    const int64_t *__restrict__ sell_ptr, const int *__restrict__ sell_nbr, const double4 *__restrict__ sell_geo,
    const int *__restrict__ deg, const int *__restrict__ n2b_ptr, const int *__restrict__ n2b,
    const int2 *__restrict__ bn, const double4 *__restrict__ bg, const double *__restrict__ vol,
    const double *__restrict__ dt, const double *__restrict__ res, const double *__restrict__ resd, int add_time,
    int include_diss, Flow f, double *__restrict__ A64, TA *__restrict__ Alow, double *__restrict__ B) {
    f.rup = RUP ? 1 : 0;  // a compile-time constant below
    using TS = std::conditional_t<HIGH, double, TA>;  // staged blocks
    __shared__ TS stage[JAC_WARPS][32][25];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x) / LANES, sub = lane % LANES;
    if (i - lane / LANES >= nnode) return;  // whole warps past the end
    const bool live = i < nnode;
    const int row = live ? i : nnode - 1;
    const int d = live ? deg[row] : 0, first = IA[row];
    const int64_t base = sell_ptr[row >> 5] + (row & 31);
    const int steps = (int)((sell_ptr[(row >> 5) + 1] - sell_ptr[row >> 5]) / 32);
    double qi[5], D[25];
#pragma unroll
    for (int v = 0; v < 5; v++) qi[v] = Q[v * ldq + row];
    const double vd = add_time ? vol[row] / dt[row] : 0.0;
    if (MODE == 1 && add_time) {
        // preconditioned pseudo-time term (V/dt) Cinv (Roe_Jacobian.cpp:241-264)
        pc_node_cinv(qi, f, D);
#pragma unroll
        for (int k = 0; k < 25; k++) D[k] *= vd;
    } else if (RUP) {
        // (V/dt) dQ/dW
        state_time_matrix(qi, f, D);
#pragma unroll
        for (int k = 0; k < 25; k++) D[k] *= vd;
    } else {
        // no product with the zeros of the identity: V/dt may be infinite
#pragma unroll
        for (int k = 0; k < 25; k++) D[k] = k % 6 == 0 ? vd : 0.0;
    }
    if (sub > 0) {
#pragma unroll
        for (int k = 0; k < 25; k++) D[k] = 0.0;
    }
    auto dissipation = [&](const double qL[5], const double qR[5], const double4 &g, double Ab[25]) {
        if (MODE == 1) {
            pc_abs_jacobian(qL, qR, g.x, g.y, g.z, f, Ab);
        } else if (MODE == 2) {
            double mL[5], mR[5];
            thornber_states(qL, qR, f, mL, mR);
            roe_abs_jacobian(mL, mR, g.x, g.y, g.z, f, Ab);
        } else {
            roe_abs_jacobian(qL, qR, g.x, g.y, g.z, f, Ab);
        }
    };
    // the warp's staged blocks to their slots; slot < 0: none
    auto store = [&](int slot) {
        __syncwarp();
        if constexpr (HIGH && LOW) {
            // all 32 lanes, 800 elements as they lie
#pragma unroll 5
            for (int k = 0; k < 25; k++) {
                const int e = lane + 32 * k, b = e / 25;
                const int at = __shfl_sync(0xffffffffu, slot, b);
                const TS v = stage[w][b][e - 25 * b];
                if (at < 0) continue;
                const int64_t to = (int64_t)at * 25 + (e - 25 * b);
                A64[to] = v;
                store_low(Alow + to, v);
            }
        } else {
            // a block per step, lane m element m
            auto put_block = [&](int b) {
                const int at = __shfl_sync(0xffffffffu, slot, b);
                if (at < 0 || lane >= 25) return;
                const TS v = stage[w][b][lane];
                if constexpr (HIGH) A64[(int64_t)at * 25 + lane] = v;
                else Alow[(int64_t)at * 25 + lane] = v;
            };
            if constexpr (sizeof(TS) == 2 || MODE == 2) {
#pragma unroll 8
                for (int b = 0; b < 32; b++) put_block(b);
            } else {
                for (int b = 0; b < 32; b++) put_block(b);
            }
        }
        __syncwarp();
    };
    auto put = [&](int k, double v) {
        if constexpr (HIGH) stage[w][lane][k] = v;
        else store_low(&stage[w][lane][k], v);
    };
    for (int k0 = 0; k0 < steps; k0 += LANES) {
        const int k = k0 + sub;
        int slot = -1;
        if (k < d) {
            const int sn = sell_nbr[base + 32 * k];
            const double4 g = sell_geo[base + 32 * k];
            const bool own_is_L = sn >= 0;
            const int j = own_is_L ? sn : ~sn;
            double qj[5], qL[5], qR[5];
#pragma unroll
            for (int v = 0; v < 5; v++) {
                qj[v] = Q[v * ldq + j];
                qL[v] = own_is_L ? qi[v] : qj[v];
                qR[v] = own_is_L ? qj[v] : qi[v];
            }
            double Ab[25], J[25];
            dissipation(qL, qR, g, Ab);
            // own block 0.5 (+-J(Q_j) - |A|) area, transposed one 0.5 (-+J(Q_i) - |A|) area
            const double ha = 0.5 * g.w, sg = own_is_L ? 1.0 : -1.0;
            flux_jacobian(qj, g.x, g.y, g.z, f, J);
#pragma unroll
            for (int m = 0; m < 25; m++) put(m, ha * (sg * J[m] - Ab[m]));
            flux_jacobian(qi, g.x, g.y, g.z, f, J);
#pragma unroll
            for (int m = 0; m < 25; m++) {
                const double other = ha * (-sg * J[m] - Ab[m]);
                D[m] -= HIGH ? other : round_low<TA>(other);
            }
            // block k of the row, the diagonal one lying before those of larger
            // columns (the block pattern is that of the edges: require_edge_graph)
            slot = first + k + (j > row ? 1 : 0);
        }
        store(slot);
    }
    if (live)
        for (int k = n2b_ptr[row] + sub; k < n2b_ptr[row + 1]; k += LANES) {
            const int b = n2b[k];
            const int2 nd = bn[b];
            const double4 g = bg[b];
            double qR[5], Ab[25], J[25];
#pragma unroll
            for (int v = 0; v < 5; v++) qR[v] = Q[v * ldq + nd.y];
            dissipation(qi, qR, g, Ab);
            flux_jacobian(qi, g.x, g.y, g.z, f, J);
            const double ha = 0.5 * g.w;
#pragma unroll
            for (int m = 0; m < 25; m++) D[m] += ha * (J[m] + Ab[m]);
        }
#pragma unroll
    for (int o = 1; o < LANES; o *= 2)
#pragma unroll
        for (int m = 0; m < 25; m++) D[m] += __shfl_xor_sync(0xffffffffu, D[m], o);
#pragma unroll
    for (int m = 0; m < 25; m++) put(m, D[m]);
    store(live && sub == 0 ? IAU[row] : -1);
    if (live && sub == 0) {
#pragma unroll
        for (int v = 0; v < 5; v++) {
            double r = res[v * (int64_t)nnode + row];
            if (include_diss) r += resd[v * (int64_t)nnode + row];
            B[(int64_t)row * 5 + v] = -r;
        }
    }
}

// The approximate Roe Jacobian and right-hand side (MODE as k_jacobian).
template <typename TA, int MODE>
static void launch_jacobian(cfd_ctx *c, int add_time, int include_diss, double *A64, TA *Alow) {
    auto run = [&](auto kern, int lanes) {
        kern<<<grid_for((int64_t)c->nnode * lanes, 32 * JAC_WARPS), 32 * JAC_WARPS, 0, c->stream>>>(
            c->nnode, c->ldq, c->Q.p, c->IA.p, c->IAU.p, c->sell_ptr.p, c->sell_nbr.p, c->sell_geo.p, c->deg.p,
            c->n2b_ptr.p, c->n2b.p, c->bedge_nodes.p, c->bedge_geo.p, c->cvol.p, c->dt.p, c->res.p, c->resd.p,
            add_time, include_diss, c->flow, A64, Alow, c->B.p);
    };
    const bool rup = c->flow.rup != 0, split = c->nnode <= kJacLanesRows;
    if (A64 && Alow && split)
        run(rup ? k_jacobian<TA, MODE, true, true, true, 4> : k_jacobian<TA, MODE, false, true, true, 4>, 4);
    else if (A64 && Alow)
        run(rup ? k_jacobian<TA, MODE, true, true, true, 2> : k_jacobian<TA, MODE, false, true, true, 2>, 2);
    else if (A64 && split)
        run(rup ? k_jacobian<TA, MODE, true, true, false, 4> : k_jacobian<TA, MODE, false, true, false, 4>, 4);
    else if (A64)
        run(rup ? k_jacobian<TA, MODE, true, true, false, 1> : k_jacobian<TA, MODE, false, true, false, 1>, 1);
    else if (split)
        run(rup ? k_jacobian<TA, MODE, true, false, true, 4> : k_jacobian<TA, MODE, false, false, true, 4>, 4);
    else
        run(rup ? k_jacobian<TA, MODE, true, false, true, 1> : k_jacobian<TA, MODE, false, false, true, 1>, 1);
}

template <typename TA>
static void dispatch_jacobian(int mode, cfd_ctx *c, int add_time, int include_diss, double *A64, TA *Alow) {
    if (mode == 1) launch_jacobian<TA, 1>(c, add_time, include_diss, A64, Alow);
    else if (mode == 2) launch_jacobian<TA, 2>(c, add_time, include_diss, A64, Alow);
    else launch_jacobian<TA, 0>(c, add_time, include_diss, A64, Alow);
}

// ---- block Gauss-Seidel (MC_Iterative_Block_LU_Jacobi_CRS,
//      MATH/src/MC_Iterative_Jacobi.c:346-535), level scheduled.
// All arithmetic uses explicitly rounded intrinsics so no multiply-add is
// fused: the row updates then round exactly like the reference's scalar
// loops, and with identical A, B the iterates agree bit for bit.

__global__ void k_lu_nopivot(int nnode, const double *__restrict__ A, const int *__restrict__ IAU,
                             double *__restrict__ LU) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nnode) return;
    double a[25];
    const double *src = A + (int64_t)IAU[r] * 25;
#pragma unroll
    for (int k = 0; k < 25; k++) a[k] = src[k];
    // MC_Iterative_Jacobi.c:383-394
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int j = k + 1; j < 5; j++) a[j * 5 + k] = __ddiv_rn(a[j * 5 + k], a[k * 5 + k]);
#pragma unroll
        for (int j = k + 1; j < 5; j++)
#pragma unroll
            for (int i = k + 1; i < 5; i++) a[i * 5 + j] = __dsub_rn(a[i * 5 + j], __dmul_rn(a[i * 5 + k], a[k * 5 + j]));
    }
    double *dst = LU + (int64_t)r * 25;
#pragma unroll
    for (int k = 0; k < 25; k++) dst[k] = a[k];
}

__global__ void __launch_bounds__(128) k_gs_level(int nrows, const int *__restrict__ rows, const int *__restrict__ IA,
                                                  const int *__restrict__ JA, const int *__restrict__ IAU,
                                                  const double *__restrict__ A, const double *__restrict__ B,
                                                  const double *__restrict__ LU, double *__restrict__ X,
                                                  double *__restrict__ rowrms) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nrows) return;
    const int r = rows[t];
    double rhs[5];
#pragma unroll
    for (int m = 0; m < 5; m++) rhs[m] = B[(int64_t)r * 5 + m];
    for (int k = IA[r]; k < IA[r + 1]; k++) {
        const double *a = A + (int64_t)k * 25;
        const double *x = X + (int64_t)JA[k] * 5;
        double xv[5];
#pragma unroll
        for (int m = 0; m < 5; m++) xv[m] = x[m];
#pragma unroll
        for (int ii = 0; ii < 5; ii++) {
            double tv = 0.0;
#pragma unroll
            for (int jj = 0; jj < 5; jj++) tv = __dadd_rn(tv, __dmul_rn(a[ii * 5 + jj], xv[jj]));
            rhs[ii] = __dsub_rn(rhs[ii], tv);
        }
    }
    double s = 0.0;
#pragma unroll
    for (int m = 0; m < 5; m++) s = __dadd_rn(s, __dmul_rn(rhs[m], rhs[m]));
    rowrms[r] = s;
    {
        const double *a = A + (int64_t)IAU[r] * 25;
        const double *x = X + (int64_t)r * 5;
#pragma unroll
        for (int ii = 0; ii < 5; ii++) {
            double tv = 0.0;
#pragma unroll
            for (int jj = 0; jj < 5; jj++) tv = __dadd_rn(tv, __dmul_rn(a[ii * 5 + jj], x[jj]));
            rhs[ii] = __dadd_rn(rhs[ii], tv);
        }
    }
    const double *lu = LU + (int64_t)r * 25;
    double tv[5];
#pragma unroll
    for (int ii = 0; ii < 5; ii++) {
        tv[ii] = rhs[ii];
#pragma unroll
        for (int jj = 0; jj < ii; jj++) tv[ii] = __dsub_rn(tv[ii], __dmul_rn(lu[ii * 5 + jj], tv[jj]));
    }
    double xo[5];
#pragma unroll
    for (int ii = 4; ii >= 0; ii--) {
        double v = tv[ii];
#pragma unroll
        for (int jj = 4; jj > ii; jj--) v = __dsub_rn(v, __dmul_rn(lu[ii * 5 + jj], xo[jj]));
        xo[ii] = __ddiv_rn(v, lu[ii * 5 + ii]);
    }
#pragma unroll
    for (int m = 0; m < 5; m++) X[(int64_t)r * 5 + m] = xo[m];
}

// A whole sweep in one launch: one cluster of kGsCtas CTAs walks the levels,
// separated by the cluster's hardware barrier, where a launch per level costs
// 28 us for some hundred rows.  Five lanes per row (six rows per warp), lane m
// forming component m with k_gs_level's operations in the same order.  What
// does not depend on X -- a row's blocks, its LU factors and column ids -- is
// copied to shared memory one chunk of rows ahead, across level bounds; after
// the barrier one round trip to L2 fetches the values of X.
constexpr int kGsCtas = 8, kGsWarps = 4, kGsRows = 6 * kGsWarps, kGsThreads = 32 * kGsWarps;
constexpr int kGsBlocks = 16;  // blocks of a row staged (the rest are read from global memory)
// Mean rows per level up to which the cluster sweeps.  The cluster pays by the
// row, 23 / 34 / 83 ns for rows of 7 / 15 / 40 blocks, the launches by the level,
// 31 / 51-62 / 167 us (no more for 1800 rows than for 800: latency).  They break
// even near 1350 rows (hexahedra; sweep of the 80^3 box, 1262 rows per level:
// launches 13.5 ms, cluster 12.6; 88^3, 1516: 15.0 and 16.5) and between 1500
// and 1800 (tets: 64^3 in natural order, 1423: 9.8 and 9.2; blocked RCM 96^3,
// 1383: 39.7 and 31.2; 112^3, 1764: 49.5 and 48.3; 120^3, 2060: 52.0 and 58.9);
// with 40 blocks 1750 rows still gain (8.4 and 7.3 ms).  20^3 (116 rows): 2.0 and
// 0.51 ms.
static bool gs_narrow(int64_t n, int64_t nnzb, int64_t levels) {
    return n <= levels * std::min<int64_t>(1750, 1000 + 35 * nnzb / n);
}
struct GsStage {
    double A[kGsRows][kGsBlocks * 25];
    double LU[kGsRows][25];
    int JA[kGsRows][kGsBlocks];
};
struct GsShared {
    GsStage stage[2];
    double x[kGsRows][kGsBlocks * 5 + 1];
};

__device__ __forceinline__ void gs_copy8(void *smem, const void *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void gs_copy4(void *smem, const void *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}

// desc[t] = {row, first block, end, diagonal block} in level order; stop[0] != 0: nothing to do
__global__ void __launch_bounds__(kGsThreads, 1) k_gs_sweep(int nlevels, const int *__restrict__ ptr,
                                                            const int4 *__restrict__ desc, const int *__restrict__ JA,
                                                            const double *__restrict__ A, const double *__restrict__ B,
                                                            const double *__restrict__ LU, double *X,
                                                            double *__restrict__ rowrms, const int *__restrict__ stop) {
    extern __shared__ __align__(16) unsigned char gs_smem[];
    GsShared &S = *reinterpret_cast<GsShared *>(gs_smem);
    if (stop[0] != 0) return;  // the whole cluster
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane / 5, m = lane - 5 * g;
    const bool on = lane < 30;
    const int q = 6 * w + min(g, 5);          // the group's row in the chunk
    const int place = blockIdx.x * kGsRows + q;  // and in the cluster's chunk
    const unsigned group = on ? 31u << (5 * g) : 0u;
    // the chunk after (level, offset): kGsCtas * kGsRows rows of one level
    auto advance = [&](int &l, int &at) {
        at += kGsCtas * kGsRows;
        while (l < nlevels && at >= ptr[l + 1]) {
            l++;
            if (l < nlevels) at = ptr[l];
        }
    };
    auto load_desc = [&](int l, int at) {
        int4 d = make_int4(-1, 0, 0, 0);
        if (on && l < nlevels && at + place < ptr[l + 1]) d = desc[at + place];
        return d;
    };
    auto copy = [&](const int4 &d, int buf) {
        if (d.x >= 0) {
            GsStage &st = S.stage[buf];
            const int nb = min(d.z - d.y, kGsBlocks);
            for (int t = m; t < nb * 25; t += 5) gs_copy8(&st.A[q][t], A + (int64_t)d.y * 25 + t);
            for (int t = m; t < 25; t += 5) gs_copy8(&st.LU[q][t], LU + (int64_t)d.x * 25 + t);
            for (int t = m; t < nb; t += 5) gs_copy4(&st.JA[q][t], JA + d.y + t);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int l = 0, at = ptr[0], ln, an, lf, af;
    int4 d = load_desc(l, at);
    copy(d, 0);
    ln = l; an = at;
    advance(ln, an);
    int4 dn = load_desc(ln, an);
    lf = ln; af = an;
    if (lf < nlevels) advance(lf, af);
    double bn = d.x >= 0 ? B[(int64_t)d.x * 5 + m] : 0.0;
    for (int buf = 0; l < nlevels; buf ^= 1) {
        copy(dn, buf ^ 1);
        const int4 df = load_desc(lf, af);
        const double b0 = bn;
        bn = dn.x >= 0 ? B[(int64_t)dn.x * 5 + m] : 0.0;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();  // a row's copies and reads stay within its warp
        const GsStage &st = S.stage[buf];
        if (d.x >= 0) {
            const int nb = d.z - d.y, ns = min(nb, kGsBlocks);
            // values of X of the staged blocks: lane m component m
            double xv[kGsBlocks];
#pragma unroll
            for (int t = 0; t < kGsBlocks; t++)
                xv[t] = t < ns ? __ldcg(X + (int64_t)st.JA[q][t] * 5 + m) : 0.0;
#pragma unroll
            for (int t = 0; t < kGsBlocks; t++)
                if (t < ns) S.x[q][5 * t + m] = xv[t];
            const double xr = __ldcg(X + (int64_t)d.x * 5 + m);
            __syncwarp(group);
            double rhs = b0;
#pragma unroll 4
            for (int t = 0; t < ns; t++) {
                double tv = 0.0;
#pragma unroll
                for (int j = 0; j < 5; j++) tv = __dadd_rn(tv, __dmul_rn(st.A[q][t * 25 + m * 5 + j], S.x[q][5 * t + j]));
                rhs = __dsub_rn(rhs, tv);
            }
            for (int k = d.y + kGsBlocks; k < d.z; k++) {
                const double *a = A + (int64_t)k * 25 + m * 5, *x = X + (int64_t)JA[k] * 5;
                double tv = 0.0;
#pragma unroll
                for (int j = 0; j < 5; j++) tv = __dadd_rn(tv, __dmul_rn(a[j], __ldcg(x + j)));
                rhs = __dsub_rn(rhs, tv);
            }
            double s = 0.0;
#pragma unroll
            for (int j = 0; j < 5; j++) {
                const double v = __shfl_sync(group, rhs, 5 * g + j);
                s = __dadd_rn(s, __dmul_rn(v, v));
            }
            if (m == 0) rowrms[d.x] = s;
            const int dg = d.w - d.y;
            double tv = 0.0;
#pragma unroll
            for (int j = 0; j < 5; j++) {
                const double a = dg < kGsBlocks ? st.A[q][dg * 25 + m * 5 + j] : A[(int64_t)d.w * 25 + m * 5 + j];
                tv = __dadd_rn(tv, __dmul_rn(a, __shfl_sync(group, xr, 5 * g + j)));
            }
            rhs = __dadd_rn(rhs, tv);
            const double *lu = st.LU[q];
            double v[5], xo[5];
#pragma unroll
            for (int ii = 0; ii < 5; ii++) {
                v[ii] = __shfl_sync(group, rhs, 5 * g + ii);
#pragma unroll
                for (int jj = 0; jj < ii; jj++) v[ii] = __dsub_rn(v[ii], __dmul_rn(lu[ii * 5 + jj], v[jj]));
            }
            double mine = 0.0;
#pragma unroll
            for (int ii = 4; ii >= 0; ii--) {
                double y = v[ii];
#pragma unroll
                for (int jj = 4; jj > ii; jj--) y = __dsub_rn(y, __dmul_rn(lu[ii * 5 + jj], xo[jj]));
                xo[ii] = __ddiv_rn(y, lu[ii * 5 + ii]);
                if (m == ii) mine = xo[ii];
            }
            X[(int64_t)d.x * 5 + m] = mine;
        }
        __syncwarp();
        // every chunk of a level finishes before the next level starts
        if (ln != l) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        l = ln; at = an;
        d = dn;
        ln = lf; an = af;
        dn = df;
        if (lf < nlevels) advance(lf, af);
    }
}

// rms[it] = sqrt(sum / n) of sweep `it`, unless an earlier one stopped; stop
// {!= 0, sweeps done} (MC_Iterative_Jacobi.c:506)
__global__ void k_gs_check(const double *__restrict__ sum, int n, int it, double *__restrict__ rms, int *__restrict__ stop) {
    if (stop[0] != 0) return;
    const double r = sqrt(sum[0] / (double)n);
    rms[0] = r;
    stop[1] = it + 1;
    if (r < 100.0 * DBL_EPSILON) stop[0] = 1;
}

// Per-iteration reset: sum(area*lambda) = 0, extrema = (DBL_MAX, DBL_MIN)
// (Solver_Steady_Implicit.cpp:45-79).
// Eigenvalue extrema of a residual pass that a limiter fix may supersede:
// reset to the empty minimum / maximum, and merged into the call's extrema
// only when no node failed a check (gate = the fix counters).
__global__ void k_ext_reset(unsigned long long *__restrict__ e) {
    const int i = threadIdx.x;
    if (i < 6) e[i] = (i & 1) ? (unsigned long long)__double_as_longlong(DBL_MIN)
                              : (unsigned long long)__double_as_longlong(DBL_MAX);
}

__global__ void k_ext_merge(const int *__restrict__ gate, const unsigned long long *__restrict__ e,
                            unsigned long long *__restrict__ ext) {
    const int i = threadIdx.x;
    if (i >= 6 || gate[0] != 0 || gate[1] != 0) return;
    if (i & 1) atomicMax(&ext[i], e[i]);
    else atomicMin(&ext[i], e[i]);
}

__global__ void k_begin_iteration(int nnode, double *__restrict__ dt, unsigned long long *__restrict__ ext) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nnode) dt[i] = 0.0;
    if (i < 8) ext[i] = (i & 1) ? (unsigned long long)__double_as_longlong(DBL_MIN)
                                : (unsigned long long)__double_as_longlong(DBL_MAX);
}

__global__ void k_update(int nnode, int64_t ldq, double relax, const double *__restrict__ X, double *__restrict__ Q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nnode) return;
#pragma unroll
    for (int v = 0; v < 5; v++) Q[v * ldq + i] += relax * X[(int64_t)i * 5 + v];
}

__global__ void k_freestream(int n, int64_t ldq, Flow f, double *__restrict__ Q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool r = f.rup != 0;
    Q[i] = f.inf_rho;
    Q[ldq + i] = r ? f.inf_u : f.inf_rho * f.inf_u;
    Q[2 * ldq + i] = r ? f.inf_v : f.inf_rho * f.inf_v;
    Q[3 * ldq + i] = r ? f.inf_w : f.inf_rho * f.inf_w;
    Q[4 * ldq + i] = r ? f.inf_p : f.inf_rho * f.inf_et;
}

// ------------------------------------------------------------- host helpers

int reduce_sum_sq(cfd_ctx *c, const double *x, int64_t n, int64_t stride, int nvec, double *out_host) {
    const int nblk = 296, bs = 256;
    CFD_CUDA(c->red.alloc(std::max<size_t>(c->red.n, (size_t)nblk * 128)));
    CFD_CUDA(c->red_out.alloc(std::max<size_t>(c->red_out.n, 64)));
    k_sumsq_partial<<<nblk, bs, bs * sizeof(double), c->stream>>>(x, n, stride, nvec, c->red.p);
    CFD_LAUNCH_CHECK();
    k_sum_final<<<1, bs, bs * sizeof(double), c->stream>>>(c->red.p, nblk, nvec, c->red_out.p);
    CFD_LAUNCH_CHECK();
    CFD_CUDA(cudaMemcpyAsync(out_host, c->red_out.p, nvec * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    return CFD_OK;
}

int check_device_error(cfd_ctx *c) {
    int h = 0;
    CFD_CUDA(cudaMemcpyAsync(&h, c->err.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    if (h) {
        CFD_CUDA(cudaMemsetAsync(c->err.p, 0, sizeof(int), c->stream));
        set_error("device reported numerical failure (flags 0x%x)", h);
        return CFD_ERR_NUMERIC;
    }
    return CFD_OK;
}

int require_edge_graph(cfd_ctx *c, const char *who) {
    if (c->graph_is_edges) return CFD_OK;
    set_error("%s: the rows of the mesh's node graph (n2n) are not the neighbours that its edges give", who);
    return CFD_ERR_MESH;
}

// Far-field state with Mach ramping (ComputeFarFieldCondition,
// Euler3D/src/Material.cpp:185-210) under the generic non-dimensionalisation
// (Material.cpp:119-124: R = 1/gamma, rho = 1, T = gamma, p = 1).
static void compute_flow(cfd_ctx *c, int iteration) {
    const cfd_params &p = c->params;
    Flow &f = c->flow;
    f.gamma = p.gamma;
    f.gm1 = p.gamma - 1.0;
    f.inv_gm1 = 1.0 / (p.gamma - 1.0);
    double mach;
    if (p.mach_ramp > 1 && p.mach > p.mach_min) {
        mach = iteration < p.mach_ramp
                   ? p.mach_min + (p.mach - p.mach_min) * ((double)iteration / (double)(p.mach_ramp - 1))
                   : p.mach;
    } else {
        mach = p.mach;
    }
    const double R = 1.0 / p.gamma, rho = 1.0, T = p.gamma, pr = R * rho * T;
    const double alpha = p.alpha_deg * M_PI / 180.0, beta = p.beta_deg * M_PI / 180.0;
    f.pinf = p.pinf;
    f.gpinf = p.gamma * p.pinf;
    f.inf_mach = mach;
    f.inf_rho = rho;
    f.inf_p = pr;
    // stiffened gas: c^2 = gamma (p + pinf) / rho (the ideal-gas expression when pinf = 0)
    f.inf_c = p.pinf != 0.0 ? sqrt(p.gamma * (pr + p.pinf) / rho) : sqrt(p.gamma * R * T);
    f.inf_u = mach * f.inf_c * cos(alpha) * cos(beta);
    f.inf_v = mach * f.inf_c * sin(alpha);
    f.inf_w = mach * f.inf_c * sin(beta) * cos(alpha);
    f.inf_et = (pr + f.gpinf) / ((p.gamma - 1.0) * rho) + 0.5 * (f.inf_u * f.inf_u + f.inf_v * f.inf_v + f.inf_w * f.inf_w);
    f.outflow_p = 0.935 * pr;  // Material.cpp:171
    f.frac = p.limiter_order == 1 ? 0.5 : 0.0;
    f.venkat_eps_k3 = pow(p.venkat_k, 3.0);
    f.flux = p.flux_scheme;
    f.lmfix = p.flux_scheme == CFD_FLUX_ROE_LMFIX ? 1 : 0;
    f.pc_method = p.precond_method;
    f.pc_type = p.precond_type;
    f.pc_mach = p.precond_mach;
    f.pc_outflow_p = p.outflow_pressure != 0.0 ? p.outflow_pressure : pr;
    f.rup = p.variables == CFD_VARS_RUP ? 1 : 0;
    f.order = p.order;
    f.limiter = p.limiter;
    f.limiter_smooth = p.limiter_smooth;
    f.entropy_fix = p.entropy_fix;
    f.zpg_iteration = p.zpg_iteration;
    f.iteration = iteration;
    // CFL ramp (Time_Step.cpp:27-34)
    if (p.cfl_ramp > 1 && p.cfl_max > p.cfl_min)
        c->cfl = iteration < p.cfl_ramp
                     ? p.cfl_min + (p.cfl_max - p.cfl_min) * ((double)iteration / (double)(p.cfl_ramp - 1))
                     : p.cfl_max;
    else
        c->cfl = p.cfl_max;
}


template <int FLUX, bool SECOND>
static int launch_residual(cfd_ctx *c, int add_time, bool check_roe, bool check_pc, const int *gate,
                           unsigned long long *ext) {
    if (patch_kernel(c)) {
        const size_t smem = patch_smem_bytes(c->patch_nlocmax, SECOND);
        if (smem > 48 * 1024) {
            int smax = 0;
            CFD_CUDA(allow_max_dynamic_smem(k_residual_patch<FLUX, SECOND>, c->device, &smax));
            if (smem > (size_t)smax) {
                set_error("residual patch kernel: %zu bytes of shared memory needed, %d available", smem, smax);
                return CFD_ERR_RANGE;
            }
        }
        k_residual_patch<FLUX, SECOND><<<c->npatch, PATCH_CHUNK, smem, c->stream>>>(
            c->nnode, c->ldq, c->Q.p, c->grad.p, c->phi.p, c->xyz.p, c->pe_ptr.p, c->pe_loc.p, c->pe_geo.p,
            c->ph_ptr.p, c->halo.p, c->inc_ptr.p, c->inc.p, c->n2b_ptr.p, c->n2b.p, c->bedge_nodes.p, c->bedge_geo.p,
            c->flow, add_time, c->patch_nlocmax, check_roe ? 1 : 0, c->roeflag.p, c->fixcount.p, gate, c->res.p,
            c->resd.p, c->dt.p, ext);
    } else {
        const bool k0 = SECOND && c->flow.frac == 0.0;
        const int checks = (check_roe ? 1 : 0) | (check_pc ? 2 : 0);
        // limited gradients phi * grad formed with these limiters by the fused
        // Green-Gauss + limiter pass (first pass only: a gated re-evaluation
        // follows limiter fixes, which change phi)
        const bool lgk = k0 && !gate && c->lgrad_valid && c->params.limiter != CFD_LIMITER_NONE;
        const bool rup = c->flow.rup != 0;
#define GATHER_LAUNCH_ARGS                                                                                          \
    c->nnode, c->ldq, c->Q.p, c->grad.p, c->phi.p, c->xyz.p, c->sell_ptr.p, c->sell_nbr.p, c->sell_geo.p, c->deg.p, \
        c->flow, add_time, checks, c->roeflag.p, c->fixcount.p, c->res.p, c->resd.p, c->dt.p, c->lgrad.p
        const int key = c->flow.rup ? -1 : batch_key(FLUX, SECOND, k0, lgk);
        if (!gate && c->batcher && key >= 0) {
            // the serving loop fuses this launch with other requests' (same per-node code)
            GatherJob job{c->nnode, c->ldq, c->Q.p, c->grad.p, c->phi.p, c->xyz.p, c->sell_ptr.p, c->sell_nbr.p,
                          c->sell_geo.p, c->deg.p, c->flow, add_time, checks, c->roeflag.p, c->fixcount.p,
                          c->res.p, c->resd.p, c->dt.p, lgk ? c->lgrad.p : nullptr, ext, 0};
            const int st = c->batch_submit(c->batcher, c, key, &job);
            if (st) return st;
        } else if (lgk) {
            auto kern = rup ? k_residual_gather<FLUX, SECOND, SECOND, true, true>
                            : k_residual_gather<FLUX, SECOND, SECOND, true, false>;
            kern<<<grid_for(c->nnode, 128), 128, 0, c->stream>>>(GATHER_LAUNCH_ARGS, ext, 0, c->nnode);
        } else if (gate) {
            auto kern = rup ? (k0 ? k_residual_gather_rerun<FLUX, SECOND, SECOND, true>
                                  : k_residual_gather_rerun<FLUX, SECOND, false, true>)
                            : (k0 ? k_residual_gather_rerun<FLUX, SECOND, SECOND, false>
                                  : k_residual_gather_rerun<FLUX, SECOND, false, false>);
            const int grid = std::min(grid_for(c->nnode, 128), 3 * c->nsm);
            kern<<<grid, 128, 0, c->stream>>>(GATHER_LAUNCH_ARGS, gate, ext);
        } else {
            auto kern = rup ? (k0 ? k_residual_gather<FLUX, SECOND, SECOND, false, true>
                                  : k_residual_gather<FLUX, SECOND, false, false, true>)
                            : (k0 ? k_residual_gather<FLUX, SECOND, SECOND, false, false>
                                  : k_residual_gather<FLUX, SECOND, false, false, false>);
            kern<<<grid_for(c->nnode, 128), 128, 0, c->stream>>>(GATHER_LAUNCH_ARGS, ext, 0, c->nnode);
        }
#undef GATHER_LAUNCH_ARGS
        if (c->nbnode > 0) {
            CFD_LAUNCH_CHECK();
            k_residual_bnd<FLUX><<<grid_for(c->nbnode, 128), 128, 0, c->stream>>>(
                c->nbnode, c->bnode.p, c->nnode, c->ldq, c->Q.p, c->n2b_ptr.p, c->n2b.p, c->bedge_nodes.p,
                c->bedge_geo.p, c->flow, add_time, gate, c->res.p, c->resd.p, c->dt.p, ext);
        }
    }
    CFD_LAUNCH_CHECK();
    return CFD_OK;
}

// ---- block LU-SGS (MC_Iterative_Block_LUSGS_CRS, MATH/src/MC_Iterative_Jacobi.c:539-717)
// Pivoted Gaussian LU of each diagonal block (GaussainLUDecompose,
// MATH/src/LinearAlgebra.c:117-150, partial pivoting by row permutation P,
// first largest |entry| wins).  The reference factors the block again in
// every sweep; the factors depend only on the block, so they are formed once
// per call.  Explicitly rounded intrinsics keep every operation as the
// reference's scalar code rounds it.
__global__ void k_lu_pivot(int nnode, const double *__restrict__ A, const int *__restrict__ IAU,
                           double *__restrict__ LU, int *__restrict__ piv) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nnode) return;
    double a[25];
    int P[5] = {0, 1, 2, 3, 4};
    const double *src = A + (int64_t)IAU[r] * 25;
#pragma unroll
    for (int k = 0; k < 25; k++) a[k] = src[k];
    for (int c = 0; c < 5; c++) {
        double pmax = a[P[c] * 5 + c];
        int pi = c;
        for (int i = c + 1; i < 5; i++)
            if (fabs(a[P[i] * 5 + c]) > fabs(pmax)) { pmax = a[P[i] * 5 + c]; pi = i; }
        if (pi != c) { const int t = P[c]; P[c] = P[pi]; P[pi] = t; }
        for (int i = c + 1; i < 5; i++) a[P[i] * 5 + c] = __ddiv_rn(a[P[i] * 5 + c], a[P[c] * 5 + c]);
        for (int i = c + 1; i < 5; i++)
            for (int j = c + 1; j < 5; j++)
                a[P[i] * 5 + j] = __dsub_rn(a[P[i] * 5 + j], __dmul_rn(a[P[i] * 5 + c], a[P[c] * 5 + j]));
    }
    double *dst = LU + (int64_t)r * 25;
#pragma unroll
    for (int k = 0; k < 25; k++) dst[k] = a[k];
#pragma unroll
    for (int k = 0; k < 5; k++) piv[(int64_t)r * 5 + k] = P[k];
}

// X_i = mean of B_i's five components (MC_Iterative_Jacobi.c:574-581).
__global__ void k_lusgs_init(int nnode, const double *__restrict__ B, double *__restrict__ X) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nnode) return;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 5; j++) s = __dadd_rn(s, B[(int64_t)r * 5 + j]);
    s = __ddiv_rn(s, 5.0);
#pragma unroll
    for (int j = 0; j < 5; j++) X[(int64_t)r * 5 + j] = s;
}

// One level of a forward or backward sweep: rhs = B_i - sum_{k != diag} A_k X_JA[k]
// in CRS order, then the pivoted substitutions (Solve_PivotForwardSubstitution,
// Solve_PivotBackSubstitution, LinearAlgebra.c:20-43).
__global__ void __launch_bounds__(128) k_lusgs_level(int nrows, const int *__restrict__ rows,
                                                    const int *__restrict__ IA, const int *__restrict__ JA,
                                                    const int *__restrict__ IAU, const double *__restrict__ A,
                                                    const double *__restrict__ B, const double *__restrict__ LU,
                                                    const int *__restrict__ piv, double *__restrict__ X) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nrows) return;
    const int r = rows[t];
    double rhs[5];
#pragma unroll
    for (int m = 0; m < 5; m++) rhs[m] = B[(int64_t)r * 5 + m];
    const int dg = IAU[r];
    for (int k = IA[r]; k < IA[r + 1]; k++) {
        if (k == dg) continue;
        const double *a = A + (int64_t)k * 25;
        const double *x = X + (int64_t)JA[k] * 5;
        double xv[5];
#pragma unroll
        for (int m = 0; m < 5; m++) xv[m] = x[m];
#pragma unroll
        for (int ii = 0; ii < 5; ii++) {
            double tv = 0.0;
#pragma unroll
            for (int jj = 0; jj < 5; jj++) tv = __dadd_rn(tv, __dmul_rn(a[ii * 5 + jj], xv[jj]));
            rhs[ii] = __dsub_rn(rhs[ii], tv);
        }
    }
    const double *lu = LU + (int64_t)r * 25;
    int P[5];
#pragma unroll
    for (int k = 0; k < 5; k++) P[k] = piv[(int64_t)r * 5 + k];
    double y[5], xo[5];
    y[0] = rhs[P[0]];
    for (int i = 1; i < 5; i++) {
        double v = rhs[P[i]];
        for (int j = 0; j < i; j++) v = __dsub_rn(v, __dmul_rn(y[j], lu[P[i] * 5 + j]));
        y[i] = v;
    }
    xo[4] = __ddiv_rn(y[4], lu[P[4] * 5 + 4]);
    for (int i = 3; i >= 0; i--) {
        double v = y[i];
        for (int j = 4; j > i; j--) v = __dsub_rn(v, __dmul_rn(xo[j], lu[P[i] * 5 + j]));
        xo[i] = __ddiv_rn(v, lu[P[i] * 5 + i]);
    }
#pragma unroll
    for (int m = 0; m < 5; m++) X[(int64_t)r * 5 + m] = xo[m];
}

template <int FLUX, bool SECOND>
static int residual_with_fix(cfd_ctx *c, int add_time) {
    // Second order with a limiter: the limiter's pressure fixes are decided by
    // the residual's own reconstruction (the same face states) and applied,
    // followed by a gated re-evaluation, only when some node failed a check;
    // nothing is read back to the host.  The patch kernel carries only the
    // Roe check, so a pending reconstructed-pressure correction runs first.
    if (!SECOND) return launch_residual<FLUX, SECOND>(c, add_time, false, false, nullptr, c->ext.p);
    if (c->pc_fix_pending && patch_kernel(c)) {
        const bool roe = c->roe_fix_pending;
        c->roe_fix_pending = false;
        int st = limiter_fix_standalone(c);
        c->roe_fix_pending = roe;
        if (st) return st;
    }
    const bool check_roe = is_roe_flux(FLUX) && c->roe_fix_pending;
    const bool check_pc = c->pc_fix_pending;
    if (!(check_roe || check_pc)) return launch_residual<FLUX, SECOND>(c, add_time, false, false, nullptr, c->ext.p);
    // The first pass's eigenvalue extrema go to a scratch copy: they count only
    // when no node fails a check (Compute_Residual sees the fixed limiters
    // alone); otherwise the gated re-evaluation records them.
    if (!c->ext_scratch.p) CFD_CUDA(c->ext_scratch.alloc(8));
    k_ext_reset<<<1, 32, 0, c->stream>>>(c->ext_scratch.p);
    int st = launch_residual<FLUX, SECOND>(c, add_time, check_roe, check_pc, nullptr, c->ext_scratch.p);
    if (st) return st;
    const bool redo_roe = check_roe && check_pc;
    if (redo_roe) CFD_CUDA(c->work.alloc(std::max<size_t>(c->work.n, (size_t)5 * c->nnode)));
    k_limiter_fix_apply<<<std::min(grid_for(c->nnode, 256), 4 * c->nsm), 256, 0, c->stream>>>(
        c->nnode, c->fixcount.p, c->roeflag.p, redo_roe ? 1 : 0, c->phi.p, c->work.p);
    CFD_LAUNCH_CHECK();
    c->lgrad_valid = false;  // the fixes may have changed phi
    if (redo_roe) {
        st = launch_roe_pressure_fix(c, c->fixcount.p);
        if (st) return st;
    }
    c->roe_fix_pending = false;
    c->pc_fix_pending = false;
    k_ext_merge<<<1, 32, 0, c->stream>>>(c->fixcount.p, c->ext_scratch.p, c->ext.p);
    CFD_LAUNCH_CHECK();
    return launch_residual<FLUX, SECOND>(c, add_time, false, false, c->fixcount.p, c->ext.p);
}

static Levels *build_levels(const std::vector<int> &IA, const std::vector<int> &JA, int n, bool forward,
                            Levels &L, cudaStream_t s, int &err) {
    std::vector<int> lev(n, 0);
    int maxl = 0;
    if (forward) {
        for (int i = 0; i < n; i++) {
            int l = 0;
            for (int k = IA[i]; k < IA[i + 1]; k++)
                if (JA[k] < i) l = std::max(l, lev[JA[k]] + 1);
            lev[i] = l;
            maxl = std::max(maxl, l);
        }
    } else {
        for (int i = n - 1; i >= 0; i--) {
            int l = 0;
            for (int k = IA[i]; k < IA[i + 1]; k++)
                if (JA[k] > i) l = std::max(l, lev[JA[k]] + 1);
            lev[i] = l;
            maxl = std::max(maxl, l);
        }
    }
    const int nl = n ? maxl + 1 : 0;
    L.ptr.assign(nl + 1, 0);
    for (int i = 0; i < n; i++) L.ptr[lev[i] + 1]++;
    for (int l = 0; l < nl; l++) L.ptr[l + 1] += L.ptr[l];
    std::vector<int> rows(n), fill(L.ptr.begin(), L.ptr.end() - 1);
    // rows of a level keep ascending order (coalesced loads)
    for (int i = 0; i < n; i++) rows[fill[lev[i]]++] = i;
    L.max_width = 0;
    for (int l = 0; l < nl; l++) L.max_width = std::max(L.max_width, L.ptr[l + 1] - L.ptr[l]);
    L.desc_built = false;
    err = L.rows.upload(rows.data(), rows.size(), s) == cudaSuccess ? 0 : 1;
    return &L;
}

}  // namespace cfd

using namespace cfd;

// ====================================================================== C ABI
// ---------------------------------------------------- pipelined residual step
// cfd_residual_step with a host state in and both residuals out overlaps its
// copies with its kernels.  The nodes are cut into K chunks of >= 128K nodes
// (multiples of 128).  The state goes up chunk by chunk on a copy stream;
// chunk g's boundary ghosts and its Green-Gauss + limiter pass start when the
// chunks holding its neighbours have arrived, chunk c's residual when the
// gradients of the chunks holding its neighbours are formed, and its two
// residual rows go down on a second copy stream while the next chunks are
// computed.  Every kernel computes each node as the whole-mesh launch does,
// and the limiter-fix passes run after the last chunk as in residual_with_fix;
// when they changed some residual (a node failed a check), the residuals are
// copied again whole after them.  Used for second order with Green-Gauss
// gradients and a limiter on the gather kernel and a stream of the caller's;
// otherwise the step runs its calls one after the other.
static bool pipe_eligible(const cfd_ctx *c) {
    const cfd_params &p = c->params;
    return c->stream && !c->batcher && !patch_kernel(c) && p.order == CFD_ORDER_SECOND &&
           p.gradient == CFD_GRAD_GG && p.limiter != CFD_LIMITER_NONE && c->pipe.request != 0 &&
           c->pipe.request != 1;
}

static int pipe_build(cfd_ctx *c) {
    StepPipe &P = c->pipe;
    if (P.built) return CFD_OK;
    const int n = c->nnode;
    const int K = P.request > 1 ? std::min(P.request, n / 256) : std::min(16, n / 131072);
    P.K = K;
    P.built = true;
    if (K <= 1) return CFD_OK;
    P.lo.assign(K + 1, n);
    for (int k = 0; k < K; k++) P.lo[k] = (int)(((int64_t)n * k / K) / 128 * 128);
    // the chunk holding the farthest neighbour of each chunk's nodes (the
    // graph's reach grows along a reverse Cuthill-McKee order)
    auto chunk_of = [&](int node) { return (int)(std::upper_bound(P.lo.begin(), P.lo.end() - 1, node) - P.lo.begin()) - 1; };
    P.dep.resize(K);
    for (int k = 0; k < K; k++) {
        int far = P.lo[k + 1] - 1;
        for (int i = P.lo[k]; i < P.lo[k + 1]; i++)
            for (int e = c->h_IA[i]; e < c->h_IA[i + 1]; e++) far = std::max(far, c->h_JA[e]);
        P.dep[k] = std::max(k, chunk_of(far));
    }
    // a later chunk's neighbours lie no nearer: keep the dependencies monotone
    for (int k = 1; k < K; k++) P.dep[k] = std::max(P.dep[k], P.dep[k - 1]);
    // boundary edges by physical node, nodes with boundary edges
    std::vector<int2> bn(c->nbedge);
    std::vector<int> bnode(c->nbnode);
    if (c->nbedge)
        CFD_CUDA(cudaMemcpyAsync(bn.data(), c->bedge_nodes.p, sizeof(int2) * c->nbedge, cudaMemcpyDeviceToHost, c->stream));
    if (c->nbnode)
        CFD_CUDA(cudaMemcpyAsync(bnode.data(), c->bnode.p, sizeof(int) * c->nbnode, cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    std::vector<int> order(c->nbedge);
    for (int b = 0; b < c->nbedge; b++) order[b] = b;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return bn[a].x < bn[b].x; });
    P.bc_lo.assign(K + 1, c->nbedge);
    P.bn_lo.assign(K + 1, c->nbnode);
    for (int k = 0, b = 0; k < K; k++) {
        while (b < c->nbedge && bn[order[b]].x < P.lo[k]) b++;
        P.bc_lo[k] = b;
        P.bn_lo[k] = (int)(std::lower_bound(bnode.begin(), bnode.end(), P.lo[k]) - bnode.begin());
    }
    CFD_CUDA(P.bc_list.alloc(std::max(1, c->nbedge)));
    if (c->nbedge)
        CFD_CUDA(cudaMemcpyAsync(P.bc_list.p, order.data(), sizeof(int) * c->nbedge, cudaMemcpyHostToDevice, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    if (!P.s_in) CFD_CUDA(cudaStreamCreateWithFlags(&P.s_in, cudaStreamNonBlocking));
    if (!P.s_out) CFD_CUDA(cudaStreamCreateWithFlags(&P.s_out, cudaStreamNonBlocking));
    if (!P.ev_start) CFD_CUDA(cudaEventCreateWithFlags(&P.ev_start, cudaEventDisableTiming));
    if (!P.ev_ghost) CFD_CUDA(cudaEventCreateWithFlags(&P.ev_ghost, cudaEventDisableTiming));
    P.release_events();
    P.ev_q.assign(K, nullptr);
    P.ev_r.assign(K, nullptr);
    for (int k = 0; k < K; k++) {
        CFD_CUDA(cudaEventCreateWithFlags(&P.ev_q[k], cudaEventDisableTiming));
        CFD_CUDA(cudaEventCreateWithFlags(&P.ev_r[k], cudaEventDisableTiming));
    }
    if (!P.h_flags) CFD_CUDA(cudaMallocHost(&P.h_flags, 4 * sizeof(int)));
    return CFD_OK;
}

template <int FLUX>
static int residual_step_pipelined_flux(cfd_ctx *c, int iteration, const double *Q_host, double *conv, double *diss) {
    StepPipe &P = c->pipe;
    const int n = c->nnode, K = P.K;
    const int64_t nt = (int64_t)n + c->nghost;
    const size_t dq = (size_t)c->ldq * sizeof(double), hq = (size_t)nt * sizeof(double), hr = (size_t)n * sizeof(double);
    // cfd_set_state
    c->phi_next_valid = false;
    c->lgrad_valid = c->lgrad_pending = false;
    CFD_CUDA(cudaEventRecord(P.ev_start, c->stream));
    CFD_CUDA(cudaStreamWaitEvent(P.s_in, P.ev_start, 0));
    CFD_CUDA(cudaStreamWaitEvent(P.s_out, P.ev_start, 0));
    if (c->nghost)
        CFD_CUDA(cudaMemcpy2DAsync(c->Q.p + n, dq, Q_host + n, hq, (size_t)c->nghost * sizeof(double), 5,
                                   cudaMemcpyHostToDevice, P.s_in));
    CFD_CUDA(cudaEventRecord(P.ev_ghost, P.s_in));
    for (int k = 0; k < K; k++) {
        const int lo = P.lo[k], hi = P.lo[k + 1];
        CFD_CUDA(cudaMemcpy2DAsync(c->Q.p + lo, dq, Q_host + lo, hq, (size_t)(hi - lo) * sizeof(double), 5,
                                   cudaMemcpyHostToDevice, P.s_in));
        CFD_CUDA(cudaEventRecord(P.ev_q[k], P.s_in));
    }
    // cfd_begin_iteration (no state read), then the buffers and flags that
    // cfd_gradient + cfd_limiter leave for the residual: the fused pass writes
    // the limiters straight into phi
    int st = cfd_begin_iteration(c, iteration);
    if (st) return st;
    c->flow.iteration = iteration;
    const bool kappa0 = c->flow.frac == 0.0;
    CFD_CUDA(c->grad.alloc((size_t)15 * n));
    CFD_CUDA(c->phi_next.alloc((size_t)5 * n));
    CFD_CUDA(c->phi.alloc((size_t)5 * n));
    if (kappa0) CFD_CUDA(c->lgrad.alloc((size_t)15 * n));
    c->has_grad = true;
    c->phi_next_valid = false;
    c->lgrad_valid = kappa0;
    c->pc_fix_pending = true;
    c->roe_fix_pending = is_roe_flux(FLUX);
    CFD_CUDA(cudaMemsetAsync(c->fixcount.p, 0, 2 * sizeof(int), c->stream));
    // residual_with_fix: the first pass's extrema go to the scratch copy
    const bool check_roe = is_roe_flux(FLUX);
    const int checks = (check_roe ? 1 : 0) | 2;
    if (!c->ext_scratch.p) CFD_CUDA(c->ext_scratch.alloc(8));
    k_ext_reset<<<1, 32, 0, c->stream>>>(c->ext_scratch.p);
    CFD_LAUNCH_CHECK();
    CFD_CUDA(cudaStreamWaitEvent(c->stream, P.ev_ghost, 0));
    int g_done = -1;
    for (int k = 0; k < K; k++) {
        while (g_done < P.dep[k]) {
            const int g = ++g_done;
            CFD_CUDA(cudaStreamWaitEvent(c->stream, P.ev_q[P.dep[g]], 0));
            const int nb = P.bc_lo[g + 1] - P.bc_lo[g];
            if (nb > 0) {
                k_apply_bc<<<grid_for(nb, 128), 128, 0, c->stream>>>(nb, c->ldq, c->Q.p, c->bedge_nodes.p,
                                                                      c->bedge_geo.p, c->bedge_type.p, c->flow,
                                                                      c->err.p, P.bc_list.p + P.bc_lo[g]);
                CFD_LAUNCH_CHECK();
            }
            if ((st = gg_limiter_range(c, c->phi.p, P.lo[g], P.lo[g + 1]))) return st;
        }
        const int lo = P.lo[k], hi = P.lo[k + 1];
        auto kern = c->flow.rup ? (kappa0 ? k_residual_gather<FLUX, true, true, true, true>
                                          : k_residual_gather<FLUX, true, false, false, true>)
                                : (kappa0 ? k_residual_gather<FLUX, true, true, true, false>
                                          : k_residual_gather<FLUX, true, false, false, false>);
        kern<<<grid_for(hi - lo, 128), 128, 0, c->stream>>>(
            n, c->ldq, c->Q.p, c->grad.p, c->phi.p, c->xyz.p, c->sell_ptr.p, c->sell_nbr.p, c->sell_geo.p, c->deg.p,
            c->flow, 1, checks, c->roeflag.p, c->fixcount.p, c->res.p, c->resd.p, c->dt.p, c->lgrad.p,
            c->ext_scratch.p, lo, hi);
        CFD_LAUNCH_CHECK();
        const int nbn = P.bn_lo[k + 1] - P.bn_lo[k];
        if (nbn > 0) {
            k_residual_bnd<FLUX><<<grid_for(nbn, 128), 128, 0, c->stream>>>(
                nbn, c->bnode.p + P.bn_lo[k], n, c->ldq, c->Q.p, c->n2b_ptr.p, c->n2b.p, c->bedge_nodes.p,
                c->bedge_geo.p, c->flow, 1, nullptr, c->res.p, c->resd.p, c->dt.p, c->ext_scratch.p);
            CFD_LAUNCH_CHECK();
        }
        CFD_CUDA(cudaEventRecord(P.ev_r[k], c->stream));
        CFD_CUDA(cudaStreamWaitEvent(P.s_out, P.ev_r[k], 0));
        CFD_CUDA(cudaMemcpy2DAsync(conv + lo, hr, c->res.p + lo, hr, (size_t)(hi - lo) * sizeof(double), 5,
                                   cudaMemcpyDeviceToHost, P.s_out));
        CFD_CUDA(cudaMemcpy2DAsync(diss + lo, hr, c->resd.p + lo, hr, (size_t)(hi - lo) * sizeof(double), 5,
                                   cudaMemcpyDeviceToHost, P.s_out));
    }
    // residual_with_fix after its first pass: the fixes, then the gated re-evaluation
    const bool redo_roe = check_roe;
    if (redo_roe) CFD_CUDA(c->work.alloc(std::max<size_t>(c->work.n, (size_t)5 * n)));
    k_limiter_fix_apply<<<std::min(grid_for(n, 256), 4 * c->nsm), 256, 0, c->stream>>>(
        n, c->fixcount.p, c->roeflag.p, redo_roe ? 1 : 0, c->phi.p, c->work.p);
    CFD_LAUNCH_CHECK();
    c->lgrad_valid = false;
    if (redo_roe && (st = launch_roe_pressure_fix(c, c->fixcount.p))) return st;
    c->roe_fix_pending = false;
    c->pc_fix_pending = false;
    k_ext_merge<<<1, 32, 0, c->stream>>>(c->fixcount.p, c->ext_scratch.p, c->ext.p);
    CFD_LAUNCH_CHECK();
    if ((st = launch_residual<FLUX, true>(c, 1, false, false, c->fixcount.p, c->ext.p))) return st;
    if ((st = cfd_deltat(c, iteration))) return st;
    CFD_CUDA(cudaMemcpyAsync(P.h_flags, c->fixcount.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(cudaMemcpyAsync(P.h_flags + 2, c->err.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    CFD_CUDA(stream_wait(P.s_out));
    if (P.h_flags[0] || P.h_flags[1]) {
        // a limiter fix re-evaluated the residual after some chunks went down
        CFD_CUDA(cudaMemcpyAsync(conv, c->res.p, hr * 5, cudaMemcpyDeviceToHost, c->stream));
        CFD_CUDA(cudaMemcpyAsync(diss, c->resd.p, hr * 5, cudaMemcpyDeviceToHost, c->stream));
        CFD_CUDA(stream_wait(c->stream));
    }
    if (P.h_flags[2]) {
        CFD_CUDA(cudaMemsetAsync(c->err.p, 0, sizeof(int), c->stream));
        set_error("device reported numerical failure (flags 0x%x)", P.h_flags[2]);
        return CFD_ERR_NUMERIC;
    }
    return CFD_OK;
}

static int residual_step_pipelined_any(cfd_ctx *c, int iteration, const double *Q_host, double *conv, double *diss) {
    switch (c->params.flux_scheme) {
        case CFD_FLUX_ROE: return residual_step_pipelined_flux<CFD_FLUX_ROE>(c, iteration, Q_host, conv, diss);
        case CFD_FLUX_HLLC: return residual_step_pipelined_flux<CFD_FLUX_HLLC>(c, iteration, Q_host, conv, diss);
        case CFD_FLUX_AUSM: return residual_step_pipelined_flux<CFD_FLUX_AUSM>(c, iteration, Q_host, conv, diss);
        case CFD_FLUX_ROE_LMFIX:
            return residual_step_pipelined_flux<CFD_FLUX_ROE_LMFIX>(c, iteration, Q_host, conv, diss);
        case CFD_FLUX_ROE_PRECOND:
            return residual_step_pipelined_flux<CFD_FLUX_ROE_PRECOND>(c, iteration, Q_host, conv, diss);
        case CFD_FLUX_ROE_THORNBER:
            return residual_step_pipelined_flux<CFD_FLUX_ROE_THORNBER>(c, iteration, Q_host, conv, diss);
        case CFD_FLUX_VANLEER: return residual_step_pipelined_flux<CFD_FLUX_VANLEER>(c, iteration, Q_host, conv, diss);
        default: set_error("cfd_residual_step: bad flux scheme"); return CFD_ERR_ARG;
    }
}

// The step's copies read and write the caller's host buffers: whatever path
// the step leaves by, its copy streams have finished before it returns.
static int residual_step_pipelined(cfd_ctx *c, int iteration, const double *Q_host, double *conv, double *diss) {
    const int st = residual_step_pipelined_any(c, iteration, Q_host, conv, diss);
    if (st) {
        cudaStreamSynchronize(c->pipe.s_in);
        cudaStreamSynchronize(c->pipe.s_out);
        cudaStreamSynchronize(c->stream);
    }
    return st;
}

extern "C" {

int cfd_abi_version(void) { return CFD_ABI_VERSION; }
const char *cfd_last_error(void) { return cfd::g_err; }

void cfd_params_default(cfd_params *p) {
    if (!p) return;
    std::memset(p, 0, sizeof(*p));
    p->flux_scheme = CFD_FLUX_ROE;
    p->order = CFD_ORDER_FIRST;
    p->limiter = CFD_LIMITER_NONE;
    p->limiter_order = 0;
    p->limiter_smooth = 0;
    p->gradient = CFD_GRAD_LSQ;
    p->ls_weight = 0;
    p->entropy_fix = 0;
    p->global_time = 0;
    p->cfl_ramp = 0;
    p->mach_ramp = 0;
    p->zpg_iteration = 0;
    p->gamma = 1.4;
    p->mach = 0.5;
    p->mach_min = 0.5;
    p->alpha_deg = 2.0;
    p->beta_deg = 0.0;
    p->cfl_min = 10.0;
    p->cfl_max = 10.0;
    p->venkat_k = 5.0;
}

int cfd_create(int device, cfd_ctx **out) {
    if (!out) { set_error("cfd_create: out is NULL"); return CFD_ERR_ARG; }
    *out = nullptr;
    int ndev = 0;
    CFD_CUDA(cudaGetDeviceCount(&ndev));
    if (device < 0 || device >= ndev) { set_error("cfd_create: device %d of %d", device, ndev); return CFD_ERR_ARG; }
    CFD_CUDA(cudaSetDevice(device));
    int nsm = 0;
    CFD_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
    cfd_ctx *c = new cfd_ctx();
    c->device = device;
    c->nsm = nsm;
    if (g_alloc_async) c->stream = g_alloc_stream;  // serving worker: its own stream from the start
    cfd_params_default(&c->params);
    if (c->err.alloc(1) != cudaSuccess || c->ext.alloc(8) != cudaSuccess) {
        delete c;
        set_error("cfd_create: device allocation failed");
        return CFD_ERR_CUDA;
    }
    if (g_alloc_async) cudaMemsetAsync(c->err.p, 0, sizeof(int), c->stream);
    else cudaMemset(c->err.p, 0, sizeof(int));
    compute_flow(c, 0);
    *out = c;
    return CFD_OK;
}

int cfd_destroy(cfd_ctx *c) {
    if (!c) return CFD_OK;
    cudaSetDevice(c->device);
    stream_wait(c->stream);
    delete c;
    return CFD_OK;
}

int cfd_set_stream(cfd_ctx *c, void *stream) {
    if (!c) return CFD_ERR_ARG;
    c->stream = (cudaStream_t)stream;
    return CFD_OK;
}

static int build_patch_layout(cfd_ctx *c);

int cfd_set_params(cfd_ctx *c, const cfd_params *p) {
    if (!c || !p) { set_error("cfd_set_params: NULL"); return CFD_ERR_ARG; }
    c->phi_next_valid = false;
    c->lgrad_valid = c->lgrad_pending = false;
    if (p->flux_scheme < CFD_FLUX_ROE || p->flux_scheme > CFD_FLUX_VANLEER) {
        set_error("cfd_set_params: invalid flux scheme %d", p->flux_scheme);
        return CFD_ERR_ARG;
    }
    if (!(p->gamma > 1.0)) { set_error("cfd_set_params: gamma must be > 1"); return CFD_ERR_ARG; }
    if (p->flux_scheme == CFD_FLUX_ROE_PRECOND) {
        const int m = p->precond_method, t = p->precond_type;
        if ((m != CFD_PRECOND_BTW && m != CFD_PRECOND_ERIKSSON && m != CFD_PRECOND_TURKEL) ||
            (t != CFD_PRECOND_LOCAL && t != CFD_PRECOND_GLOBAL && t != CFD_PRECOND_URLOCAL) ||
            (t != CFD_PRECOND_URLOCAL && !(p->precond_mach > 0.0))) {
            set_error("cfd_set_params: preconditioned Roe needs precond_method BTW/ERIKSSON/TURKEL, "
                      "precond_type LOCAL/GLOBAL/URLOCAL and precond_mach > 0");
            return CFD_ERR_ARG;
        }
    }
    if (p->flux_scheme == CFD_FLUX_VANLEER && p->pinf != 0.0) {
        set_error("cfd_set_params: the Van Leer splitting is written for the ideal gas (pinf = 0)");
        return CFD_ERR_ARG;
    }
    if (!(p->pinf >= 0.0 && p->pinf < 1.0e300)) {
        set_error("cfd_set_params: pinf must be finite and >= 0");
        return CFD_ERR_ARG;
    }
    if (p->variables != CFD_VARS_CONSERVATIVE && p->variables != CFD_VARS_RUP) {
        set_error("cfd_set_params: variables must be CFD_VARS_CONSERVATIVE or CFD_VARS_RUP");
        return CFD_ERR_ARG;
    }
    if (p->residual_kernel < 0 || p->residual_kernel > 1) {
        set_error("cfd_set_params: residual_kernel must be 0 or 1");
        return CFD_ERR_ARG;
    }
    if (p->order != CFD_ORDER_FIRST && p->order != CFD_ORDER_SECOND) {
        set_error("cfd_set_params: invalid order %d", p->order);
        return CFD_ERR_ARG;
    }
    c->params = *p;
    compute_flow(c, 0);
    if (c->has_mesh && p->residual_kernel == 1 && !c->patch_built) {
        CFD_CUDA(cudaSetDevice(c->device));
        const int st = build_patch_layout(c);
        if (st) return st;
    }
    return CFD_OK;
}

int cfd_synchronize(cfd_ctx *c) {
    if (!c) return CFD_ERR_ARG;
    CFD_CUDA(cudaSetDevice(c->device));
    CFD_CUDA(stream_wait(c->stream));
    return CFD_OK;
}

// Patch layout of the residual kernel variant (residual_kernel = 1), from the
// installed mesh's node -> edge incidence and edge arrays (read back from the
// device): node ranges of CFD_PATCH_NODES nodes; per patch its halo
// (neighbours outside the range, sorted), every interior edge touching the
// patch with patch-local endpoint indices (owned 0..np-1, halo np..), and per
// owned node its incident edges as patch-local edge indices in increasing
// order (the fixed summation order).  Only callers of that kernel pay for it.
static int build_patch_layout(cfd_ctx *c) {
    const int nnode = c->nnode, nedge = c->nedge;
    cudaStream_t s = c->stream;
    std::vector<int> ptr(nnode + 1), lst;
    std::vector<int2> en(nedge);
    std::vector<double4> eg(nedge);
    CFD_CUDA(cudaMemcpyAsync(ptr.data(), c->n2e_ptr.p, sizeof(int) * (nnode + 1), cudaMemcpyDeviceToHost, s));
    CFD_CUDA(stream_wait(s));
    lst.resize(ptr[nnode]);
    if (ptr[nnode]) CFD_CUDA(cudaMemcpyAsync(lst.data(), c->n2e.p, sizeof(int) * ptr[nnode], cudaMemcpyDeviceToHost, s));
    if (nedge) {
        CFD_CUDA(cudaMemcpyAsync(en.data(), c->edge_nodes.p, sizeof(int2) * nedge, cudaMemcpyDeviceToHost, s));
        CFD_CUDA(cudaMemcpyAsync(eg.data(), c->edge_geo.p, sizeof(double4) * nedge, cudaMemcpyDeviceToHost, s));
    }
    CFD_CUDA(stream_wait(s));
    {
        const int P = CFD_PATCH_NODES;
        const int np = (nnode + P - 1) / P;
        std::vector<int> pptr(np + 1, 0), hptr(np + 1, 0), halo, stamp(nedge, -1), local(nedge, 0);
        std::vector<int> iptr(nnode + 1, 0), ilist, pl;
        std::vector<double4> pg;
        std::vector<int> hstamp(nnode, -1), hloc(nnode, 0);
        ilist.reserve(ptr[nnode]);
        pl.reserve((size_t)nedge + nedge / 2);
        pg.reserve((size_t)nedge + nedge / 2);
        int nlocmax = 0;
        for (int p = 0; p < np; p++) {
            const int n0 = p * P, n1 = std::min(nnode, n0 + P), nown = n1 - n0;
            // halo, sorted by global index
            std::vector<int> h;
            for (int i = n0; i < n1; i++)
                for (int k = ptr[i]; k < ptr[i + 1]; k++) {
                    const int sg = lst[k], e = sg >= 0 ? sg : ~sg;
                    const int j = sg >= 0 ? en[e].y : en[e].x;
                    if ((j < n0 || j >= n1) && hstamp[j] != p) { hstamp[j] = p; h.push_back(j); }
                }
            std::sort(h.begin(), h.end());
            for (size_t q = 0; q < h.size(); q++) hloc[h[q]] = nown + (int)q;
            halo.insert(halo.end(), h.begin(), h.end());
            hptr[p + 1] = (int)halo.size();
            nlocmax = std::max(nlocmax, nown + (int)h.size());
            auto lid = [&](int g) { return (g >= n0 && g < n1) ? g - n0 : hloc[g]; };
            int cnt = 0;
            for (int i = n0; i < n1; i++)
                for (int k = ptr[i]; k < ptr[i + 1]; k++) {
                    const int sg = lst[k], e = sg >= 0 ? sg : ~sg;
                    if (stamp[e] != p) {
                        stamp[e] = p;
                        local[e] = cnt++;
                        pl.push_back(lid(en[e].x) | (lid(en[e].y) << 16));
                        pg.push_back(eg[e]);
                    }
                }
            for (int i = n0; i < n1; i++) {
                const size_t b = ilist.size();
                for (int k = ptr[i]; k < ptr[i + 1]; k++) {
                    const int sg = lst[k], e = sg >= 0 ? sg : ~sg;
                    ilist.push_back((local[e] << 1) | (sg < 0 ? 1 : 0));
                }
                std::sort(ilist.begin() + b, ilist.end());
                iptr[i + 1] = (int)ilist.size();
            }
            pptr[p + 1] = pptr[p] + cnt;
        }
        if (ilist.empty()) ilist.push_back(0);  // keep the device arrays non-empty
        if (halo.empty()) halo.push_back(0);
        if (pl.empty()) { pl.push_back(0); pg.push_back(make_double4(0, 0, 0, 0)); }
        c->npatch = np;
        c->patch_nlocmax = nlocmax;
        c->use_patch = nlocmax < 65536 && patch_smem_bytes(nlocmax, true) <= kPatchSmemMax;
        if (c->use_patch) {
            CFD_CUDA(c->pe_ptr.upload(pptr.data(), pptr.size(), s));
            CFD_CUDA(c->pe_loc.upload(pl.data(), pl.size(), s));
            CFD_CUDA(c->pe_geo.upload(pg.data(), pg.size(), s));
            CFD_CUDA(c->ph_ptr.upload(hptr.data(), hptr.size(), s));
            CFD_CUDA(c->halo.upload(halo.data(), halo.size(), s));
            CFD_CUDA(c->inc_ptr.upload(iptr.data(), iptr.size(), s));
            CFD_CUDA(c->inc.upload(ilist.data(), ilist.size(), s));
            CFD_CUDA(stream_wait(s));
        }
    }
    c->patch_built = true;
    return CFD_OK;
}

int cfd_set_mesh(cfd_ctx *c, int nnode, int nghost, int nedge, const int *edge_nodes, const double *edge_areav,
                 int nbedge, const int *bedge_nodes, const double *bedge_areav, const int *bedge_type,
                 const double *cvol, const double *coords, const int *n2n_ia, const int *n2n_ja) {
    if (!c) return CFD_ERR_ARG;
    if (nnode <= 0 || nghost < 0 || nedge < 0 || nbedge < 0 || (nedge && (!edge_nodes || !edge_areav)) ||
        (nbedge && (!bedge_nodes || !bedge_areav || !bedge_type)) || !cvol || !coords || !n2n_ia || !n2n_ja) {
        set_error("cfd_set_mesh: invalid sizes or NULL arrays");
        return CFD_ERR_ARG;
    }
    CFD_CUDA(cudaSetDevice(c->device));
    // ---- validation (host): the device kernels index with these values
    for (int e = 0; e < nedge; e++) {
        const int a = edge_nodes[2 * e], b = edge_nodes[2 * e + 1];
        if (a < 0 || b >= nnode || a >= b) {
            set_error("cfd_set_mesh: interior edge %d has nodes (%d,%d); need 0 <= L < R < nNode", e, a, b);
            return CFD_ERR_MESH;
        }
    }
    std::vector<char> ghost_used(nghost, 0);
    for (int e = 0; e < nbedge; e++) {
        const int a = bedge_nodes[2 * e], g = bedge_nodes[2 * e + 1];
        if (a < 0 || a >= nnode || g < nnode || g >= nnode + nghost || ghost_used[g - nnode]) {
            set_error("cfd_set_mesh: boundary edge %d has nodes (%d,%d)", e, a, g);
            return CFD_ERR_MESH;
        }
        ghost_used[g - nnode] = 1;
        if (bedge_type[e] < 0 || bedge_type[e] > 7) {
            set_error("cfd_set_mesh: boundary edge %d has unsupported BC type %d", e, bedge_type[e]);
            return CFD_ERR_UNSUPPORTED;
        }
    }
    if (n2n_ia[0] != 0) { set_error("cfd_set_mesh: n2n_ia[0] != 0"); return CFD_ERR_MESH; }
    for (int i = 0; i < nnode; i++) {
        if (n2n_ia[i + 1] < n2n_ia[i]) { set_error("cfd_set_mesh: n2n_ia not monotone"); return CFD_ERR_MESH; }
        for (int k = n2n_ia[i]; k < n2n_ia[i + 1]; k++)
            if (n2n_ja[k] < 0 || n2n_ja[k] >= nnode || n2n_ja[k] == i) {
                set_error("cfd_set_mesh: n2n_ja entry %d of row %d out of range", k, i);
                return CFD_ERR_MESH;
            }
    }
    if ((int64_t)n2n_ia[nnode] != 2 * (int64_t)nedge) {
        set_error("cfd_set_mesh: node graph has %d entries, expected 2*nEdge=%lld", n2n_ia[nnode], 2LL * nedge);
        return CFD_ERR_MESH;
    }
    for (int i = 0; i < nnode; i++)
        if (!(cvol[i] > 0.0)) { set_error("cfd_set_mesh: cVolume[%d] = %g", i, cvol[i]); return CFD_ERR_MESH; }

    cudaStream_t s = c->stream;
    c->has_mesh = false;
    c->has_system = false;
    c->has_grad = false;
    c->phi_next_valid = false;
    c->lgrad_valid = c->lgrad_pending = false;
    c->lsq_weight = -1;
    c->nnode = nnode;
    c->nghost = nghost;
    c->nedge = nedge;
    c->nbedge = nbedge;
    c->ldq = ((int64_t)nnode + nghost + 31) / 32 * 32;

    // ---- edges: unit normal + magnitude (Vector3D::normalize/magnitude, MATH/src/Vector3D.cpp:216-229)
    auto geo = [](const double *a, double4 &g, double4 &sv) {
        const double mag = sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
        double nx = a[0], ny = a[1], nz = a[2];
        if (mag > 1.0e-20) { nx = a[0] / mag; ny = a[1] / mag; nz = a[2] / mag; }
        g = make_double4(nx, ny, nz, mag);
        sv = make_double4(a[0], a[1], a[2], 0.0);
    };
    std::vector<int2> en(nedge);
    std::vector<double4> eg(nedge);
    {
        std::vector<double4> es(nedge);
        parallel_ranges(nedge, [&](int, int64_t lo, int64_t hi) {
            for (int64_t e = lo; e < hi; e++) {
                en[e] = make_int2(edge_nodes[2 * e], edge_nodes[2 * e + 1]);
                geo(edge_areav + 3 * (size_t)e, eg[e], es[e]);
            }
        });
        std::vector<int2> bnv(nbedge);
        std::vector<double4> bgv(nbedge), bsv(nbedge);
        for (int e = 0; e < nbedge; e++) {
            bnv[e] = make_int2(bedge_nodes[2 * e], bedge_nodes[2 * e + 1]);
            geo(bedge_areav + 3 * (size_t)e, bgv[e], bsv[e]);
        }
        CFD_CUDA(c->edge_nodes.upload(en.data(), nedge, s));
        CFD_CUDA(c->edge_geo.upload(eg.data(), nedge, s));
        CFD_CUDA(c->edge_sv.upload(es.data(), nedge, s));
        CFD_CUDA(c->bedge_nodes.upload(bnv.data(), nbedge, s));
        CFD_CUDA(c->bedge_geo.upload(bgv.data(), nbedge, s));
        CFD_CUDA(c->bedge_sv.upload(bsv.data(), nbedge, s));
        CFD_CUDA(c->bedge_type.upload(bedge_type, nbedge, s));
        CFD_CUDA(stream_wait(s));
    }
    CFD_CUDA(c->cvol.upload(cvol, nnode, s));
    {
        std::vector<double> x(3 * (size_t)nnode);
        for (int i = 0; i < nnode; i++)
            for (int d = 0; d < 3; d++) x[(size_t)d * nnode + i] = coords[3 * (size_t)i + d];
        CFD_CUDA(c->xyz.upload(x.data(), x.size(), s));
        CFD_CUDA(stream_wait(s));
    }
    // physical graph, rows sorted (the reference's list order is insertion order;
    // gradients and limiters are order-insensitive to round-off)
    std::vector<int> gia(n2n_ia, n2n_ia + nnode + 1), gja(n2n_ja, n2n_ja + n2n_ia[nnode]);
    parallel_ranges(nnode, [&](int, int64_t lo, int64_t hi) {
        for (int64_t i = lo; i < hi; i++) std::sort(gja.begin() + gia[i], gja.begin() + gia[i + 1]);
    });
    CFD_CUDA(c->n2n_ia.upload(gia.data(), gia.size(), s));
    CFD_CUDA(c->n2n_ja.upload(gja.data(), gja.size(), s));

    // ---- node -> incident interior edges, ordered by neighbour id
    std::vector<int> ptr(nnode + 1, 0), lst;
    {
        for (int e = 0; e < nedge; e++) { ptr[edge_nodes[2 * e] + 1]++; ptr[edge_nodes[2 * e + 1] + 1]++; }
        for (int i = 0; i < nnode; i++) ptr[i + 1] += ptr[i];
        lst.assign(ptr[nnode], 0);
        std::vector<int> fill(ptr.begin(), ptr.end() - 1), nb(ptr[nnode]);
        for (int e = 0; e < nedge; e++) {
            const int a = edge_nodes[2 * e], b = edge_nodes[2 * e + 1];
            nb[fill[a]] = b; lst[fill[a]++] = e;
            nb[fill[b]] = a; lst[fill[b]++] = ~e;
        }
        std::atomic<bool> same{true};
        parallel_ranges(nnode, [&](int, int64_t r0, int64_t r1) {
            std::vector<int> idx, tmp;
            for (int64_t i = r0; i < r1; i++) {
                const int lo = ptr[i], hi = ptr[i + 1];
                idx.resize(hi - lo);
                std::iota(idx.begin(), idx.end(), lo);
                std::sort(idx.begin(), idx.end(), [&](int x, int y) { return nb[x] < nb[y]; });
                tmp.resize(hi - lo);
                for (int k = 0; k < hi - lo; k++) tmp[k] = lst[idx[k]];
                std::copy(tmp.begin(), tmp.end(), lst.begin() + lo);
                bool ok = hi - lo == gia[i + 1] - gia[i];
                for (int k = 0; ok && k < hi - lo; k++)
                    ok = nb[idx[k]] == gja[gia[i] + k] && (k == 0 || nb[idx[k]] > nb[idx[k - 1]]);
                if (!ok) same = false;
            }
        });
        c->graph_is_edges = same;
        CFD_CUDA(c->n2e_ptr.upload(ptr.data(), ptr.size(), s));
        CFD_CUDA(c->n2e.upload(lst.data(), lst.size(), s));
        CFD_CUDA(stream_wait(s));
    }
    // ---- sliced-ELL incidence of the node-gather kernel (slices of 32 nodes)
    {
        const int nsl = (nnode + 31) / 32;
        std::vector<int64_t> sp(nsl + 1, 0);
        std::vector<int> dg(nnode);
        for (int i = 0; i < nnode; i++) dg[i] = ptr[i + 1] - ptr[i];
        for (int sl = 0; sl < nsl; sl++) {
            int w = 0;
            for (int i = sl * 32; i < std::min(nnode, sl * 32 + 32); i++) w = std::max(w, dg[i]);
            sp[sl + 1] = sp[sl] + 32 * (int64_t)w;
        }
        std::vector<int> sn(std::max<int64_t>(sp[nsl], 1), 0);
        std::vector<double4> sg(std::max<int64_t>(sp[nsl], 1), make_double4(0, 0, 0, 0));
        parallel_ranges(nnode, [&](int, int64_t r0, int64_t r1) {
            for (int64_t i = r0; i < r1; i++) {
                const int64_t b = sp[i >> 5] + (i & 31);
                for (int k = ptr[i]; k < ptr[i + 1]; k++) {
                    const int t = lst[k], e = t >= 0 ? t : ~t;
                    const int64_t slot = b + 32 * (int64_t)(k - ptr[i]);
                    sn[slot] = t >= 0 ? en[e].y : ~en[e].x;
                    sg[slot] = eg[e];
                }
            }
        });
        CFD_CUDA(c->sell_ptr.upload(sp.data(), sp.size(), s));
        CFD_CUDA(c->sell_nbr.upload(sn.data(), sn.size(), s));
        CFD_CUDA(c->sell_geo.upload(sg.data(), sg.size(), s));
        CFD_CUDA(c->deg.upload(dg.data(), dg.size(), s));
        CFD_CUDA(stream_wait(s));
    }
    // ---- patch layout of the residual kernel (variant): built when that kernel is requested
    c->patch_built = false;
    c->use_patch = false;
    if (c->params.residual_kernel == 1) {
        const int st = build_patch_layout(c);
        if (st) return st;
    }
    CFD_CUDA(c->roeflag.alloc(nnode));
    CFD_CUDA(c->fixcount.alloc(2));
    CFD_CUDA(cudaMemsetAsync(c->roeflag.p, 0, sizeof(int) * nnode, s));
    CFD_CUDA(cudaMemsetAsync(c->fixcount.p, 0, 2 * sizeof(int), s));
    c->roe_fix_pending = false;
    c->pc_fix_pending = false;
    {
        std::vector<int> ptr(nnode + 1, 0);
        for (int e = 0; e < nbedge; e++) ptr[bedge_nodes[2 * e] + 1]++;
        for (int i = 0; i < nnode; i++) ptr[i + 1] += ptr[i];
        std::vector<int> lst(std::max(ptr[nnode], 1)), fill(ptr.begin(), ptr.end() - 1);
        for (int e = 0; e < nbedge; e++) lst[fill[bedge_nodes[2 * e]]++] = e;
        CFD_CUDA(c->n2b_ptr.upload(ptr.data(), ptr.size(), s));
        CFD_CUDA(c->n2b.upload(lst.data(), lst.size(), s));
        std::vector<int> bnode;
        for (int i = 0; i < nnode; i++)
            if (ptr[i + 1] > ptr[i]) bnode.push_back(i);
        c->nbnode = (int)bnode.size();
        if (bnode.empty()) bnode.push_back(0);
        CFD_CUDA(c->bnode.upload(bnode.data(), bnode.size(), s));
        CFD_CUDA(stream_wait(s));
    }
    // ---- block CRS pattern (Create_CRS_SolverBlockMatrix, Euler3D/src/Solver.cpp:612-672)
    {
        c->h_IA.assign(nnode + 1, 0);
        for (int i = 0; i < nnode; i++) c->h_IA[i + 1] = c->h_IA[i] + (gia[i + 1] - gia[i]) + 1;
        c->nnzb = c->h_IA[nnode];
        c->h_JA.assign(c->nnzb, 0);
        c->h_IAU.assign(nnode, 0);
        parallel_ranges(nnode, [&](int, int64_t r0, int64_t r1) {
            for (int i = (int)r0; i < (int)r1; i++) {
                int k = c->h_IA[i];
                bool placed = false;
                for (int m = gia[i]; m < gia[i + 1]; m++) {
                    if (!placed && gja[m] > i) { c->h_IAU[i] = k; c->h_JA[k++] = i; placed = true; }
                    c->h_JA[k++] = gja[m];
                }
                if (!placed) { c->h_IAU[i] = k; c->h_JA[k++] = i; }
            }
        });
        auto slot = [&](int r, int col) {
            auto b = c->h_JA.begin() + c->h_IA[r], e = c->h_JA.begin() + c->h_IA[r + 1];
            auto it = std::lower_bound(b, e, col);
            return (int)(it - c->h_JA.begin());
        };
        std::vector<int> ts(c->nnzb);
        parallel_ranges(nnode, [&](int, int64_t r0, int64_t r1) {
            for (int i = (int)r0; i < (int)r1; i++)
                for (int k = c->h_IA[i]; k < c->h_IA[i + 1]; k++) ts[k] = slot(c->h_JA[k], i);
        });
        std::vector<int2> es(nedge);
        parallel_ranges(nedge, [&](int, int64_t e0, int64_t e1) {
            for (int64_t e = e0; e < e1; e++) {
                const int a = edge_nodes[2 * e], b = edge_nodes[2 * e + 1];
                es[e] = make_int2(slot(a, b), slot(b, a));
            }
        });
        CFD_CUDA(c->IA.upload(c->h_IA.data(), c->h_IA.size(), s));
        CFD_CUDA(c->JA.upload(c->h_JA.data(), c->h_JA.size(), s));
        CFD_CUDA(c->IAU.upload(c->h_IAU.data(), c->h_IAU.size(), s));
        CFD_CUDA(c->tslot.upload(ts.data(), ts.size(), s));
        CFD_CUDA(c->eslot.upload(es.data(), es.size(), s));
        int e1 = 0, e2 = 0;
        c->mc.built = false;  // block multicolour ILU ordering is rebuilt on first use
        c->mc.clear_graphs();
        c->pc_valid = false;
        build_levels(c->h_IA, c->h_JA, nnode, true, c->lv_fwd, s, e1);
        build_levels(c->h_IA, c->h_JA, nnode, false, c->lv_bwd, s, e2);
        if (e1 || e2) { set_error("cfd_set_mesh: level upload failed"); return CFD_ERR_CUDA; }
        CFD_CUDA(stream_wait(s));
    }
    // ---- state and work arrays
    CFD_CUDA(c->Q.alloc((size_t)5 * c->ldq));
    CFD_CUDA(c->res.alloc((size_t)5 * nnode));
    CFD_CUDA(c->resd.alloc((size_t)5 * nnode));
    CFD_CUDA(c->dt.alloc(nnode));
    CFD_CUDA(cudaMemsetAsync(c->Q.p, 0, sizeof(double) * 5 * c->ldq, s));
    CFD_CUDA(cudaMemsetAsync(c->res.p, 0, sizeof(double) * 5 * nnode, s));
    CFD_CUDA(cudaMemsetAsync(c->resd.p, 0, sizeof(double) * 5 * nnode, s));
    CFD_CUDA(cudaMemsetAsync(c->dt.p, 0, sizeof(double) * nnode, s));
    CFD_CUDA(stream_wait(s));
    c->pipe.built = false;  // the pipelined step's plan belongs to the mesh
    c->has_mesh = true;
    return cfd_set_freestream(c);
}

int cfd_get_block_pattern(cfd_ctx *c, int64_t *nnzb, int *IA, int *JA, int *IAU) {
    if (!c || !c->has_mesh) { set_error("cfd_get_block_pattern: no mesh"); return CFD_ERR_STATE; }
    if (nnzb) *nnzb = c->nnzb;
    if (IA) std::memcpy(IA, c->h_IA.data(), sizeof(int) * c->h_IA.size());
    if (JA) std::memcpy(JA, c->h_JA.data(), sizeof(int) * c->h_JA.size());
    if (IAU) std::memcpy(IAU, c->h_IAU.data(), sizeof(int) * c->h_IAU.size());
    return CFD_OK;
}

#define NEED_MESH(fn)                                                      \
    if (!c) { set_error(fn ": NULL context"); return CFD_ERR_ARG; }        \
    if (!c->has_mesh) { set_error(fn ": no mesh installed"); return CFD_ERR_STATE; } \
    CFD_CUDA(cudaSetDevice(c->device))

int cfd_set_state(cfd_ctx *c, const double *Q) {
    NEED_MESH("cfd_set_state");
    if (!Q) return CFD_ERR_ARG;
    c->phi_next_valid = false;
    c->lgrad_valid = c->lgrad_pending = false;
    const int64_t n = (int64_t)c->nnode + c->nghost;
    CFD_CUDA(cudaMemcpy2DAsync(c->Q.p, c->ldq * sizeof(double), Q, n * sizeof(double), n * sizeof(double), 5,
                               cudaMemcpyHostToDevice, c->stream));
    return CFD_OK;
}

int cfd_get_state(cfd_ctx *c, double *Q) {
    NEED_MESH("cfd_get_state");
    if (!Q) return CFD_ERR_ARG;
    const int64_t n = (int64_t)c->nnode + c->nghost;
    CFD_CUDA(cudaMemcpy2DAsync(Q, n * sizeof(double), c->Q.p, c->ldq * sizeof(double), n * sizeof(double), 5,
                               cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    return CFD_OK;
}

int cfd_state_device_ptr(cfd_ctx *c, double **dQ, int64_t *ld) {
    NEED_MESH("cfd_state_device_ptr");
    c->phi_next_valid = false;  // the caller may write the state
    c->lgrad_valid = c->lgrad_pending = false;
    if (dQ) *dQ = c->Q.p;
    if (ld) *ld = c->ldq;
    return CFD_OK;
}

int cfd_set_freestream(cfd_ctx *c) {
    NEED_MESH("cfd_set_freestream");
    c->phi_next_valid = false;
    c->lgrad_valid = c->lgrad_pending = false;
    compute_flow(c, 0);
    const int n = c->nnode + c->nghost;
    k_freestream<<<grid_for(n, 256), 256, 0, c->stream>>>(n, c->ldq, c->flow, c->Q.p);
    CFD_LAUNCH_CHECK();
    return CFD_OK;
}

int cfd_begin_iteration(cfd_ctx *c, int iteration) {
    NEED_MESH("cfd_begin_iteration");
    compute_flow(c, iteration);
    k_begin_iteration<<<grid_for(c->nnode, 256), 256, 0, c->stream>>>(c->nnode, c->dt.p, c->ext.p);
    CFD_LAUNCH_CHECK();
    return CFD_OK;
}

int cfd_apply_bc(cfd_ctx *c, int iteration) {
    NEED_MESH("cfd_apply_bc");
    c->flow.iteration = iteration;
    if (c->nbedge == 0) return CFD_OK;
    k_apply_bc<<<grid_for(c->nbedge, 128), 128, 0, c->stream>>>(c->nbedge, c->ldq, c->Q.p, c->bedge_nodes.p,
                                                                  c->bedge_geo.p, c->bedge_type.p, c->flow, c->err.p,
                                                                  nullptr);
    CFD_LAUNCH_CHECK();
    return CFD_OK;
}

int cfd_residual(cfd_ctx *c, int add_time) {
    NEED_MESH("cfd_residual");
    const bool second = c->params.order == CFD_ORDER_SECOND;
    if (second && !c->has_grad) {
        set_error("cfd_residual: second order needs cfd_gradient first");
        return CFD_ERR_STATE;
    }
    if (second && c->params.limiter != CFD_LIMITER_NONE && !c->phi.p) {
        set_error("cfd_residual: limiter requested but cfd_limiter not called");
        return CFD_ERR_STATE;
    }
    switch (c->params.flux_scheme * 2 + (second ? 1 : 0)) {
        case 0: return residual_with_fix<CFD_FLUX_ROE, false>(c, add_time);
        case 1: return residual_with_fix<CFD_FLUX_ROE, true>(c, add_time);
        case 2: return residual_with_fix<CFD_FLUX_HLLC, false>(c, add_time);
        case 3: return residual_with_fix<CFD_FLUX_HLLC, true>(c, add_time);
        case 4: return residual_with_fix<CFD_FLUX_AUSM, false>(c, add_time);
        case 5: return residual_with_fix<CFD_FLUX_AUSM, true>(c, add_time);
        case 6: return residual_with_fix<CFD_FLUX_ROE_LMFIX, false>(c, add_time);
        case 7: return residual_with_fix<CFD_FLUX_ROE_LMFIX, true>(c, add_time);
        case 8: return residual_with_fix<CFD_FLUX_ROE_PRECOND, false>(c, add_time);
        case 9: return residual_with_fix<CFD_FLUX_ROE_PRECOND, true>(c, add_time);
        case 10: return residual_with_fix<CFD_FLUX_ROE_THORNBER, false>(c, add_time);
        case 11: return residual_with_fix<CFD_FLUX_ROE_THORNBER, true>(c, add_time);
        case 12: return residual_with_fix<CFD_FLUX_VANLEER, false>(c, add_time);
        case 13: return residual_with_fix<CFD_FLUX_VANLEER, true>(c, add_time);
        default: set_error("cfd_residual: bad flux scheme"); return CFD_ERR_ARG;
    }
}

int cfd_deltat(cfd_ctx *c, int iteration) {
    NEED_MESH("cfd_deltat");
    compute_flow(c, iteration);
    k_deltat<<<grid_for(c->nnode, 256), 256, 0, c->stream>>>(c->nnode, c->cvol.p, c->cfl, c->dt.p, c->ext.p);
    CFD_LAUNCH_CHECK();
    if (c->params.global_time) {
        k_fill_global_dt<<<grid_for(c->nnode, 256), 256, 0, c->stream>>>(c->nnode, c->ext.p, c->dt.p);
        CFD_LAUNCH_CHECK();
    }
    return CFD_OK;
}

int cfd_residual_rms(cfd_ctx *c, int include_diss, double out[6]) {
    NEED_MESH("cfd_residual_rms");
    if (!out) return CFD_ERR_ARG;
    const int64_t n = c->nnode;
    const double *src = c->res.p;
    if (include_diss) {
        CFD_CUDA(c->work.alloc(std::max<size_t>(c->work.n, (size_t)5 * n)));
        k_add_diss<<<grid_for(5 * n, 256), 256, 0, c->stream>>>(5 * n, c->res.p, c->resd.p, c->work.p);
        CFD_LAUNCH_CHECK();
        src = c->work.p;
    }
    double s[5];
    int st = reduce_sum_sq(c, src, n, n, 5, s);
    if (st) return st;
    // Solver_Steady_Implicit.cpp:107-126
    double tot = s[0] + s[1] + s[2] + s[3] + s[4];
    out[5] = sqrt(tot / (5.0 * (double)n));
    for (int k = 0; k < 5; k++) out[k] = sqrt(s[k] / (double)n);
    return CFD_OK;
}

int cfd_jacobian(cfd_ctx *c, int add_time, int include_diss, int precision) {
    NEED_MESH("cfd_jacobian");
    const bool low_only = (precision & CFD_PREC_LOW_ONLY) != 0;
    precision &= ~CFD_PREC_LOW_ONLY;
    if (precision < CFD_PREC_FP64 || precision > CFD_PREC_BF16 || (low_only && precision == CFD_PREC_FP64)) {
        set_error("cfd_jacobian: precision must be FP64, FP32 or BF16 (LOW_ONLY with FP32/BF16)");
        return CFD_ERR_ARG;
    }
    int st = require_edge_graph(c, "cfd_jacobian");
    if (st) return st;
    if (!low_only) CFD_CUDA(c->A64.alloc((size_t)c->nnzb * 25));
    CFD_CUDA(c->B.alloc((size_t)c->nnode * 5));
    CFD_CUDA(c->X.alloc((size_t)c->nnode * 5));
    c->a_precision = precision;
    c->a64_valid = !low_only;
    double *A64 = low_only ? nullptr : c->A64.p;
    const int mode = c->params.flux_scheme == CFD_FLUX_ROE_PRECOND ? 1
                     : (c->params.flux_scheme == CFD_FLUX_ROE_THORNBER ? 2 : 0);
    if (precision == CFD_PREC_FP32) {
        CFD_CUDA(c->A32.alloc((size_t)c->nnzb * 25));
        dispatch_jacobian<float>(mode, c, add_time, include_diss, A64, c->A32.p);
    } else if (precision == CFD_PREC_BF16) {
        CFD_CUDA(c->A16.alloc((size_t)c->nnzb * 25));
        dispatch_jacobian<uint16_t>(mode, c, add_time, include_diss, A64, c->A16.p);
    } else {
        dispatch_jacobian<float>(mode, c, add_time, include_diss, A64, (float *)nullptr);
    }
    CFD_LAUNCH_CHECK();
    c->has_system = true;
    return CFD_OK;
}

// Level bounds and row records of k_gs_sweep on the device, once per mesh and direction.
static int gs_prepare(cfd_ctx *c, int direction) {
    for (int dir = 0; dir < 2; dir++) {
        if (direction != 2 && direction != dir) continue;
        Levels &L = dir == 0 ? c->lv_fwd : c->lv_bwd;
        if (L.desc_built) continue;
        std::vector<int> rows(c->nnode);
        std::vector<int4> desc(c->nnode);
        CFD_CUDA(cudaMemcpyAsync(rows.data(), L.rows.p, sizeof(int) * c->nnode, cudaMemcpyDeviceToHost, c->stream));
        CFD_CUDA(stream_wait(c->stream));
        for (int t = 0; t < c->nnode; t++)
            desc[t] = make_int4(rows[t], c->h_IA[rows[t]], c->h_IA[rows[t] + 1], c->h_IAU[rows[t]]);
        CFD_CUDA(L.dptr.upload(L.ptr.data(), L.ptr.size(), c->stream));
        CFD_CUDA(L.desc.upload(desc.data(), desc.size(), c->stream));
        CFD_CUDA(stream_wait(c->stream));
        L.desc_built = true;
    }
    return CFD_OK;
}

int cfd_block_gs(cfd_ctx *c, int iterations, int direction, double *rms) {
    NEED_MESH("cfd_block_gs");
    if (!c->has_system) { set_error("cfd_block_gs: no system (call cfd_jacobian)"); return CFD_ERR_STATE; }
    if (!c->a64_valid) {
        set_error("cfd_block_gs: the system is stored in low precision only (CFD_PREC_LOW_ONLY)");
        return CFD_ERR_STATE;
    }
    if (direction < 0 || direction > 2) return CFD_ERR_ARG;
    const int n = c->nnode;
    CFD_CUDA(c->LUd.alloc((size_t)n * 25));
    CFD_CUDA(c->rowrms.alloc(n));
    CFD_CUDA(cudaMemsetAsync(c->X.p, 0, sizeof(double) * 5 * n, c->stream));  // MC_Iterative_Jacobi.c:375
    k_lu_nopivot<<<grid_for(n, 128), 128, 0, c->stream>>>(n, c->A64.p, c->IAU.p, c->LUd.p);
    CFD_LAUNCH_CHECK();
    const int maxit = 10000;
    if (iterations <= 0) iterations = maxit;
    double r = 0.0;
    // A cluster's sweep while the levels are narrow enough for its eight SMs;
    // wider ones a launch each, and all of them where no such cluster can be
    // resident (a partitioned GPU).
    auto narrow = [&](const Levels &L) { return gs_narrow(n, c->nnzb, (int64_t)L.ptr.size() - 1); };
    bool cluster = (direction == 1 || narrow(c->lv_fwd)) && (direction == 0 || narrow(c->lv_bwd));
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kGsCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(kGsCtas);
    lc.blockDim = dim3(kGsThreads);
    lc.dynamicSmemBytes = sizeof(GsShared);
    lc.stream = c->stream;
    lc.attrs = at;
    lc.numAttrs = 1;
    if (cluster) {
        int smax = 0, resident = 0;
        CFD_CUDA(allow_max_dynamic_smem(k_gs_sweep, c->device, &smax));
        cluster = sizeof(GsShared) <= (size_t)smax &&
                  cudaOccupancyMaxActiveClusters(&resident, k_gs_sweep, &lc) == cudaSuccess && resident > 0;
        if (!cluster) (void)cudaGetLastError();
    }
    if (cluster) {
        int st = gs_prepare(c, direction);
        if (st) return st;
        CFD_CUDA(c->red.alloc(std::max<size_t>(c->red.n, (size_t)296 * 128)));
        CFD_CUDA(c->red_out.alloc(std::max<size_t>(c->red_out.n, 64)));
        double *out = c->red_out.p;  // [0] sum, [1] rms, [2] the stop words
        int *stop = reinterpret_cast<int *>(out + 2);
        CFD_CUDA(cudaMemsetAsync(out, 0, 4 * sizeof(double), c->stream));
        struct { double rms; int stop[2]; } back{};
        // the sweeps' results come back a batch at a time
        for (int done = 0; done < iterations && !back.stop[0];) {
            const int last = std::min(iterations, done + 16);
            for (; done < last; done++) {
                const bool fwd = direction == 0 || (direction == 2 && done % 2 == 0);
                const Levels &L = fwd ? c->lv_fwd : c->lv_bwd;
                CFD_CUDA(cudaLaunchKernelEx(&lc, k_gs_sweep, (int)L.ptr.size() - 1, (const int *)L.dptr.p,
                                            (const int4 *)L.desc.p, (const int *)c->JA.p, (const double *)c->A64.p,
                                            (const double *)c->B.p, (const double *)c->LUd.p, c->X.p, c->rowrms.p,
                                            (const int *)stop));
                k_sum_partial<<<296, 256, 0, c->stream>>>(c->rowrms.p, n, c->red.p);
                k_sum_one<<<1, 256, 0, c->stream>>>(c->red.p, 296, out);
                k_gs_check<<<1, 1, 0, c->stream>>>(out, n, done, out + 1, stop);
            }
            CFD_LAUNCH_CHECK();
            CFD_CUDA(cudaMemcpyAsync(&back, out + 1, sizeof back, cudaMemcpyDeviceToHost, c->stream));
            CFD_CUDA(stream_wait(c->stream));
        }
        r = back.rms;
        if (rms) *rms = r;
        return std::isnan(r) ? CFD_ERR_NUMERIC : CFD_OK;
    }
    for (int it = 0; it < iterations; it++) {
        const bool fwd = direction == 0 || (direction == 2 && it % 2 == 0);
        Levels &L = fwd ? c->lv_fwd : c->lv_bwd;
        const int nl = (int)L.ptr.size() - 1;
        for (int l = 0; l < nl; l++) {
            const int lo = L.ptr[l], cnt = L.ptr[l + 1] - lo;
            k_gs_level<<<grid_for(cnt, 128), 128, 0, c->stream>>>(cnt, L.rows.p + lo, c->IA.p, c->JA.p, c->IAU.p,
                                                                    c->A64.p, c->B.p, c->LUd.p, c->X.p, c->rowrms.p);
        }
        CFD_LAUNCH_CHECK();
        double s = 0.0;
        int st = reduce_sum_plain(c, c->rowrms.p, n, &s);
        if (st) return st;
        r = sqrt(s / (double)n);
        if (r < 100.0 * DBL_EPSILON) break;  // MC_Iterative_Jacobi.c:506
    }
    if (rms) *rms = r;
    return std::isnan(r) ? CFD_ERR_NUMERIC : CFD_OK;
}

int cfd_block_lusgs(cfd_ctx *c, int iterations, double *rms) {
    NEED_MESH("cfd_block_lusgs");
    if (!c->has_system) { set_error("cfd_block_lusgs: no system (call cfd_jacobian)"); return CFD_ERR_STATE; }
    if (!c->a64_valid) {
        set_error("cfd_block_lusgs: the system is stored in low precision only (CFD_PREC_LOW_ONLY)");
        return CFD_ERR_STATE;
    }
    const int n = c->nnode;
    if (c->nnzb < 6) { set_error("cfd_block_lusgs: fewer than 6 blocks"); return CFD_ERR_RANGE; }
    CFD_CUDA(c->LUd.alloc((size_t)n * 25));
    CFD_CUDA(c->lupiv.alloc((size_t)n * 5));
    k_lu_pivot<<<grid_for(n, 128), 128, 0, c->stream>>>(n, c->A64.p, c->IAU.p, c->LUd.p, c->lupiv.p);
    k_lusgs_init<<<grid_for(n, 256), 256, 0, c->stream>>>(n, c->B.p, c->X.p);
    CFD_LAUNCH_CHECK();
    if (iterations <= 0) iterations = 100;  // MC_Iterative_Jacobi.c:584-585
    for (int it = 0; it < iterations; it++) {
        for (int dir = 0; dir < 2; dir++) {
            Levels &L = dir == 0 ? c->lv_fwd : c->lv_bwd;
            for (int l = 0; l + 1 < (int)L.ptr.size(); l++) {
                const int lo = L.ptr[l], cnt = L.ptr[l + 1] - lo;
                k_lusgs_level<<<grid_for(cnt, 128), 128, 0, c->stream>>>(cnt, L.rows.p + lo, c->IA.p, c->JA.p,
                                                                           c->IAU.p, c->A64.p, c->B.p, c->LUd.p,
                                                                           c->lupiv.p, c->X.p);
            }
        }
        CFD_LAUNCH_CHECK();
    }
    // The reference's closing RMS (MC_Iterative_Jacobi.c:689-701) multiplies
    // block 6 of the CRS storage by X at that block's column for every row and
    // divides the running sum by 5 after each row; it is reproduced exactly,
    // on the host, as the value the drivers test for NaN.
    std::vector<double> Bh((size_t)n * 5), blk(25), xj(5);
    CFD_CUDA(cudaMemcpyAsync(Bh.data(), c->B.p, sizeof(double) * Bh.size(), cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(cudaMemcpyAsync(blk.data(), c->A64.p + 5 * 25, sizeof(double) * 25, cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(cudaMemcpyAsync(xj.data(), c->X.p + (int64_t)c->h_JA[5] * 5, sizeof(double) * 5,
                             cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    double tv[5];
    for (int ii = 0; ii < 5; ii++) {
        tv[ii] = 0.0;
        for (int jj = 0; jj < 5; jj++) tv[ii] += blk[ii * 5 + jj] * xj[jj];
    }
    double r = 0.0;
    for (int i = 0; i < n; i++) {
        for (int j = 0; j < 5; j++) {
            const double d = Bh[(size_t)i * 5 + j] - tv[j];
            r += d * d;
        }
        r /= 5;
    }
    r = sqrt(r / (double)n);
    if (rms) *rms = r;
    return std::isnan(r) ? CFD_ERR_NUMERIC : check_device_error(c);
}

int cfd_update(cfd_ctx *c, double relax) {
    NEED_MESH("cfd_update");
    if (!c->X.p) { set_error("cfd_update: no solution vector"); return CFD_ERR_STATE; }
    c->phi_next_valid = false;
    c->lgrad_valid = c->lgrad_pending = false;
    k_update<<<grid_for(c->nnode, 256), 256, 0, c->stream>>>(c->nnode, c->ldq, relax, c->X.p, c->Q.p);
    CFD_LAUNCH_CHECK();
    return CFD_OK;
}

int cfd_get_residual(cfd_ctx *c, double *conv, double *diss) {
    NEED_MESH("cfd_get_residual");
    const size_t bytes = sizeof(double) * 5 * c->nnode;
    if (conv) CFD_CUDA(cudaMemcpyAsync(conv, c->res.p, bytes, cudaMemcpyDeviceToHost, c->stream));
    if (diss) CFD_CUDA(cudaMemcpyAsync(diss, c->resd.p, bytes, cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    return check_device_error(c);
}

int cfd_get_deltat(cfd_ctx *c, double *dt) {
    NEED_MESH("cfd_get_deltat");
    if (!dt) return CFD_ERR_ARG;
    CFD_CUDA(cudaMemcpyAsync(dt, c->dt.p, sizeof(double) * c->nnode, cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    return CFD_OK;
}

int cfd_get_extrema(cfd_ctx *c, double out[8]) {
    NEED_MESH("cfd_get_extrema");
    unsigned long long h[8];
    CFD_CUDA(cudaMemcpyAsync(h, c->ext.p, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    for (int k = 0; k < 8; k++) out[k] = bitsd(h[k]);
    return CFD_OK;
}

int cfd_get_farfield(cfd_ctx *c, double out[8]) {
    if (!c || !out) return CFD_ERR_ARG;
    const Flow &f = c->flow;
    out[0] = f.inf_rho; out[1] = f.inf_u; out[2] = f.inf_v; out[3] = f.inf_w;
    out[4] = f.inf_et; out[5] = f.inf_p; out[6] = f.inf_c; out[7] = f.inf_mach;
    return CFD_OK;
}

int cfd_set_farfield(cfd_ctx *c, const double in[8]) {
    if (!c || !in) return CFD_ERR_ARG;
    Flow &f = c->flow;
    f.inf_rho = in[0]; f.inf_u = in[1]; f.inf_v = in[2]; f.inf_w = in[3];
    f.inf_et = in[4]; f.inf_p = in[5]; f.inf_c = in[6]; f.inf_mach = in[7];
    return CFD_OK;
}

int cfd_get_system(cfd_ctx *c, double *A, double *B, double *X) {
    NEED_MESH("cfd_get_system");
    if (!c->has_system) { set_error("cfd_get_system: no system"); return CFD_ERR_STATE; }
    if (A && c->a64_valid) {
        CFD_CUDA(cudaMemcpyAsync(A, c->A64.p, sizeof(double) * 25 * c->nnzb, cudaMemcpyDeviceToHost, c->stream));
    } else if (A) {  // low-precision-only system: widen on the host
        const size_t nz = (size_t)c->nnzb * 25;
        if (c->a_precision == CFD_PREC_FP32) {
            std::vector<float> h(nz);
            CFD_CUDA(cudaMemcpyAsync(h.data(), c->A32.p, sizeof(float) * nz, cudaMemcpyDeviceToHost, c->stream));
            CFD_CUDA(stream_wait(c->stream));
            for (size_t k = 0; k < nz; k++) A[k] = h[k];
        } else {
            std::vector<uint16_t> h(nz);
            CFD_CUDA(cudaMemcpyAsync(h.data(), c->A16.p, sizeof(uint16_t) * nz, cudaMemcpyDeviceToHost, c->stream));
            CFD_CUDA(stream_wait(c->stream));
            for (size_t k = 0; k < nz; k++) {
                const uint32_t bits = (uint32_t)h[k] << 16;
                float f;
                std::memcpy(&f, &bits, sizeof f);
                A[k] = f;
            }
        }
    }
    if (B) CFD_CUDA(cudaMemcpyAsync(B, c->B.p, sizeof(double) * 5 * c->nnode, cudaMemcpyDeviceToHost, c->stream));
    if (X) CFD_CUDA(cudaMemcpyAsync(X, c->X.p, sizeof(double) * 5 * c->nnode, cudaMemcpyDeviceToHost, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    return CFD_OK;
}

int cfd_set_system(cfd_ctx *c, const double *A, const double *B) {
    NEED_MESH("cfd_set_system");
    if (!A || !B) return CFD_ERR_ARG;
    CFD_CUDA(c->A64.upload(A, (size_t)c->nnzb * 25, c->stream));
    CFD_CUDA(c->B.upload(B, (size_t)c->nnode * 5, c->stream));
    CFD_CUDA(c->X.alloc((size_t)c->nnode * 5));
    CFD_CUDA(cudaMemsetAsync(c->X.p, 0, sizeof(double) * 5 * c->nnode, c->stream));
    CFD_CUDA(stream_wait(c->stream));
    c->a_precision = CFD_PREC_FP64;
    c->a64_valid = true;
    c->has_system = true;
    return CFD_OK;
}

int cfd_set_step_pipeline(cfd_ctx *c, int chunks) {
    if (!c || chunks < -1) { set_error("cfd_set_step_pipeline: bad argument"); return CFD_ERR_ARG; }
    c->pipe.request = chunks;
    c->pipe.built = false;
    return CFD_OK;
}

int cfd_residual_step(cfd_ctx *c, int iteration, const double *Q_host, double *conv_host, double *diss_host) {
    NEED_MESH("cfd_residual_step");
    int st;
    if (Q_host && conv_host && diss_host && pipe_eligible(c)) {
        if ((st = pipe_build(c))) return st;
        if (c->pipe.K > 1) return residual_step_pipelined(c, iteration, Q_host, conv_host, diss_host);
    }
    if (Q_host && (st = cfd_set_state(c, Q_host))) return st;
    if ((st = cfd_begin_iteration(c, iteration))) return st;
    if ((st = cfd_apply_bc(c, iteration))) return st;
    if (c->params.order == CFD_ORDER_SECOND) {
        if ((st = cfd_gradient(c))) return st;
        if (c->params.limiter != CFD_LIMITER_NONE && (st = cfd_limiter(c))) return st;
    }
    if ((st = cfd_residual(c, 1))) return st;
    if ((st = cfd_deltat(c, iteration))) return st;
    if (conv_host || diss_host) return cfd_get_residual(c, conv_host, diss_host);
    return CFD_OK;
}

// ---------------------------------------------------------- restart files
int cfd_restart_write(const char *path, int iteration, int nnode, int nghost, const double *Q) {
    if (!path || !Q || nnode <= 0 || nghost < 0) return CFD_ERR_ARG;
    FILE *f = std::fopen(path, "wb");
    if (!f) { set_error("cfd_restart_write: cannot open %s", path); return CFD_ERR_IO; }
    const int hdr[4] = {iteration, nnode, nghost, 5};
    std::fwrite(hdr, sizeof(int), 4, f);
    const int64_t n = (int64_t)nnode + nghost;
    std::vector<double> row(5);
    for (int64_t i = 0; i < n; i++) {
        for (int k = 0; k < 5; k++) row[k] = Q[k * n + i];
        std::fwrite(row.data(), sizeof(double), 5, f);
    }
    std::fclose(f);
    return CFD_OK;
}

int cfd_restart_read(const char *path, int *iteration, int nnode, int nghost, double *Q) {
    if (!path || !Q) return CFD_ERR_ARG;
    FILE *f = std::fopen(path, "rb");
    if (!f) { set_error("cfd_restart_read: cannot open %s", path); return CFD_ERR_IO; }
    int hdr[4];
    if (std::fread(hdr, sizeof(int), 4, f) != 4 || hdr[1] != nnode || hdr[2] != nghost || hdr[3] != 5) {
        std::fclose(f);
        set_error("cfd_restart_read: header mismatch in %s", path);
        return CFD_ERR_IO;
    }
    if (iteration) *iteration = hdr[0];
    const int64_t n = (int64_t)nnode + nghost;
    double row[5];
    for (int64_t i = 0; i < n; i++) {
        if (std::fread(row, sizeof(double), 5, f) != 5) {
            std::fclose(f);
            set_error("cfd_restart_read: short file %s", path);
            return CFD_ERR_IO;
        }
        for (int k = 0; k < 5; k++) Q[k * n + i] = row[k];
    }
    std::fclose(f);
    return CFD_OK;
}

// ------------------------------------------------------------ mesh builder
int cfd_mesh_box(int nx, int ny, int nz, double lx, double ly, double lz, double jitter, uint64_t seed, int rcm,
                 const int face_bc[6], cfd_mesh **out) {
    if (!out) return CFD_ERR_ARG;
    *out = nullptr;
    int fb[6] = {1, 1, 1, 1, 1, 1};
    if (face_bc) std::memcpy(fb, face_bc, sizeof(fb));
    cfd_mesh *m = new cfd_mesh();
    int st = build_box(m->m, nx, ny, nz, lx, ly, lz, jitter, seed, rcm, fb);
    if (st) { delete m; set_error("cfd_mesh_box: build failed (%d)", st); return st; }
    *out = m;
    return CFD_OK;
}

int cfd_mesh_from_cells(int nnode, const double *coords, int64_t ntet, const int *tets, int64_t ntri,
                        const int *tris, const int *tri_bc, cfd_mesh **out) {
    if (!out || !coords || !tets || (ntri && (!tris || !tri_bc)) || nnode <= 0) return CFD_ERR_ARG;
    cfd_mesh *m = new cfd_mesh();
    int st = build_from_cells(m->m, nnode, coords, ntet, tets, ntri, tris, tri_bc);
    if (st) { delete m; set_error("cfd_mesh_from_cells: build failed (%d)", st); return st; }
    *out = m;
    return CFD_OK;
}

int cfd_mesh_read_ugrid(const char *path, int ntag, const int *tag_bc, int numbering, cfd_mesh **out) {
    if (!out || !path || (tag_bc && ntag < 1) || numbering < CFD_NUMBERING_NATURAL ||
        numbering > CFD_NUMBERING_PATCH_RCM)
        return CFD_ERR_ARG;
    *out = nullptr;
    cfd_mesh *m = new cfd_mesh();
    int st = read_ugrid(m->m, path, ntag, tag_bc, numbering);
    if (st) { delete m; return st; }
    *out = m;
    return CFD_OK;
}

int cfd_mesh_sizes(const cfd_mesh *mm, int64_t sizes[7]) {
    if (!mm || !sizes) return CFD_ERR_ARG;
    const HostMesh &m = mm->m;
    sizes[0] = m.nnode; sizes[1] = m.nghost; sizes[2] = m.nedge; sizes[3] = m.nbedge;
    sizes[4] = (int64_t)m.tets.size() / 4; sizes[5] = (int64_t)m.tris.size() / 3;
    sizes[6] = m.n2n_ia.empty() ? 0 : m.n2n_ia.back();
    return CFD_OK;
}

int cfd_mesh_export(const cfd_mesh *mm, int *edge_nodes, double *edge_areav, int *bedge_nodes, double *bedge_areav,
                    int *bedge_type, double *cvol, double *coords, int *n2n_ia, int *n2n_ja) {
    if (!mm) return CFD_ERR_ARG;
    const HostMesh &m = mm->m;
    auto cp = [](auto *dst, const auto &v) {
        if (dst && !v.empty()) std::memcpy(dst, v.data(), v.size() * sizeof(v[0]));
    };
    cp(edge_nodes, m.edge_nodes); cp(edge_areav, m.edge_areav);
    cp(bedge_nodes, m.bedge_nodes); cp(bedge_areav, m.bedge_areav); cp(bedge_type, m.bedge_type);
    cp(cvol, m.cvol); cp(coords, m.coords); cp(n2n_ia, m.n2n_ia); cp(n2n_ja, m.n2n_ja);
    return CFD_OK;
}

int cfd_mesh_export_cells(const cfd_mesh *mm, int *tets, int *tris, int *tri_bc) {
    if (!mm) return CFD_ERR_ARG;
    const HostMesh &m = mm->m;
    if (tets) std::memcpy(tets, m.tets.data(), m.tets.size() * sizeof(int));
    if (tris) std::memcpy(tris, m.tris.data(), m.tris.size() * sizeof(int));
    if (tri_bc) std::memcpy(tri_bc, m.tri_bc.data(), m.tri_bc.size() * sizeof(int));
    return CFD_OK;
}

int cfd_mesh_write_ugrid(const cfd_mesh *mm, const char *path) {
    if (!mm || !path) return CFD_ERR_ARG;
    return write_ugrid(mm->m, path, nullptr);
}

int cfd_set_mesh_from(cfd_ctx *c, const cfd_mesh *mm) {
    if (!c || !mm) return CFD_ERR_ARG;
    const HostMesh &m = mm->m;
    return cfd_set_mesh(c, m.nnode, m.nghost, m.nedge, m.edge_nodes.data(), m.edge_areav.data(), m.nbedge,
                        m.bedge_nodes.data(), m.bedge_areav.data(), m.bedge_type.data(), m.cvol.data(),
                        m.coords.data(), m.n2n_ia.data(), m.n2n_ja.data());
}

void cfd_mesh_free(cfd_mesh *m) { delete m; }

}  // extern "C"
