// Batched implicit-Euler time stepping of many independent systems in one
// persistent launch (the HeatEquation time loop, Examples/src/HeatEquation.java:81-94,
// for a whole batch).
//
// Layout: every system keeps its own K = M + dt A (SELL-32-sigma, FP64 and
// FP32 values) and M (FP64) as built by jfg_matrix_from_coo; a device
// descriptor table holds the pointers plus per-system work vectors carved
// from one pool.  A cluster of C CTAs owns one system at a time: the CTA of
// rank c owns a contiguous range of SELL slots (rows), cluster barriers
// separate the phases, and dot products are reduced across the cluster
// through distributed shared memory (fixed order, deterministic).  Clusters
// take systems from a global counter over a largest-first order.
//
// Per step:  rhs = M u + f;  repeat  r = rhs - K u (FP64);  stop when
// ||r|| <= rtol ||rhs||;  solve K e = r/||r|| by FP32 Jacobi-PCG to
// inner_rtol;  u += ||r|| e.
// The inner PCG folds the direction update into the product:
// A p_new = A z + beta A p_old, so one iteration needs two cluster barriers.
//
// Two kernels.  k_batch_heat above takes any matrix and keeps the vectors of a
// system in global memory (L2).  k_batch_onchip takes the systems whose K and M
// carry the values-only 9-point layout (Q1 grids) and that fit the shared
// memory and registers of one cluster: see there.  A call that leaves the
// configuration to the library runs every system on the kernel that takes it;
// a call that names a cluster size, threads or rows runs all of them on
// k_batch_heat with that configuration.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "jfg_ops.cuh"

namespace cg = cooperative_groups;

struct jfg_ctx;
struct jfg_mat;

namespace jfg {
cudaStream_t ctx_stream(jfg_ctx* ctx);
int ctx_device(jfg_ctx* ctx);
void ctx_set_error(jfg_ctx* ctx, const std::string& msg);
Matrix* mat_of(jfg_mat* m);
jfg_ctx* mat_ctx(jfg_mat* m);
}  // namespace jfg

namespace {

using namespace jfg;

struct SysDesc {
    int n, nslots;
    const int *k_off, *k_perm, *k_col;
    const int16_t* k_col16;      // 16-bit column offsets from the row, or null
    const double* k_v64;
    const float* k_v32;
    const int *m_off, *m_perm, *m_col;
    const double* m_v64;
    const float* dinv;
    double *u, *rhs, *r64;
    const double* f;
    float *e, *r, *z, *p, *Ap;
};

struct BatchParams {
    const SysDesc* sys;
    const int* order;
    int nsys;
    int steps;
    double rtol, inner_rtol;
    int inner_max, max_refine;
    unsigned* queue;
    int* iters;
    double* relres;
    int* refines;
    int* status;
};

// Block sum of two values; result valid in every thread.
__device__ __forceinline__ void block_sum2(double& a, double& b, double* sh)
{
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int nw = blockDim.x >> 5;
    a = warp_sum(a);
    b = warp_sum(b);
    if (l == 0) {
        sh[2 * w] = a;
        sh[2 * w + 1] = b;
    }
    __syncthreads();
    double ta = 0, tb = 0;
    for (int i = 0; i < nw; i++) {
        ta += sh[2 * i];
        tb += sh[2 * i + 1];
    }
    a = ta;
    b = tb;
    __syncthreads();
}

// Cluster-wide sum of two values (deterministic: rank order).  slot is a
// double-buffered shared array [2][2] of every CTA.
__device__ __forceinline__ void cluster_sum2(cg::cluster_group& cl, double& a, double& b, double* sh, double* slot,
                                             int& parity)
{
    block_sum2(a, b, sh);
    if (threadIdx.x == 0) {
        slot[2 * parity] = a;
        slot[2 * parity + 1] = b;
    }
    cl.sync();
    double ta = 0, tb = 0;
    const unsigned nb = cl.num_blocks();
    for (unsigned r = 0; r < nb; r++) {
        const double* rs = cl.map_shared_rank(slot, r);
        ta += rs[2 * parity];
        tb += rs[2 * parity + 1];
    }
    a = ta;
    b = tb;
    parity ^= 1;
}

template <typename V, typename X>
__device__ __forceinline__ double sell_row(const int* off, const int* col, const V* val, const X* x, int slot)
{
    const int s = slot >> 5, lane = slot & 31;
    const int o = off[s];
    const int len = (off[s + 1] - o) >> 5;
    double sum = 0;
    for (int k = 0; k < len; k++) sum += (double)val[o + 32 * k + lane] * (double)x[col[o + 32 * k + lane]];
    return sum;
}
// The two passes of an inner PCG iteration take U rows of a thread
// at once (slots t, t + B, t + 2B, ... as in a plain strided loop): all loads
// of those rows are issued before any of their results is used, so a thread
// has several rows' gathers in flight instead of one dependent chain per row.
// Row sums keep the entry order and partial dot products the row order of the
// one-row-at-a-time loop, so the results are the same bits.
constexpr int kRowChunk = 3;     // entries of each row loaded together

template <int U, int CH, bool I16>
__device__ __forceinline__ void sell_rows32(const SysDesc& S, const int (&slot)[U], const int (&row)[U],
                                            float (&q)[U])
{
    const int* __restrict__ off = S.k_off;
    const float* __restrict__ val = S.k_v32;
    const float* x = S.z;                 // written inside the kernel: coherent loads
    int o[U], len[U];
    int maxlen = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
        q[u] = 0.f;
        o[u] = 0;
        len[u] = 0;
        if (row[u] >= 0) {
            const int s = slot[u] >> 5;
            const int a = __ldg(off + s);
            o[u] = a + (slot[u] & 31);
            len[u] = (__ldg(off + s + 1) - a) >> 5;
        }
        maxlen = max(maxlen, len[u]);
    }
    for (int k = 0; k < maxlen; k += CH) {
        int c[U][CH];
        float v[U][CH], xv[U][CH];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int j = 0; j < CH; j++) {
                const bool ok = k + j < len[u];
                const int idx = o[u] + 32 * (k + j);
                if constexpr (I16)
                    c[u][j] = ok ? row[u] + (int)__ldg(S.k_col16 + idx) : 0;
                else
                    c[u][j] = ok ? __ldg(S.k_col + idx) : 0;
                v[u][j] = ok ? __ldg(val + idx) : 0.f;
            }
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int j = 0; j < CH; j++) xv[u][j] = k + j < len[u] ? x[c[u][j]] : 0.f;
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int j = 0; j < CH; j++)
                if (k + j < len[u]) q[u] += v[u][j] * xv[u][j];
    }
}

// p = z + beta p ; Ap = K z + beta Ap ; returns this thread's part of p.Ap.
template <int U, bool I16>
__device__ __forceinline__ double pass_direction(const SysDesc& S, int s0, int s1, float bf)
{
    const int B = blockDim.x;
    double pap = 0;
    for (int b0 = s0 + threadIdx.x; b0 < s1; b0 += U * B) {
        int slot[U], row[U];
        float zr[U], pr[U], ar[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            slot[u] = b0 + u * B;
            row[u] = slot[u] < s1 ? __ldg(S.k_perm + slot[u]) : -1;
            zr[u] = pr[u] = ar[u] = 0.f;
            if (row[u] >= 0) {
                zr[u] = S.z[row[u]];
                pr[u] = S.p[row[u]];
                ar[u] = S.Ap[row[u]];
            }
        }
        float q[U];
        sell_rows32<U, kRowChunk, I16>(S, slot, row, q);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (row[u] < 0) continue;
            const float pn = zr[u] + bf * pr[u];
            const float apn = q[u] + bf * ar[u];
            S.p[row[u]] = pn;
            S.Ap[row[u]] = apn;
            pap += (double)pn * apn;
        }
    }
    return pap;
}

// e += alpha p ; r -= alpha Ap ; z = dinv r ; adds r.z and r.r of this thread.
template <int U>
__device__ __forceinline__ void pass_update(const SysDesc& S, int s0, int s1, float alpha, double& rzn,
                                            double& rrn)
{
    const int B = blockDim.x;
    for (int b0 = s0 + threadIdx.x; b0 < s1; b0 += U * B) {
        int row[U];
        float ev[U], pv[U], rv[U], av[U], dv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int sl = b0 + u * B;
            row[u] = sl < s1 ? __ldg(S.k_perm + sl) : -1;
            ev[u] = pv[u] = rv[u] = av[u] = dv[u] = 0.f;
            if (row[u] >= 0) {
                ev[u] = S.e[row[u]];
                pv[u] = S.p[row[u]];
                rv[u] = S.r[row[u]];
                av[u] = S.Ap[row[u]];
                dv[u] = S.dinv[row[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (row[u] < 0) continue;
            S.e[row[u]] = ev[u] + alpha * pv[u];
            const float rn = rv[u] - alpha * av[u];
            const float zn = dv[u] * rn;
            S.r[row[u]] = rn;
            S.z[row[u]] = zn;
            rzn += (double)rn * zn;
            rrn += (double)rn * rn;
        }
    }
}

// U: rows of a thread in flight per pass (2, 3 or 4; picked by the autotuner)
template <int U>
__global__ void __launch_bounds__(512, 2) k_batch_heat(BatchParams P)
{
    cg::cluster_group cl = cg::this_cluster();
    __shared__ double sh[64];
    __shared__ double slot[4];
    __shared__ int sys_sh;
    const unsigned rank = cl.block_rank();
    const unsigned C = cl.num_blocks();
    int parity = 0;
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            unsigned t = atomicAdd(P.queue, 1u);
            sys_sh = t < (unsigned)P.nsys ? P.order[t] : -1;
        }
        cl.sync();
        const int si = *cl.map_shared_rank(&sys_sh, 0);
        cl.sync();   // everyone has read the leader's slot before it is reused
        if (si < 0) break;
        const SysDesc& S = P.sys[si];   // fields re-read from L1 rather than pinned in registers
        // this CTA's slots
        const int chunk = ((S.nslots / 32 + C - 1) / C) * 32;
        const int s0 = min(S.nslots, (int)rank * chunk), s1 = min(S.nslots, s0 + chunk);
        int total_inner = 0, refines_max = 0, status = JFG_OK;
        double last_rel = 0;
        for (int step = 0; step < P.steps; step++) {
            // rhs = M u + f
            double bb = 0, dummy = 0;
            for (int slot_i = s0 + threadIdx.x; slot_i < s1; slot_i += blockDim.x) {
                const int row = S.m_perm[slot_i];
                if (row < 0) continue;
                double v = sell_row(S.m_off, S.m_col, S.m_v64, S.u, slot_i);
                if (S.f) v += S.f[row];
                S.rhs[row] = v;
                bb += v * v;
            }
            cluster_sum2(cl, bb, dummy, sh, slot, parity);
            const double bnorm = sqrt(bb);
            int ref = 0;
            for (;; ref++) {
                // r = rhs - K u (FP64) and its norm
                double rr = 0, d2 = 0;
                for (int slot_i = s0 + threadIdx.x; slot_i < s1; slot_i += blockDim.x) {
                    const int row = S.k_perm[slot_i];
                    if (row < 0) continue;
                    double v = S.rhs[row] - sell_row(S.k_off, S.k_col, S.k_v64, S.u, slot_i);
                    S.r64[row] = v;
                    rr += v * v;
                }
                cluster_sum2(cl, rr, d2, sh, slot, parity);
                const double rn = sqrt(rr);
                last_rel = bnorm > 0 ? rn / bnorm : rn;
                if (!isfinite(rn)) {
                    status = JFG_NONFINITE;
                    break;
                }
                if (rn <= P.rtol * bnorm || rn == 0.0) break;
                if (ref >= P.max_refine) {
                    status = JFG_NOT_CONVERGED;
                    break;
                }
                // inner FP32 Jacobi-PCG on K e = r / ||r||, e0 = 0
                const float inv = (float)(1.0 / rn);
                double rz = 0, rr32 = 0;
                for (int slot_i = s0 + threadIdx.x; slot_i < s1; slot_i += blockDim.x) {
                    const int row = S.k_perm[slot_i];
                    if (row < 0) continue;
                    const float rv = (float)S.r64[row] * inv;
                    const float zv = S.dinv[row] * rv;
                    S.r[row] = rv;
                    S.z[row] = zv;
                    S.e[row] = 0.f;
                    S.p[row] = 0.f;
                    S.Ap[row] = 0.f;
                    rz += (double)rv * zv;
                    rr32 += (double)rv * rv;
                }
                cluster_sum2(cl, rz, rr32, sh, slot, parity);
                double beta = 0;
                int it = 0;
                while (sqrt(rr32) > P.inner_rtol && it < P.inner_max) {
                    // p = z + beta p ; Ap = K z + beta Ap ; pAp
                    double d3 = 0;
                    const float bf = (float)beta;
                    double pap = S.k_col16 ? pass_direction<U, true>(S, s0, s1, bf)
                                           : pass_direction<U, false>(S, s0, s1, bf);
                    cluster_sum2(cl, pap, d3, sh, slot, parity);
                    const float alpha = (float)(rz / pap);
                    // e += alpha p ; r -= alpha Ap ; z = dinv r
                    double rzn = 0, rrn = 0;
                    pass_update<U>(S, s0, s1, alpha, rzn, rrn);
                    cluster_sum2(cl, rzn, rrn, sh, slot, parity);
                    beta = rzn / rz;
                    rz = rzn;
                    rr32 = rrn;
                    it++;
                    if (!isfinite(rr32)) break;
                }
                total_inner += it;
                // u += ||r|| e
                for (int slot_i = s0 + threadIdx.x; slot_i < s1; slot_i += blockDim.x) {
                    const int row = S.k_perm[slot_i];
                    if (row < 0) continue;
                    S.u[row] += rn * (double)S.e[row];
                }
                cl.sync();
            }
            refines_max = max(refines_max, ref);
            if (status != JFG_OK) break;
        }
        if (rank == 0 && threadIdx.x == 0) {
            P.iters[si] = total_inner;
            P.relres[si] = last_rel;
            P.refines[si] = refines_max;
            P.status[si] = status;
        }
        cl.sync();
    }
}

// ---------------------------------------------------------------------------
// On-chip systems
// ---------------------------------------------------------------------------
// The inner FP32 PCG of a system without a byte of global memory: CTA `rank` of
// the system's cluster owns the rows [rank R, (rank + 1) R) of the matrix's own
// order, thread t of its NT threads the rows t, t + NT, ...:
//   registers     r, p, Ap and 1/diag of the thread's rows (few enough that the
//                 inner loop spills nothing: a spilled word is an L2 access
//                 here, shared memory leaves the L1 no room);
//   shared memory the nine FP32 values of every own row (row chunk, offset,
//                 thread: immediate offsets, one word per bank), e, z of the own
//                 rows with H rows of halo on either side, 16-bit z indices for
//                 the entries of the irregular rows (first and last grid lines).
// A z value that a neighbouring CTA reads is stored into that CTA's halo as it
// is made (distributed shared memory); a dot product is a warp and CTA sum, one
// store into a slot of every CTA of the cluster, a cluster barrier and C local
// loads in rank order.  The FP64 products (M u and b - K u, about four per time
// step against ~75 inner iterations) read the FP64 layouts and u from L2.
// Every row sum, dot product operand and update is the one of k_batch_heat;
// only the order of the partial sums of the dot products differs.
// Bound by shared-memory loads (19 words per row and iteration: of ~12,000 cycles
// per iteration with 4,130 rows per CTA and C = 16, 4,500 the product, 1,700 the
// update) and by the two sums (2,300 and 2,800 at C = 16, 900 each at C = 1).  With
// the vectors in L2 every pass is a chain of dependent loads: 96 systems of 32^2
// ... 256^2 cells, ten steps: 103 ms in k_batch_heat, 39 ms here.
struct OnchipSys {
    int n, S, lo, hi, R, H;
    int k_ld, m_ld;
    const double *k_v64, *m_v64;       // 9-point layouts, then the irregular rows' entries
    const float* k_v32;
    const int *k_iptr, *k_icol, *m_iptr, *m_icol;
    const float* dinv;
    double *u, *rhs;
    const double* f;
};
struct OnchipParams {
    const OnchipSys* sys;
    const int* order;                  // systems of this launch
    int steps;
    double rtol, inner_rtol;
    int inner_max, max_refine;
    int* iters;
    double* relres;
    int* refines;
    int* status;
};
constexpr int kOcMaxCluster = 16;
// variants: threads per CTA x rows per thread, by the rows a CTA owns
struct OcVariant {
    int threads, rows;
    int cap() const { return threads * rows; }
};
constexpr int kOcVariants = 3;
constexpr OcVariant kOcVar[kOcVariants] = {{256, 2}, {512, 3}, {768, 6}};
constexpr size_t kOcSmemCap = 224 * 1024;

inline size_t onchip_smem(int var, int R, int H, int nirr)
{
    (void)R;
    return sizeof(float) * ((size_t)11 * kOcVar[var].cap() + 2 * (size_t)H) + sizeof(uint16_t) * 9 * (size_t)nirr + 16;
}

// address of a CTA-local shared address in CTA `rank`, and a store there
__device__ __forceinline__ uint32_t oc_peer(uint32_t a, int rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void oc_put(uint32_t a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// row sum in FP64: a regular row from the offset streams, an irregular one from its CSR copy
__device__ __forceinline__ double oc_row64(int r, int S, int lo, int hi, const double* __restrict__ v, int ld,
                                           const int* __restrict__ iptr, const int* __restrict__ icol, const double* u)
{
    double sum = 0;
    if (r >= lo && r < hi) {
        double a[9], x[9];
#pragma unroll
        for (int k = 0; k < 9; k++) {
            a[k] = __ldg(v + (size_t)k * ld + (r - lo));
            x[k] = __ldcg(u + r + (k / 3 - 1) * S + (k % 3 - 1));
        }
#pragma unroll
        for (int k = 0; k < 9; k++) sum += a[k] * x[k];
    } else {
        const int i = r < lo ? r : lo + (r - hi);
        const double* iv = v + (size_t)9 * ld;
        for (int k = __ldg(iptr + i); k < __ldg(iptr + i + 1); k++) sum += __ldg(iv + k) * __ldcg(u + __ldg(icol + k));
    }
    return sum;
}

// Cluster-wide sums of N values, handed to f in thread 0 of every CTA (the same
// bits in all of them: the same 16-lane tree over the same per-CTA sums); what f
// leaves in shared memory is visible to the CTA on return.  One thread, because
// an FP64 division or a sum over ranks in all 16 warps costs more issue slots
// than the rows of a pass.  slot[N][16] is used by one call site only (its next
// use lies behind another barrier).
template <int N, class F>
__device__ __forceinline__ void oc_sum(cg::cluster_group& cl, int rank, int C, double (&v)[N], double (*sh)[N],
                                       double (*slot)[kOcMaxCluster], F f)
{
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < N; q++) {
        v[q] = warp_sum(v[q]);
        if (lane == 0) sh[w][q] = v[q];
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int q = 0; q < N; q++) {
            v[q] = lane < (int)(blockDim.x >> 5) ? sh[lane][q] : 0.0;
            v[q] = warp_sum(v[q]);
            if (C > 1 && lane < C) *cl.map_shared_rank(&slot[q][rank], lane) = v[q];
        }
    }
    if (C > 1) {
        cl.sync();
        if (w == 0) {
#pragma unroll
            for (int q = 0; q < N; q++) {
                v[q] = (lane & 15) < C ? slot[q][lane & 15] : 0.0;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
            }
        }
    }
    if (threadIdx.x == 0) f(v);
    __syncthreads();
}

template <int NT, int RPT>
__global__ void __launch_bounds__(NT, NT > 512 ? 1 : 1024 / NT) k_batch_onchip(const __grid_constant__ OnchipParams P)
{
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char oc_raw[];
    __shared__ double sh1[32][1], sh2[32][2];
    __shared__ double slot_a[1][kOcMaxCluster], slot_b[2][kOcMaxCluster], slot_c[1][kOcMaxCluster],
        slot_d[1][kOcMaxCluster], slot_e[2][kOcMaxCluster];
    __shared__ double s_bnorm, s_rn;               // scalars thread 0 computes
    __shared__ float s_alpha, s_beta;
    __shared__ int s_more;
    const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
    const int si = P.order[blockIdx.x / C];
    const OnchipSys& S = P.sys[si];
    const int tid = threadIdx.x;
    const int R = S.R, H = S.H, str = S.S, lo = S.lo, hi = S.hi;
    const int r0 = min(S.n, rank * R), cnt = min(S.n, r0 + R) - r0;
    const int np = min(max(lo - r0, 0), cnt), ts = min(max(hi - r0, 0), cnt);   // regular local rows [np, ts)
    const int nirr = np + (cnt - ts);
    float* kv = reinterpret_cast<float*>(oc_raw);                  // [row chunk][offset][thread]
    float* zs = kv + 9 * NT * RPT;                          // [H][R][H], and slack up to NT * RPT rows
    float* es = zs + NT * RPT + 2 * H;                              // [NT * RPT]
    uint16_t* ic = reinterpret_cast<uint16_t*>(es + NT * RPT);      // [entry][irregular row]
    float dv[RPT], rv[RPT], pv[RPT], av[RPT];
    uint32_t regular = 0;                      // rows of this thread in the 9-point layout
#pragma unroll
    for (int j = 0; j < RPT; j++) {
        const int t = j * NT + tid, r = r0 + t;
        dv[j] = rv[j] = pv[j] = av[j] = 0.f;
        es[t] = 0.f;
        if (t >= cnt) {                        // no row: zeros, so that it adds nothing anywhere
#pragma unroll
            for (int k = 0; k < 9; k++) kv[(j * 9 + k) * NT + tid] = 0.f;
            continue;
        }
        dv[j] = __ldg(S.dinv + r);
        if (t >= np && t < ts) {
            regular |= 1u << j;
#pragma unroll
            for (int k = 0; k < 9; k++)
                kv[(j * 9 + k) * NT + tid] = __ldg(S.k_v32 + (size_t)k * S.k_ld + (r - lo));
        } else {
            const int i = r < lo ? r : lo + (r - hi), il = t < np ? t : np + (t - ts);
            const int b = __ldg(S.k_iptr + i), len = __ldg(S.k_iptr + i + 1) - b;
            for (int k = 0; k < 9; k++) {      // absent entries: value 0 at the row itself
                kv[(j * 9 + k) * NT + tid] = k < len ? __ldg(S.k_v32 + (size_t)9 * S.k_ld + b + k) : 0.f;
                ic[k * nirr + il] = (uint16_t)(H + (k < len ? __ldg(S.k_icol + b + k) - r0 : t));
            }
        }
    }
    // z of own row t, and its copy in a neighbour's halo: the lower neighbour's
    // upper halo holds my rows t < H, the upper one's lower halo t >= R - H
    const uint32_t z_up = rank > 0 ? oc_peer(smem_u32(zs + H + R), rank - 1) : 0;
    const uint32_t z_dn = rank + 1 < C ? oc_peer(smem_u32(zs), rank + 1) : 0;
    auto put_z = [&](int t, float z) {
        zs[H + t] = z;
        if (C == 1) return;
        if (t < H && z_up) oc_put(z_up + 4 * t, z);
        if (t >= R - H && z_dn) oc_put(z_dn + 4 * (t - (R - H)), z);
    };
    const int nrow = cnt > tid ? (cnt - 1 - tid) / NT + 1 : 0;     // rows of this thread
    // every row of the warp regular (or absent): the passes run without a branch
    const bool plain = __all_sync(0xffffffffu, regular == (1u << nrow) - 1u);
    // what no row writes is read all the same, against zero matrix values, by absent
    // rows: behind the rows, and in front of them the halo, which a lower neighbour
    // with fewer than H rows fills in part only
    for (int t = tid; t < NT * RPT + 2 * H; t += NT) zs[t] = 0.f;
    const float* zc = zs + H + tid;
    const float* z3[3] = {zc - str, zc, zc + str};
    cl.sync();                                      // every CTA runs before a halo store reaches it
    int total_inner = 0, refines_max = 0, status = JFG_OK;
    double last_rel = 0;
    const double tol2 = P.inner_rtol * P.inner_rtol;
    for (int step = 0; step < P.steps; step++) {
        double bb[1] = {0};                         // rhs = M u + f
#pragma unroll 1
        for (int t = tid; t < cnt; t += NT) {
            const int r = r0 + t;
            double v = oc_row64(r, str, lo, hi, S.m_v64, S.m_ld, S.m_iptr, S.m_icol, S.u);
            if (S.f) v += S.f[r];
            S.rhs[r] = v;
            bb[0] += v * v;
        }
        oc_sum<1>(cl, rank, C, bb, sh1, slot_a, [&](const double* t) { s_bnorm = sqrt(t[0]); });
        const double bnorm = s_bnorm;
        int ref = 0;
        for (;; ref++) {
            double rr[1] = {0};                     // r = rhs - K u (in FP32 in z's place) and its norm
#pragma unroll 1
            for (int t = tid; t < cnt; t += NT) {
                const int r = r0 + t;
                const double v = S.rhs[r] - oc_row64(r, str, lo, hi, S.k_v64, S.k_ld, S.k_iptr, S.k_icol, S.u);
                zs[H + t] = (float)v;
                rr[0] += v * v;
            }
            oc_sum<1>(cl, rank, C, rr, sh1, slot_c, [&](const double* t) {
                s_rn = sqrt(t[0]);
                s_alpha = (float)(1.0 / s_rn);
                last_rel = bnorm > 0 ? s_rn / bnorm : s_rn;
            });
            const double rn = s_rn;
            if (!isfinite(rn)) {
                status = JFG_NONFINITE;
                break;
            }
            if (rn <= P.rtol * bnorm || rn == 0.0) break;
            if (ref >= P.max_refine) {
                status = JFG_NOT_CONVERGED;
                break;
            }
            // inner FP32 Jacobi-PCG on K e = r / ||r||, e0 = 0
            const float inv = s_alpha;
            double d2[2] = {0, 0};                  // r.z, r.r
#pragma unroll
            for (int j = 0; j < RPT; j++) {
                const int t = j * NT + tid;
                rv[j] = j < nrow ? zs[H + t] * inv : 0.f;
                const float z = dv[j] * rv[j];
                if (j < nrow) put_z(t, z);
                es[t] = pv[j] = av[j] = 0.f;
                d2[0] += (double)rv[j] * z;
                d2[1] += (double)rv[j] * rv[j];
            }
            double rz = 0;                          // thread 0's
            int it = 0;
            oc_sum<2>(cl, rank, C, d2, sh2, slot_e, [&](const double* t) {
                rz = t[0];
                s_beta = 0.f;
                s_more = t[1] > tol2 && P.inner_max > 0;
            });
            while (s_more) {
                // p = z + beta p ; Ap = K z + beta Ap ; p.Ap
                double pap[1] = {0};
                const float bf = s_beta;
                if (plain) {
#pragma unroll
                    for (int j = 0; j < RPT; j++) {
                        float q = 0.f;
#pragma unroll
                        for (int k = 0; k < 9; k++) q += kv[(j * 9 + k) * NT + tid] * z3[k / 3][j * NT + k % 3 - 1];
                        const float z = zc[j * NT];
                        pv[j] = (j < nrow ? z : 0.f) + bf * pv[j];
                        av[j] = q + bf * av[j];
                        pap[0] += (double)pv[j] * av[j];
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < RPT; j++) {
                        const int t = j * NT + tid;
                        float q = 0.f;
                        if (regular >> j & 1) {
#pragma unroll
                            for (int k = 0; k < 9; k++) q += kv[(j * 9 + k) * NT + tid] * z3[k / 3][j * NT + k % 3 - 1];
                        } else if (j < nrow) {
                            const uint16_t* ip = ic + (t < np ? t : np + (t - ts));
#pragma unroll
                            for (int k = 0; k < 9; k++) q += kv[(j * 9 + k) * NT + tid] * zs[ip[k * nirr]];
                        }
                        const float z = zc[j * NT];
                        pv[j] = (j < nrow ? z : 0.f) + bf * pv[j];
                        av[j] = q + bf * av[j];
                        pap[0] += (double)pv[j] * av[j];
                    }
                }
                oc_sum<1>(cl, rank, C, pap, sh1, slot_d, [&](const double* t) { s_alpha = (float)(rz / t[0]); });
                const float alpha = s_alpha;
                // e += alpha p ; r -= alpha Ap ; z = dinv r
                double dn[2] = {0, 0};
#pragma unroll
                for (int j = 0; j < RPT; j++) {
                    const int t = j * NT + tid;
                    es[t] = es[t] + alpha * pv[j];
                    rv[j] = rv[j] - alpha * av[j];
                    const float z = dv[j] * rv[j];
                    if (j < nrow) put_z(t, z);
                    dn[0] += (double)rv[j] * z;
                    dn[1] += (double)rv[j] * rv[j];
                }
                oc_sum<2>(cl, rank, C, dn, sh2, slot_b, [&](const double* t) {
                    s_beta = (float)(t[0] / rz);
                    rz = t[0];
                    it++;
                    s_more = isfinite(t[1]) && t[1] > tol2 && it < P.inner_max;
                });
            }
            total_inner += it;
            // u += ||r|| e
#pragma unroll 1
            for (int t = tid; t < cnt; t += NT) S.u[r0 + t] += rn * (double)es[t];
            cl.sync();
        }
        refines_max = max(refines_max, ref);
        if (status != JFG_OK) break;
    }
    if (rank == 0 && tid == 0) {
        P.iters[si] = total_inner;
        P.relres[si] = last_rel;
        P.refines[si] = refines_max;
        P.status[si] = status;
    }
    cl.sync();                                      // no CTA leaves while another may still store into it
}

__global__ void k_dinv32(int n, const double* diag, float* dinv)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d = diag[i];
    dinv[i] = (float)(fabs(d) < 1e-300 ? 1.0 : 1.0 / d);
}

}  // namespace

struct jfg_batch {
    jfg_ctx* ctx = nullptr;
    int nsys = 0;
    std::vector<jfg::Matrix*> K, M;
    std::vector<int64_t> offs;       // packed offsets, nsys + 1
    std::vector<int> order;          // largest first
    jfg::DevBuf<double> pool64;      // u, rhs, r64
    jfg::DevBuf<float> pool32;       // e, r, z, p, Ap, dinv
    jfg::DevBuf<double> f;
    jfg::DevBuf<SysDesc> desc;
    jfg::DevBuf<int> d_order, iters, refines, status;
    jfg::DevBuf<double> relres;
    jfg::DevBuf<unsigned> queue;
    // on-chip systems: their cluster sizes (0: general kernel), descriptors, and
    // the systems of every launch (one per cluster size and variant) on a stream
    // of its own
    struct OcLaunch {
        int C = 0, var = 0, first = 0, count = 0;
        size_t smem = 0;
        cudaStream_t st = nullptr;
        cudaEvent_t done = nullptr;
    };
    std::vector<int> oc_cluster;
    std::vector<OnchipSys> oc_host;
    std::vector<OcLaunch> oc;
    jfg::DevBuf<OnchipSys> oc_sys;
    jfg::DevBuf<int> oc_order, gen_order;
    int ngen = 0;                    // systems of the general kernel when the library picks
    cudaEvent_t oc_fork = nullptr;
    ~jfg_batch()
    {
        for (auto& l : oc) {
            if (l.done) cudaEventDestroy(l.done);
            if (l.st) cudaStreamDestroy(l.st);
        }
        if (oc_fork) cudaEventDestroy(oc_fork);
    }
    int tuned_cluster = 0, tuned_threads = 0, tuned_rows = 0;
};

namespace {

void build_desc(jfg_batch* b, bool with_f)
{
    std::vector<SysDesc> h(b->nsys);
    int64_t tot = b->offs[b->nsys];
    for (int s = 0; s < b->nsys; s++) {
        jfg::Matrix* K = b->K[s];
        jfg::Matrix* M = b->M[s];
        int64_t o = b->offs[s];
        SysDesc& d = h[s];
        d.n = K->rows;
        d.nslots = K->nslices * jfg::kSliceRows;
        d.k_off = K->off.p;
        d.k_perm = K->perm.p;
        d.k_col = K->col.p;
        d.k_col16 = K->idx16 == 1 ? K->col16.p : nullptr;   // offsets from the row only
        d.k_v64 = K->val.p;
        d.k_v32 = K->val32.p;
        d.m_off = M->off.p;
        d.m_perm = M->perm.p;
        d.m_col = M->col.p;
        d.m_v64 = M->val.p;
        d.u = b->pool64.p + o;
        d.rhs = b->pool64.p + tot + o;
        d.r64 = b->pool64.p + 2 * tot + o;
        d.f = with_f ? b->f.p + o : nullptr;
        d.e = b->pool32.p + o;
        d.r = b->pool32.p + tot + o;
        d.z = b->pool32.p + 2 * tot + o;
        d.p = b->pool32.p + 3 * tot + o;
        d.Ap = b->pool32.p + 4 * tot + o;
        d.dinv = b->pool32.p + 5 * tot + o;
    }
    JFG_CUDA(cudaMemcpyAsync(b->desc.p, h.data(), sizeof(SysDesc) * b->nsys, cudaMemcpyHostToDevice,
                             jfg::ctx_stream(b->ctx)));
    if (b->oc.empty()) return;
    for (int s = 0; s < b->nsys; s++) {
        OnchipSys& d = b->oc_host[s];
        d.dinv = h[s].dinv;
        d.u = h[s].u;
        d.rhs = h[s].rhs;
        d.f = h[s].f;
    }
    JFG_CUDA(cudaMemcpyAsync(b->oc_sys.p, b->oc_host.data(), sizeof(OnchipSys) * b->nsys, cudaMemcpyHostToDevice,
                             jfg::ctx_stream(b->ctx)));
}

// One persistent launch of the general kernel over `nsys` systems of `order`
// with cluster size C and T threads per CTA, on the context's stream.
void enqueue(jfg_batch* b, const int* order, int nsys, int C, int T, int U, int steps, const jfg_batch_opts& o)
{
    void (*kern)(BatchParams) = U == 2 ? k_batch_heat<2> : (U == 4 ? k_batch_heat<4> : k_batch_heat<3>);
    cudaStream_t st = jfg::ctx_stream(b->ctx);
    BatchParams P;
    P.sys = b->desc.p;
    P.order = order;
    P.nsys = nsys;
    P.steps = steps;
    P.rtol = o.rtol;
    P.inner_rtol = o.inner_rtol;
    P.inner_max = o.inner_max;
    P.max_refine = o.max_refine;
    P.queue = b->queue.p;
    P.iters = b->iters.p;
    P.relres = b->relres.p;
    P.refines = b->refines.p;
    P.status = b->status.p;
    JFG_CUDA(cudaMemsetAsync(b->queue.p, 0, sizeof(unsigned), st));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(T);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int max_clusters = 0;
    cfg.gridDim = dim3(C);
    JFG_CUDA(cudaOccupancyMaxActiveClusters(&max_clusters, kern, &cfg));
    if (max_clusters < 1) max_clusters = 1;
    int nclusters = std::min(max_clusters, nsys);
    cfg.gridDim = dim3(nclusters * C);
    JFG_CUDA(cudaLaunchKernelEx(&cfg, kern, P));
    jfg::note_launch();
}

// Device milliseconds of what `work` queues on the context's stream.
template <class F>
float timed(jfg_batch* b, F work)
{
    cudaStream_t st = jfg::ctx_stream(b->ctx);
    cudaEvent_t e0, e1;
    JFG_CUDA(cudaEventCreate(&e0));
    JFG_CUDA(cudaEventCreate(&e1));
    JFG_CUDA(cudaEventRecord(e0, st));
    work();
    JFG_CUDA(cudaEventRecord(e1, st));
    JFG_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    JFG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return ms;
}

using OnchipKernel = void (*)(OnchipParams);
OnchipKernel onchip_kernel(int var)
{
    static const OnchipKernel k[kOcVariants] = {k_batch_onchip<kOcVar[0].threads, kOcVar[0].rows>,
                                                k_batch_onchip<kOcVar[1].threads, kOcVar[1].rows>,
                                                k_batch_onchip<kOcVar[2].threads, kOcVar[2].rows>};
    return k[var];
}

void onchip_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int var, int C, size_t smem, int count,
                   cudaStream_t st)
{
    cfg = {};
    cfg.gridDim = dim3((unsigned)(C * count));
    cfg.blockDim = dim3(kOcVar[var].threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

// Picks the systems of the on-chip kernel and their cluster sizes.  A system
// qualifies when K and M carry the 9-point layout of one grid, its irregular
// rows have at most nine entries, and some cluster size C up to 16 gives every
// CTA no more rows than the largest variant holds, a halo no larger than its rows
// and no more than kOcSmemCap of shared memory.  It gets the smallest such C: an
// iteration costs a CTA about 5,000 cycles of barriers beside ~1.6 cycles per row,
// so SM time grows with C.  While the whole batch would leave more than half
// of the SMs empty, every system's C is doubled as far as its halo allows.
void plan_onchip(jfg_batch* b)
{
    b->oc_cluster.assign(b->nsys, 0);
    b->oc_host.assign(b->nsys, OnchipSys{});
    for (int v = 0; v < kOcVariants; v++) {
        JFG_CUDA(cudaFuncSetAttribute(onchip_kernel(v), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOcSmemCap));
        JFG_CUDA(cudaFuncSetAttribute(onchip_kernel(v), cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    bool resident[kOcMaxCluster + 1] = {};       // cluster sizes that can be resident with the largest CTA
    for (int C = 1; C <= kOcMaxCluster; C++) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        onchip_config(cfg, at, kOcVariants - 1, C, kOcSmemCap, 1, nullptr);
        int nc = 0;
        resident[C] = cudaOccupancyMaxActiveClusters(&nc, onchip_kernel(kOcVariants - 1), &cfg) == cudaSuccess && nc >= 1;
        cudaGetLastError();
    }
    cudaStream_t st = jfg::ctx_stream(b->ctx);
    std::vector<std::vector<int>> ptr(b->nsys), col(b->nsys);
    struct Fit {
        int R, H, var;
        size_t smem;
    };
    auto fit = [&](int s, int C, Fit& out) -> bool {
        const jfg::Matrix* K = b->K[s];
        const int n = K->rows, S = K->st_S, lo = K->st_lo, hi = K->st_hi;
        const int R = ((n + C - 1) / C + 31) / 32 * 32;
        int H = S + 1, nirr = 0;
        const int ni = K->st_nirr;
        for (int i = 0; i < ni; i++) {           // halo of the irregular rows' own columns
            const int r = i < lo ? i : hi + (i - lo), c = r / R, r0 = c * R, r1 = std::min(n, r0 + R);
            for (int k = ptr[s][i]; k < ptr[s][i + 1]; k++)
                H = std::max(H, std::max(r0 - col[s][k], col[s][k] - (r1 - 1)));
        }
        for (int c = 0; c < C; c++) {
            const int r0 = std::min(n, c * R), r1 = std::min(n, r0 + R);
            nirr = std::max(nirr, std::max(0, std::min(lo, r1) - r0) + std::max(0, r1 - std::max(hi, r0)));
        }
        if (C == 1) H = S + 1;
        int var = 0;
        while (var < kOcVariants && R > kOcVar[var].cap()) var++;
        if (var == kOcVariants || (C > 1 && H > R) || R + 2 * H >= 65536) return false;
        out = {R, H, var, onchip_smem(var, R, H, nirr)};
        return out.smem <= kOcSmemCap;
    };
    std::vector<Fit> fits(b->nsys);
    for (int s = 0; s < b->nsys; s++) {
        const jfg::Matrix *K = b->K[s], *M = b->M[s];
        if (!K->st || !M->st || K->st_kind || M->st_kind || K->st_S != M->st_S || K->st_lo != M->st_lo ||
            K->st_hi != M->st_hi || K->rows > kOcMaxCluster * kOcVar[kOcVariants - 1].cap())
            continue;
        const int ni = K->st_nirr;
        ptr[s].assign(ni + 1, 0);
        JFG_CUDA(cudaMemcpyAsync(ptr[s].data(), K->st_iptr.p, sizeof(int) * (ni + 1), cudaMemcpyDeviceToHost, st));
        JFG_CUDA(cudaStreamSynchronize(st));
        col[s].assign(std::max(1, ptr[s][ni]), 0);
        if (ptr[s][ni])
            JFG_CUDA(cudaMemcpyAsync(col[s].data(), K->st_icol.p, sizeof(int) * ptr[s][ni], cudaMemcpyDeviceToHost, st));
        JFG_CUDA(cudaStreamSynchronize(st));
        bool ok = true;
        for (int i = 0; i < ni; i++) ok = ok && ptr[s][i + 1] - ptr[s][i] <= 9;
        for (int C = 1; ok && C <= kOcMaxCluster && !b->oc_cluster[s]; C++)
            if (resident[C] && fit(s, C, fits[s])) b->oc_cluster[s] = C;
    }
    for (bool more = true; more;) {
        long long ctas = 0;
        for (int s = 0; s < b->nsys; s++) ctas += b->oc_cluster[s] ? b->oc_cluster[s] : 1;
        more = false;
        if (2 * ctas > jfg::sm_count()) break;
        for (int s = 0; s < b->nsys; s++) {
            Fit f;
            const int C = 2 * b->oc_cluster[s];
            if (C && C <= kOcMaxCluster && resident[C] && fit(s, C, f)) {
                b->oc_cluster[s] = C;
                fits[s] = f;
                more = true;
            }
        }
    }
    // R is rounded up to whole warps, so the last CTAs of a wide cluster may own no
    // row: they are left out (the same R, so the same rows and the same sums; 32 x 32
    // cells at C = 16: R = 96, 12 CTAs)
    for (int s = 0; s < b->nsys; s++) {
        if (!b->oc_cluster[s]) continue;
        const int need = (b->K[s]->rows + fits[s].R - 1) / fits[s].R;
        if (need < b->oc_cluster[s] && resident[need]) b->oc_cluster[s] = need;
    }
    // launches: the largest clusters first (they need a whole GPC's free SMs),
    // within one the largest systems first
    std::vector<int> ord, gen;
    for (int C = kOcMaxCluster; C >= 1; C--)
        for (int v = kOcVariants - 1; v >= 0; v--) {
            jfg_batch::OcLaunch l;
            l.C = C;
            l.var = v;
            l.first = (int)ord.size();
            for (int s : b->order)
                if (b->oc_cluster[s] == C && fits[s].var == v) {
                    ord.push_back(s);
                    l.smem = std::max(l.smem, fits[s].smem);
                }
            l.count = (int)ord.size() - l.first;
            if (l.count) b->oc.push_back(l);
        }
    for (int s : b->order)
        if (!b->oc_cluster[s]) gen.push_back(s);
    b->ngen = (int)gen.size();
    for (int s : ord) {
        const jfg::Matrix *K = b->K[s], *M = b->M[s];
        OnchipSys& d = b->oc_host[s];
        d.n = K->rows;
        d.S = K->st_S;
        d.lo = K->st_lo;
        d.hi = K->st_hi;
        d.R = fits[s].R;
        d.H = fits[s].H;
        d.k_ld = K->st_ld;
        d.m_ld = M->st_ld;
        d.k_v64 = K->st_val.p;
        d.m_v64 = M->st_val.p;
        d.k_v32 = K->st_val32.p;
        d.k_iptr = K->st_iptr.p;
        d.k_icol = K->st_icol.p;
        d.m_iptr = M->st_iptr.p;
        d.m_icol = M->st_icol.p;
    }
    if (!ord.empty()) {
        b->oc_sys.alloc(b->nsys);
        b->oc_order.alloc(ord.size());
        JFG_CUDA(cudaMemcpyAsync(b->oc_order.p, ord.data(), sizeof(int) * ord.size(), cudaMemcpyHostToDevice, st));
        JFG_CUDA(cudaEventCreateWithFlags(&b->oc_fork, cudaEventDisableTiming));
        for (auto& l : b->oc) {
            JFG_CUDA(cudaStreamCreateWithFlags(&l.st, cudaStreamNonBlocking));
            JFG_CUDA(cudaEventCreateWithFlags(&l.done, cudaEventDisableTiming));
        }
    }
    if (!gen.empty()) {
        b->gen_order.alloc(gen.size());
        JFG_CUDA(cudaMemcpyAsync(b->gen_order.p, gen.data(), sizeof(int) * gen.size(), cudaMemcpyHostToDevice, st));
    }
    JFG_CUDA(cudaStreamSynchronize(st));
}

// The on-chip systems: one launch per cluster size, each on its own stream
// between the context stream's work before and after.  A failure half-way waits for
// what it has launched: device blocks are released on the word of the context's stream.
void enqueue_onchip(jfg_batch* b, int steps, const jfg_batch_opts& o)
{
    if (b->oc.empty()) return;
    cudaStream_t st = jfg::ctx_stream(b->ctx);
    JFG_CUDA(cudaEventRecord(b->oc_fork, st));
    try {
        for (auto& l : b->oc) {
            OnchipParams P = {b->oc_sys.p, b->oc_order.p + l.first, steps, o.rtol, o.inner_rtol, o.inner_max, o.max_refine,
                              b->iters.p, b->relres.p, b->refines.p, b->status.p};
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute at[1];
            onchip_config(cfg, at, l.var, l.C, l.smem, l.count, l.st);
            JFG_CUDA(cudaStreamWaitEvent(l.st, b->oc_fork, 0));
            JFG_CUDA(cudaLaunchKernelEx(&cfg, onchip_kernel(l.var), P));
            jfg::note_launch();
            JFG_CUDA(cudaEventRecord(l.done, l.st));
        }
        for (auto& l : b->oc) JFG_CUDA(cudaStreamWaitEvent(st, l.done, 0));
    } catch (...) {
        for (auto& l : b->oc) cudaStreamSynchronize(l.st);
        throw;
    }
}

}  // namespace

extern "C" {

void jfg_batch_opts_default(jfg_batch_opts* o)
{
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->rtol = 1e-10;
    o->inner_rtol = 1e-5;
    o->inner_max = 500;
    o->max_refine = 6;
}

int jfg_batch_create(jfg_ctx* ctx, int nsys, jfg_mat* const* K, jfg_mat* const* M, jfg_batch** out)
{
    if (!ctx || !out || nsys < 1 || !K || !M) return JFG_ERR_BAD_ARG;
    *out = nullptr;
    auto* b = new jfg_batch();
    try {
        JFG_CUDA(cudaSetDevice(jfg::ctx_device(ctx)));
        b->ctx = ctx;
        b->nsys = nsys;
        b->offs.assign(nsys + 1, 0);
        for (int s = 0; s < nsys; s++) {
            JFG_CHECK(K[s] && M[s] && jfg::mat_ctx(K[s]) == ctx && jfg::mat_ctx(M[s]) == ctx, JFG_ERR_BAD_ARG,
                      "batch matrix missing or from another context");
            jfg::Matrix* k = jfg::mat_of(K[s]);
            jfg::Matrix* m = jfg::mat_of(M[s]);
            JFG_CHECK(k->rows == k->cols && m->rows == m->cols && k->rows == m->rows, JFG_ERR_BAD_ARG,
                      "K and M must be square and of equal size");
            jfg::matrix_ensure_fp32(k);
            b->K.push_back(k);
            b->M.push_back(m);
            b->offs[s + 1] = b->offs[s] + k->rows;
        }
        int64_t tot = b->offs[nsys];
        b->order.resize(nsys);
        for (int s = 0; s < nsys; s++) b->order[s] = s;
        std::stable_sort(b->order.begin(), b->order.end(),
                         [&](int x, int y) { return b->K[x]->nnz > b->K[y]->nnz; });
        cudaStream_t st = jfg::ctx_stream(ctx);
        b->pool64.alloc((size_t)std::max<int64_t>(1, 3 * tot));
        b->pool32.alloc((size_t)std::max<int64_t>(1, 6 * tot));
        b->desc.alloc(nsys);
        b->d_order.alloc(nsys);
        b->iters.alloc(nsys);
        b->refines.alloc(nsys);
        b->status.alloc(nsys);
        b->relres.alloc(nsys);
        b->queue.alloc(1);
        JFG_CUDA(cudaMemcpyAsync(b->d_order.p, b->order.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, st));
        for (int s = 0; s < nsys; s++) {
            int n = b->K[s]->rows;
            if (n)
                k_dinv32<<<(n + 255) / 256, 256, 0, st>>>(n, b->K[s]->diag.p, b->pool32.p + 5 * tot + b->offs[s]);
        }
        JFG_CUDA(cudaGetLastError());
        plan_onchip(b);
        build_desc(b, false);
        JFG_CUDA(cudaStreamSynchronize(st));
    } catch (const jfg::Error& e) {
        jfg::ctx_set_error(ctx, e.msg);
        delete b;
        return e.status;
    }
    *out = b;
    return JFG_OK;
}

int jfg_batch_free(jfg_batch* b)
{
    if (!b) return JFG_ERR_BAD_ARG;
    cudaStreamSynchronize(jfg::ctx_stream(b->ctx));
    delete b;
    return JFG_OK;
}

int jfg_batch_layout(jfg_batch* b, int64_t* total, int64_t* offsets)
{
    if (!b) return JFG_ERR_BAD_ARG;
    if (total) *total = b->offs[b->nsys];
    if (offsets)
        for (int s = 0; s <= b->nsys; s++) offsets[s] = b->offs[s];
    return JFG_OK;
}

int jfg_batch_heat(jfg_batch* b, int steps, const double* h_f, double* h_u, const jfg_batch_opts* opts,
                   jfg_batch_info* info)
{
    if (!b || !h_u || steps < 0) return JFG_ERR_BAD_ARG;
    jfg_batch_opts o;
    if (opts)
        o = *opts;
    else
        jfg_batch_opts_default(&o);
    try {
        JFG_CUDA(cudaSetDevice(jfg::ctx_device(b->ctx)));
        JFG_CHECK(o.cluster == 0 || o.cluster == 1 || o.cluster == 2 || o.cluster == 4 || o.cluster == 8,
                  JFG_ERR_BAD_ARG, "cluster must be 1, 2, 4 or 8");
        JFG_CHECK(o.threads == 0 || o.threads == 256 || o.threads == 512, JFG_ERR_BAD_ARG,
                  "threads must be 256 or 512");
        JFG_CHECK(o.rows_per_thread == 0 || (o.rows_per_thread >= 2 && o.rows_per_thread <= 4), JFG_ERR_BAD_ARG,
                  "rows_per_thread must be 2, 3 or 4");
        JFG_CHECK(o.rtol > 0 && o.inner_rtol > 0 && o.inner_max > 0 && o.max_refine >= 0, JFG_ERR_BAD_ARG,
                  "bad tolerances or caps");
        cudaStream_t st = jfg::ctx_stream(b->ctx);
        int64_t tot = b->offs[b->nsys];
        if (h_f) {
            b->f.alloc((size_t)tot);
            JFG_CUDA(cudaMemcpyAsync(b->f.p, h_f, sizeof(double) * tot, cudaMemcpyHostToDevice, st));
        }
        build_desc(b, h_f != nullptr);
        int C = o.cluster, T = o.threads, U = o.rows_per_thread;
        // the library's choice: on-chip where a system fits; a named
        // configuration is the general kernel's
        const bool pick = C == 0 && T == 0 && U == 0;
        const int* order = pick ? b->gen_order.p : b->d_order.p;
        const int nsys = pick ? b->ngen : b->nsys;
        if (nsys && (C == 0 || T == 0 || U == 0)) {
            // autotune once: one step of every configuration (cluster size x
            // threads per CTA x rows per thread in flight) from the given states
            if (!b->tuned_cluster) {
                float best = 1e30f;
                for (int c : {1, 2, 4, 8})
                    for (int t : {256, 512})
                        for (int u : {2, 3, 4}) {
                            JFG_CUDA(cudaMemcpyAsync(b->pool64.p, h_u, sizeof(double) * tot, cudaMemcpyHostToDevice,
                                                     st));
                            float ms = timed(b, [&] { enqueue(b, order, nsys, c, t, u, 1, o); });
                            if (ms < best) {
                                best = ms;
                                b->tuned_cluster = c;
                                b->tuned_threads = t;
                                b->tuned_rows = u;
                            }
                        }
            }
            if (C == 0) C = b->tuned_cluster;
            if (T == 0) T = b->tuned_threads;
            if (U == 0) U = b->tuned_rows;
        }
        JFG_CUDA(cudaMemcpyAsync(b->pool64.p, h_u, sizeof(double) * tot, cudaMemcpyHostToDevice, st));
        const float ms = timed(b, [&] {
            if (pick) enqueue_onchip(b, steps, o);
            if (nsys) enqueue(b, order, nsys, C, T, U, steps, o);
        });
        if (!nsys) {                             // every system on chip: what the largest one runs with
            C = b->oc[0].C;
            T = kOcVar[b->oc[0].var].threads;
            U = kOcVar[b->oc[0].var].rows;
        }
        JFG_CUDA(cudaMemcpyAsync(h_u, b->pool64.p, sizeof(double) * tot, cudaMemcpyDeviceToHost, st));
        std::vector<int> it(b->nsys), rf(b->nsys), stt(b->nsys);
        std::vector<double> rr(b->nsys);
        JFG_CUDA(cudaMemcpyAsync(it.data(), b->iters.p, sizeof(int) * b->nsys, cudaMemcpyDeviceToHost, st));
        JFG_CUDA(cudaMemcpyAsync(rf.data(), b->refines.p, sizeof(int) * b->nsys, cudaMemcpyDeviceToHost, st));
        JFG_CUDA(cudaMemcpyAsync(stt.data(), b->status.p, sizeof(int) * b->nsys, cudaMemcpyDeviceToHost, st));
        JFG_CUDA(cudaMemcpyAsync(rr.data(), b->relres.p, sizeof(double) * b->nsys, cudaMemcpyDeviceToHost, st));
        JFG_CUDA(cudaStreamSynchronize(st));
        int worst = JFG_OK, failed = 0;
        jfg_batch_info inf{};
        for (int s = 0; s < b->nsys; s++) {
            inf.total_inner_iterations += it[s];
            inf.max_refine_used = std::max(inf.max_refine_used, rf[s]);
            inf.max_rel_residual = std::max(inf.max_rel_residual, rr[s]);
            if (stt[s] != JFG_OK) {
                failed++;
                worst = stt[s];
            }
        }
        inf.failed = failed;
        inf.cluster = C;
        inf.threads = T;
        inf.rows_per_thread = U;
        inf.ms = ms;
        if (info) *info = inf;
        return worst;
    } catch (const jfg::Error& e) {
        jfg::ctx_set_error(b->ctx, e.msg);
        return e.status;
    }
}

}  // extern "C"
