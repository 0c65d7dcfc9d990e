// Unpreconditioned CG (IterativeSolver.solveCG, IterativeSolver.java:48-103)
// for small systems in one launch: one 8-CTA thread-block cluster runs every
// iteration.  Each thread owns up to two rows and keeps their x, r, p and A p
// entries in registers; the two dot products of an iteration are reduced through
// distributed shared memory (every CTA sums the eight CTA partials in rank
// order, so every thread holds the same value and takes the same branch).
// Two or three cluster barriers per iteration with the matrix in shared memory
// (k_cg_small_smem<true>, <false>), three with p in global memory (k_cg_small),
// replace the ~5 kernel launches of the graph-captured loop, whose launch latency
// dominates at this size.  The scalar recurrences and the stopping test are those of the multi-kernel CG
// (alpha = rz / p.Ap, beta = rr' / rr, `iter < maxit && ||r|| > tol`,
// NONFINITE on a non-finite residual); the loop is bounded by maxit.
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "jfg_krylov.cuh"

namespace jfg {

namespace {

namespace cg = cooperative_groups;

constexpr int kCgCtas = 8;
constexpr int kCgThreads = 1024;
constexpr int kCgRowsPerThread = 2;
constexpr int kSmThreads = 512;      // shared-memory variant: 512 threads x 4 rows
constexpr int kSmRows = 4;
constexpr int kSmMaxRows = 2048;     // rows per CTA of the shared-memory variant
constexpr size_t kSmSmemCap = (size_t)200 * 1024;

struct CgSmallArgs {
    int n;
    const int* ptr;
    const int* col;
    const double* val;
    const double* b;
    double* x;
    double* p;          // global copy of the direction (read by the products)
    Ctl* ctl;           // tol, maxit, hist, hist_cap in; iter, status, res_norm, ... out
};

// sum of one double over the cluster: warp shuffles, the CTA's warps in
// order, then the eight CTA partials (read through DSMEM) in rank order
template <int THREADS = kCgThreads>
__device__ __forceinline__ double cluster_sum(cg::cluster_group& cl, double v, double* warp_part, double* slot)
{
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) warp_part[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < THREADS / 32; i++) s += warp_part[i];
        *slot = s;
    }
    cl.sync();
    double t = 0.0;
    for (int r = 0; r < kCgCtas; r++) t += *cl.map_shared_rank(slot, r);
    return t;
}

__device__ __forceinline__ double row_dot(const CgSmallArgs& a, int i, const double* v)
{
    double s = 0.0;
    for (int k = a.ptr[i]; k < a.ptr[i + 1]; k++) s += a.val[k] * __ldcg(v + a.col[k]);
    return s;
}

__device__ __forceinline__ bool stop_test(Ctl* c, double rn, int iter, int maxit, double tol, int* status)
{
    if (!isfinite(rn)) {
        *status = JFG_NONFINITE;
        return true;
    }
    if (!(rn > tol)) {
        *status = JFG_OK;
        return true;
    }
    if (iter >= maxit) {
        *status = JFG_NOT_CONVERGED;
        return true;
    }
    return false;
}

__global__ void __cluster_dims__(kCgCtas, 1, 1) __launch_bounds__(kCgThreads, 1) k_cg_small(CgSmallArgs a)
{
    __shared__ double warp_part[kCgThreads / 32];
    __shared__ double slots[2];
    cg::cluster_group cl = cg::this_cluster();
    const int tid = (int)cl.block_rank() * kCgThreads + threadIdx.x;
    const bool lead = tid == 0;
    Ctl* c = a.ctl;
    const double tol = c->tol;
    const int maxit = c->maxit;
    double* hist = c->hist;
    const int hist_cap = c->hist_cap;
    int rows[kCgRowsPerThread];
    double x[kCgRowsPerThread], r[kCgRowsPerThread], p[kCgRowsPerThread], ap[kCgRowsPerThread];
#pragma unroll
    for (int j = 0; j < kCgRowsPerThread; j++) {
        rows[j] = tid + j * kCgCtas * kCgThreads;
        x[j] = r[j] = p[j] = ap[j] = 0.0;
        if (rows[j] < a.n) x[j] = a.x[rows[j]];
    }
    // r = b - A x0, rr
    double part = 0.0;
#pragma unroll
    for (int j = 0; j < kCgRowsPerThread; j++)
        if (rows[j] < a.n) {
            r[j] = a.b[rows[j]] - row_dot(a, rows[j], a.x);
            part += r[j] * r[j];
        }
    double rr = cluster_sum(cl, part, warp_part, &slots[0]);
    double rz = rr;
    int iter = 0, status = JFG_NOT_CONVERGED, not_pd = 0;
    double res = sqrt(rr);
    bool done = stop_test(c, res, iter, maxit, tol, &status);
    // p = r
#pragma unroll
    for (int j = 0; j < kCgRowsPerThread; j++)
        if (rows[j] < a.n) {
            p[j] = r[j];
            a.p[rows[j]] = p[j];
        }
    cl.sync();
    while (!done) {
        // A p and p.Ap
        part = 0.0;
#pragma unroll
        for (int j = 0; j < kCgRowsPerThread; j++)
            if (rows[j] < a.n) {
                ap[j] = row_dot(a, rows[j], a.p);
                part += p[j] * ap[j];
            }
        const double pap = cluster_sum(cl, part, warp_part, &slots[1]);
        const double alpha = rz / pap;
        if (!(pap > 0)) not_pd = 1;
        // x += p alpha, r -= A p alpha, ||r||^2
        part = 0.0;
#pragma unroll
        for (int j = 0; j < kCgRowsPerThread; j++)
            if (rows[j] < a.n) {
                x[j] = x[j] + p[j] * alpha;
                r[j] = r[j] - ap[j] * alpha;
                part += r[j] * r[j];
            }
        const double rr_new = cluster_sum(cl, part, warp_part, &slots[0]);
        iter++;
        const double beta = rr_new / rr;
        rz = rr_new;
        rr = rr_new;
        res = sqrt(rr_new);
        if (lead && hist && iter <= hist_cap) hist[iter - 1] = res;
        done = stop_test(c, res, iter, maxit, tol, &status);
        if (done) break;
        // p = r + p beta
#pragma unroll
        for (int j = 0; j < kCgRowsPerThread; j++)
            if (rows[j] < a.n) {
                p[j] = r[j] + p[j] * beta;
                a.p[rows[j]] = p[j];
            }
        cl.sync();
    }
#pragma unroll
    for (int j = 0; j < kCgRowsPerThread; j++)
        if (rows[j] < a.n) a.x[rows[j]] = x[j];
    if (lead) {
        c->iter = iter;
        c->status = status;
        c->res_norm = res;
        c->rr = rr;
        c->rz = rz;
        c->not_pd = not_pd;
        c->done = 1;
    }
    cl.sync();      // no CTA leaves while another may still read its shared memory
}

// The same iteration with the matrix rows in shared memory: CTA q owns the
// contiguous rows [q R, (q + 1) R), keeps their CSR slice and the window [lo, hi)
// of p and r that the slice's columns (and its own rows) span.  Every thread
// stores the new r of its rows into the windows that hold them (DSMEM stores),
// before the barrier of the ||r||^2 sum; each CTA then updates p = r + p beta over
// its own window, the arithmetic of the row's owner, so no barrier separates the
// direction update from the next product: two cluster barriers per iteration.  A
// sum is one push per CTA into a slot of every other, then eight local loads in
// rank order.  Bound by those two rounds (~1,400 cycles each); with p itself
// broadcast to all CTAs, a third barrier for it and sums read remotely, an
// iteration at 4,225 rows took 5.2 us.
// R_WINDOW = false keeps the window of p alone: the owners push p once beta is
// known and a third barrier follows.  The same sums, the same bits, in half of the
// windows' bytes: it takes numberings whose windows are too wide for both (random
// orders, ~6,800 to ~9,300 rows at nine entries each).
// 100 iterations at 8,464 rows in random order, the whole call: 779 us, against
// 1,456 us in k_cg_small; in the grid's order, with both windows, 547 us.
struct CgRange {
    int nnz, lo, hi;    // CSR slice and window of a CTA
};
struct CgWindows {
    CgRange c[kCgCtas];
};

__global__ void __launch_bounds__(256) k_cg_small_range(int n, int R, const int* __restrict__ ptr,
                                                        const int* __restrict__ col, CgRange* __restrict__ out)
{
    __shared__ int slo[8], shi[8];
    const int r0 = min(n, (int)blockIdx.x * R), r1 = min(n, r0 + R);
    int lo = r0, hi = r1;
    for (int k = ptr[r0] + threadIdx.x; k < ptr[r1]; k += 256) {
        lo = min(lo, col[k]);
        hi = max(hi, col[k] + 1);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        slo[threadIdx.x >> 5] = lo;
        shi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) {
            lo = min(lo, slo[w]);
            hi = max(hi, shi[w]);
        }
        out[blockIdx.x] = CgRange{ptr[r1] - ptr[r0], lo, hi};
    }
}

// cluster_sum with the partials pushed: the same sums in the same order.  Between two
// uses of one slot[kCgCtas] lies a sum through another, or the start of the loop:
// its readers are past it (slot_rr is used before the loop and at its end, slot_pap
// between the two).
__device__ __forceinline__ double pushed_sum(cg::cluster_group& cl, double v, double* warp_part, double* slot)
{
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) warp_part[w] = v;
    __syncthreads();
    if (w == 0) {                                             // the CTA's warps in order, by every lane that pushes
        v = 0.0;
#pragma unroll
        for (int i = 0; i < kSmThreads / 32; i++) v += warp_part[i];
        if (l < kCgCtas) *cl.map_shared_rank(slot + cl.block_rank(), l) = v;
    }
    cl.sync();
    double t = 0.0;
#pragma unroll
    for (int r = 0; r < kCgCtas; r++) t += slot[r];
    return t;
}

template <bool R_WINDOW>
__global__ void __cluster_dims__(kCgCtas, 1, 1) __launch_bounds__(kSmThreads, 1)
    k_cg_small_smem(CgSmallArgs a, const __grid_constant__ CgWindows win, int R, int max_nnz, int max_win)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double warp_part[kSmThreads / 32];
    __shared__ double slot_pap[kCgCtas], slot_rr[kCgCtas];
    double* pw = reinterpret_cast<double*>(smem);                          // max_win
    double* rw = pw + max_win;                                             // max_win (R_WINDOW)
    double* lval = R_WINDOW ? rw + max_win : rw;                           // max_nnz
    int* lptr = reinterpret_cast<int*>(lval + max_nnz);                    // R + 1
    int* lcol = lptr + R + 1;                                              // max_nnz
    cg::cluster_group cl = cg::this_cluster();
    const int q = (int)cl.block_rank();
    const int r0 = min(a.n, q * R), r1 = min(a.n, r0 + R), nr = r1 - r0;
    const int lo = win.c[q].lo, W = win.c[q].hi - lo;
    const bool lead = q == 0 && threadIdx.x == 0;
    Ctl* c = a.ctl;
    const double tol = c->tol;
    const int maxit = c->maxit;
    double* hist = c->hist;
    const int hist_cap = c->hist_cap;
    // the CTA's CSR slice, row pointers relative to its first entry, columns to the window
    const int e0 = a.ptr[r0], ne = a.ptr[r1] - e0;
    for (int i = threadIdx.x; i <= nr; i += kSmThreads) lptr[i] = a.ptr[r0 + i] - e0;
    for (int k = threadIdx.x; k < ne; k += kSmThreads) {
        lcol[k] = a.col[e0 + k] - lo;
        lval[k] = a.val[e0 + k];
    }
    for (int i = threadIdx.x; i < W; i += kSmThreads) pw[i] = a.x[lo + i];      // x0, for the first residual
    int rows[kSmRows];
    double x[kSmRows], r[kSmRows], p[kSmRows], ap[kSmRows];
#pragma unroll
    for (int j = 0; j < kSmRows; j++) {
        rows[j] = threadIdx.x + j * kSmThreads;               // local row
        x[j] = r[j] = p[j] = ap[j] = 0.0;
        if (rows[j] < nr) x[j] = a.x[r0 + rows[j]];
    }
    cl.sync();                                                // every CTA runs before a store reaches it
    auto local_dot = [&](int lr) {                            // five entries loaded at a time, summed in order
        double s = 0.0;
        const int k1 = lptr[lr + 1];
        for (int k = lptr[lr]; k < k1; k += 5) {
            int cc[5];
            double v[5];
#pragma unroll
            for (int u = 0; u < 5; u++) {
                cc[u] = k + u < k1 ? lcol[k + u] : 0;
                v[u] = k + u < k1 ? lval[k + u] : 0.0;
            }
            double pv[5];
#pragma unroll
            for (int u = 0; u < 5; u++) pv[u] = pw[cc[u]];
#pragma unroll
            for (int u = 0; u < 5; u++)
                if (k + u < k1) s += v[u] * pv[u];
        }
        return s;
    };
    auto push = [&](double* w, const double (&v)[kSmRows]) {  // the own rows' v into the windows w that hold them
#pragma unroll
        for (int j = 0; j < kSmRows; j++)
            if (rows[j] < nr) {
                const int g = r0 + rows[j];
#pragma unroll
                for (int t = 0; t < kCgCtas; t++)
                    if (g >= win.c[t].lo && g < win.c[t].hi) *cl.map_shared_rank(w + (g - win.c[t].lo), t) = v[j];
            }
    };
    // r = b - A x0, rr
    double part = 0.0;
#pragma unroll
    for (int j = 0; j < kSmRows; j++)
        if (rows[j] < nr) {
            r[j] = a.b[r0 + rows[j]] - local_dot(rows[j]);
            part += r[j] * r[j];
        }
    if constexpr (R_WINDOW) push(rw, r);
    double rr = pushed_sum(cl, part, warp_part, slot_rr);
    double rz = rr;
    int iter = 0, status = JFG_NOT_CONVERGED, not_pd = 0;
    double res = sqrt(rr);
    bool done = stop_test(c, res, iter, maxit, tol, &status);
#pragma unroll
    for (int j = 0; j < kSmRows; j++) p[j] = r[j];
    if constexpr (R_WINDOW) {
        for (int i = threadIdx.x; i < W; i += kSmThreads) pw[i] = rw[i];
        __syncthreads();
    } else {
        push(pw, p);                                          // x0 has been read: the sum's barrier
        cl.sync();
    }
    while (!done) {
        part = 0.0;
#pragma unroll
        for (int j = 0; j < kSmRows; j++)
            if (rows[j] < nr) {
                ap[j] = local_dot(rows[j]);
                part += p[j] * ap[j];
            }
        const double pap = pushed_sum(cl, part, warp_part, slot_pap);
        const double alpha = rz / pap;
        if (!(pap > 0)) not_pd = 1;
        part = 0.0;
#pragma unroll
        for (int j = 0; j < kSmRows; j++)
            if (rows[j] < nr) {
                x[j] = x[j] + p[j] * alpha;
                r[j] = r[j] - ap[j] * alpha;
                part += r[j] * r[j];
            }
        if constexpr (R_WINDOW) push(rw, r);
        const double rr_new = pushed_sum(cl, part, warp_part, slot_rr);
        iter++;
        const double beta = rr_new / rr;
        rz = rr_new;
        rr = rr_new;
        res = sqrt(rr_new);
        if (lead && hist && iter <= hist_cap) hist[iter - 1] = res;
        done = stop_test(c, res, iter, maxit, tol, &status);
        if (done) break;
#pragma unroll
        for (int j = 0; j < kSmRows; j++)
            if (rows[j] < nr) p[j] = r[j] + p[j] * beta;
        if constexpr (R_WINDOW) {
            for (int i = threadIdx.x; i < W; i += kSmThreads) pw[i] = rw[i] + pw[i] * beta;
            __syncthreads();
        } else {
            push(pw, p);
            cl.sync();
        }
    }
#pragma unroll
    for (int j = 0; j < kSmRows; j++)
        if (rows[j] < nr) a.x[r0 + rows[j]] = x[j];
    if (lead) {
        c->iter = iter;
        c->status = status;
        c->res_norm = res;
        c->rr = rr;
        c->rz = rz;
        c->not_pd = not_pd;
        c->done = 1;
    }
    cl.sync();      // no CTA leaves while another may still write its shared memory
}

}  // namespace

bool cg_small_fits(const Matrix* A)
{
    const char* e = getenv("JFEM_SMALL_CG");        // "0": always the multi-kernel loop
    return !(e && e[0] == '0') && A->rows <= kCgCtas * kCgThreads * kCgRowsPerThread;
}

static size_t cg_small_bytes(int n, int max_nnz, int max_win, int windows)
{
    const size_t R = (size_t)(n + kCgCtas - 1) / kCgCtas;
    return sizeof(double) * ((size_t)windows * max_win + max_nnz) + sizeof(int) * (R + 1 + max_nnz) + 16;
}

// Windows that the shared-memory variant keeps beside the largest CSR slice of a
// row block: of p and r (2), of p alone (1), or 0: k_cg_small.
int cg_small_windows(int n, int max_nnz, int max_win)
{
    if ((n + kCgCtas - 1) / kCgCtas > kSmMaxRows) return 0;
    for (int w : {2, 1})
        if (cg_small_bytes(n, max_nnz, max_win, w) <= kSmSmemCap) return w;
    return 0;
}

// Runs the whole CG; the control block w.ctl[0] holds tol / maxit / history
// on entry and the results on return (as the multi-kernel loop leaves them).
void run_cg_small(SolverWork& w, Matrix* A, const double* b, double* x)
{
    cudaStream_t st = w.c->stream;
    const int n = A->rows;
    w.v64[0].alloc((size_t)n);
    CgSmallArgs a{n, A->csr_ptr.p, A->csr_col.p, A->csr_val.p, b, x, w.v64[0].p, w.ctl.p};
    // shared-memory variant when a CTA's CSR slice and its windows of p and r, or of p, fit
    const int R = (n + kCgCtas - 1) / kCgCtas;
    if (A->cg_small_win.size() != kCgCtas * 3) {      // once per matrix: slices and windows of the row blocks
        DevBuf<CgRange> d;
        d.alloc(kCgCtas);
        k_cg_small_range<<<kCgCtas, 256, 0, st>>>(n, R, A->csr_ptr.p, A->csr_col.p, d.p);
        JFG_CUDA(cudaGetLastError());
        note_launch();
        A->cg_small_win.resize(kCgCtas * 3);
        static_assert(sizeof(CgRange) == 3 * sizeof(int), "three ints per row block");
        JFG_CUDA(cudaMemcpyAsync(A->cg_small_win.data(), d.p, sizeof(CgRange) * kCgCtas, cudaMemcpyDeviceToHost, st));
        JFG_CUDA(cudaStreamSynchronize(st));
    }
    CgWindows win;
    int max_nnz = 0, max_win = 0;
    for (int q = 0; q < kCgCtas; q++) {
        win.c[q] = CgRange{A->cg_small_win[3 * q], A->cg_small_win[3 * q + 1], A->cg_small_win[3 * q + 2]};
        max_nnz = std::max(max_nnz, win.c[q].nnz);
        max_win = std::max(max_win, win.c[q].hi - win.c[q].lo);
    }
    // JFEM_SMALL_CG_SMEM: "0" keeps p in global memory, "p" the window of p alone
    const char* e = getenv("JFEM_SMALL_CG_SMEM");
    int windows = cg_small_windows(n, max_nnz, max_win);
    if (e && e[0] == '0') windows = 0;
    if (e && e[0] == 'p') windows = std::min(windows, 1);
    if (windows) {
        const size_t bytes = cg_small_bytes(n, max_nnz, max_win, windows);
        static PerDevice once;
        once.get([] {
            for (auto kern : {k_cg_small_smem<true>, k_cg_small_smem<false>})
                JFG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmSmemCap));
            return 1;
        });
        auto* kern = windows == 2 ? k_cg_small_smem<true> : k_cg_small_smem<false>;
        kern<<<kCgCtas, kSmThreads, bytes, st>>>(a, win, R, max_nnz, max_win);
    } else {
        k_cg_small<<<kCgCtas, kCgThreads, 0, st>>>(a);
    }
    JFG_CUDA(cudaGetLastError());
    note_launch();
}

}  // namespace jfg
