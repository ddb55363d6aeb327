// Jacobi-preconditioned conjugate gradients on an element-by-element system,
// the solver of solvegc2 (SPH_GCsolver_2019.f90:16-316), on the device.
//
// The element matrices gstif(nevab, nevab, nelem) are assembled once (FP64)
// into rows laid out by warps of 32: entry k of row i at first[i >> 5] + 32 k +
// (i & 31), columns ascending, entries that assemble to 0 left out (the
// coupling pass has two unconnected components per node).  A solve is one
// set-up kernel (the preconditioner and the -999 marks of getqmat, x = fixed,
// r = b - K x, the initial dot products) and one persistent cooperative kernel
// that runs every iteration: per iteration two phases over the dofs separated
// by grid barriers,
//   A: p = s + beta p_old for the thread's own rows and ap = K p with the
//      reference's mask, each term forming p_j = s_j + beta p_old_j from the
//      same two values, so the product equals that of the materialised
//      direction bit for bit; the partial sums of p.ap;
//   B: alpha = prod1 / prod2, x += alpha p, r1 = r - alpha ap, s = q r1, the
//      partial sums of r1.r1 and r1.s; then beta and the convergence test
//      r.r / r0.r0 <= tol on squared norms (:112).
// Every block adds all the block partials itself in the same fixed order, so
// alpha, beta and the stop decision are identical in every block and every
// solve is bit-reproducible.  A barrier is one counter that only grows; a wait
// gives up after a bounded number of polls and sets an error word that every
// block then sees, so a solve can end with an error but never hang.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <vector>

#include "../../include/gfsph.h"

namespace {

constexpr int kCgThreads = 256;
// The persistent kernel: one block of 1024 per SM, since a barrier's cost grows
// with the blocks (592 of 256 threads: 22 us an iteration on 180k dofs, 148: 11), and
// kCgRows rows a thread with their x, r, 1/diag, p and ap in registers.
constexpr int kCgIterThreads = 1024;
constexpr int kCgRows = 2;

struct CgScalars {
    double rnorm0;   // r0.r0 (all dofs)
    double prod1;    // r.s over free dofs of the current iterate
    double fnorm;    // fixed.fixed (rnormX of :93-103 with rnorm0)
    double tol;
    int done;        // converged, or nothing to do
    int trivial;     // rnormX below tol: the solution is 0 and nothing runs
    int iters;
    int max_iters;
    int err;         // a grid barrier gave up
    int masked;      // some dof is prescribed or singular
    unsigned int ticket;
    unsigned int bar_count;  // blocks that have arrived, over all barriers
};

struct CgDev {
    int n;
    const int* first;       // first entry of each warp of rows
    const int* len;         // entries of each row
    const int* col;
    const double* val;
    const double* diag;     // assembled diagonal
    double* q;              // 1/diag (0 where the diagonal vanishes)
    int* fix;               // iffix (device copy, -999 marks singular free dofs)
    double *x, *r;
    double2* sp;            // (s, p_old): what phase A gathers of a column
    double *ap, *p;         // rows beyond kCgRows a thread
    double* part;           // block partial sums, 3 x nblocks
    CgScalars* S;
};

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the block in a fixed order; valid in thread 0.
__device__ __forceinline__ double block_reduce(double v, double* sh) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    if (w == 0) t = warp_sum(lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0);
    __syncthreads();
    return t;
}

// Sum of nb block partials in a fixed order, by one warp, valid in all lanes.
__device__ __forceinline__ double sum_partials(const double* part, int nb) {
    double v = 0.0;
    for (int k = threadIdx.x & 31; k < nb; k += 32) v += __ldcg(part + k);
    return warp_sum(v);
}

// Polls of a barrier wait before it gives up: two reads of L2 and a pause each,
// about a microsecond, so about a second in all (a barrier of co-resident blocks
// takes microseconds).
constexpr long long kBarrierPolls = 1LL << 20;

// Grid barrier over the co-resident blocks of a cooperative launch, with a
// reduction: thread 0 holds the block's nr sums in mine; they go to part[r*nb +
// block], and once every block has arrived at this barrier (the phase-th, from
// 1) each adds all the partials, so that out[r] is the same in every thread of
// the grid.  A wait that polls kBarrierPolls times, or sees the error word set,
// sets it and returns false, and every block then leaves the solve.  part is
// not rewritten before every block has passed the next barrier.
__device__ bool barrier_reduce(CgScalars* S, double* part, int nb, int nr, const double* mine, unsigned int phase,
                               double* out) {
    __shared__ double res[2];
    __shared__ int ok;
    if (threadIdx.x == 0) {
        for (int r = 0; r < nr; r++) part[(size_t)r * nb + blockIdx.x] = mine[r];
        __threadfence();
        atomicAdd(&S->bar_count, 1u);
        const unsigned int want = phase * (unsigned int)nb;
        volatile unsigned int* count = &S->bar_count;
        volatile int* err = &S->err;
        ok = 1;
        for (long long k = 0; (int)(*count - want) < 0; k++) {
            if (*err || k >= kBarrierPolls) {
                atomicExch(&S->err, 1);
                ok = 0;
                break;
            }
            if (k >= 64) __nanosleep(64);
        }
        __threadfence();
    }
    __syncthreads();
    if (!ok) return false;
    const int w = threadIdx.x >> 5;
    if (w < nr) {
        const double t = sum_partials(part + (size_t)w * nb, nb);
        if ((threadIdx.x & 31) == 0) res[w] = t;
    }
    __syncthreads();
    for (int r = 0; r < nr; r++) out[r] = res[r];
    __syncthreads();  // res is rewritten by the next barrier
    return true;
}

// One row of K times a vector given by f(column).
template <class F>
__device__ __forceinline__ double row_product(const CgDev& d, int i, F&& f) {
    const int at = d.first[i >> 5] + (i & 31), len = d.len[i];
    double sum = 0.0;
    int k = 0;
    for (; k + 4 <= len; k += 4) {
        int j[4];
        double a[4], v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            j[u] = d.col[at + 32 * (k + u)];
            a[u] = d.val[at + 32 * (k + u)];
        }
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = f(j[u]);
#pragma unroll
        for (int u = 0; u < 4; u++) sum += a[u] * v[u];
    }
    for (; k < len; k++) sum += d.val[at + 32 * k] * f(d.col[at + 32 * k]);
    return sum;
}

// Set-up of a solve (getqmat :124-159 and initcg :165-205): q = 1/diag, a
// free dof with a vanishing diagonal marked -999 (q = 0); x = fixed,
// r = b - K x (unmasked), s = q r, p = s, r0.r0 over all dofs, then
// r = s = p = 0 on prescribed dofs and prod1 = r.s; fixed.fixed for rnormX.
// Two kernels: x must be complete before the product.
__global__ void k_cg_init_x(CgDev d, const float* fixed) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.n) {
        d.x[i] = fixed ? (double)fixed[i] : 0.0;
        const double dg = d.diag[i];
        if (fabs(dg) <= 1.e-35) {
            if (d.fix[i] == 0) d.fix[i] = -999;
            d.q[i] = 0.0;
        } else {
            d.q[i] = 1.0 / dg;
        }
    }
}

__global__ void k_cg_init_rest(CgDev d, const float* rhs) {
    __shared__ double sh[32];
    __shared__ bool last;
    CgScalars* S = d.S;
    double rr = 0.0, rs = 0.0, ff = 0.0;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.n) {
        double r = (double)rhs[i] - row_product(d, i, [&](int j) { return d.x[j]; });
        double s = d.q[i] * r;
        rr = r * r;
        ff = d.x[i] * d.x[i];
        if (d.fix[i] != 0) {
            r = 0.0;
            s = 0.0;
            S->masked = 1;
        }
        rs = r * s;
        d.r[i] = r;
        d.sp[i] = make_double2(s, 0.0);  // with beta = 0 the first direction is p = s
    }
    const int nb = gridDim.x;
    double t0 = block_reduce(rr, sh);
    double t1 = block_reduce(rs, sh);
    double t2 = block_reduce(ff, sh);
    if (threadIdx.x == 0) {
        d.part[blockIdx.x] = t0;
        d.part[nb + blockIdx.x] = t1;
        d.part[2 * nb + blockIdx.x] = t2;
        __threadfence();
        last = (atomicAdd(&S->ticket, 1u) == (unsigned)nb - 1u);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // sums over up to n/256 partials: the block, then thread 0
    double v[3] = {0.0, 0.0, 0.0};
    for (int k = threadIdx.x; k < nb; k += blockDim.x)
        for (int r = 0; r < 3; r++) v[r] += __ldcg(d.part + (size_t)r * nb + k);
    const double rn0 = block_reduce(v[0], sh), p1 = block_reduce(v[1], sh), fn = block_reduce(v[2], sh);
    if (threadIdx.x == 0) {
        S->rnorm0 = rn0;
        S->prod1 = p1;
        S->fnorm = fn;
        S->ticket = 0u;
        // rnormX (:93-103): sqrt(fixed.fixed + r0.r0) below tol: the solution is 0
        if (sqrt(fn + rn0) < S->tol) { S->done = 1; S->trivial = 1; }
    }
}

// Every iteration of jcg (:208-268) in one cooperative launch.  R > 0: at most
// R rows a thread, their vectors in registers; R = 0: any number, in memory.
template <int R>
__global__ void __launch_bounds__(kCgIterThreads) k_cg_iterate(CgDev d) {
    __shared__ double sh[32];
    CgScalars* S = d.S;
    if (S->done) return;  // uniform: set before the launch
    const int nb = gridDim.x;
    const int stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    const bool masked = S->masked != 0;
    double prod1 = S->prod1;
    const double rnorm0 = S->rnorm0, tol = S->tol;
    const int max_iters = S->max_iters;
    constexpr int K = R > 0 ? R : 1;
    double x[K], r[K], q[K], p[K], ap[K];
    bool own[K], free_[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int i = i0 + k * stride;
        own[k] = R > 0 && i < d.n;
        free_[k] = own[k] && (!masked || d.fix[i] == 0);
        x[k] = own[k] ? d.x[i] : 0.0;
        r[k] = own[k] ? d.r[i] : 0.0;
        q[k] = own[k] ? d.q[i] : 0.0;
        p[k] = 0.0;
        ap[k] = 0.0;
    }
    double beta = 0.0;  // first direction: p = s
    double mine[2], red[2];
    unsigned int phase = 0;
    // ap_i and p_i of row i; a masked row's product is over the dofs whose marks cancel (kbyp :273-313)
    auto phase_a = [&](int i, double& pi, double& api) {
        const double2 o = d.sp[i];
        pi = o.x + beta * o.y;
        if (!masked) {
            api = row_product(d, i, [&](int j) {
                const double2 v = d.sp[j];
                return v.x + beta * v.y;
            });
        } else {
            const int fi = d.fix[i], at = d.first[i >> 5] + (i & 31), len = d.len[i];
            api = 0.0;
            for (int k = 0; k < len; k++) {
                const int j = d.col[at + 32 * k];
                if (fi + d.fix[j] != 0) continue;
                const double2 v = d.sp[j];
                api += d.val[at + 32 * k] * (v.x + beta * v.y);
            }
        }
    };
    for (int it = 0;; it++) {
        // A
        double acc = 0.0;
        if (R > 0) {
#pragma unroll
            for (int k = 0; k < K; k++)
                if (own[k]) {
                    phase_a(i0 + k * stride, p[k], ap[k]);
                    if (free_[k]) acc += p[k] * ap[k];
                }
        } else {
            for (int i = i0; i < d.n; i += stride) {
                double pi, api;
                phase_a(i, pi, api);
                d.p[i] = pi;
                d.ap[i] = api;
                if (!masked || d.fix[i] == 0) acc += pi * api;
            }
        }
        mine[0] = block_reduce(acc, sh);
        if (!barrier_reduce(S, d.part, nb, 1, mine, ++phase, red)) return;
        const double alpha = prod1 / red[0];
        // B: x += alpha p, r1 = r - alpha ap, s = q r1 (:233-241)
        double rr = 0.0, rs = 0.0;
        if (R > 0) {
#pragma unroll
            for (int k = 0; k < K; k++)
                if (own[k]) {
                    x[k] = x[k] + alpha * p[k];
                    const double v = r[k] - alpha * ap[k];
                    const double si = q[k] * v;
                    d.sp[i0 + k * stride] = make_double2(si, p[k]);
                    rr += v * v;
                    rs += v * si;
                }
        } else {
            for (int i = i0; i < d.n; i += stride) {
                const double pi = d.p[i];
                d.x[i] = d.x[i] + alpha * pi;
                const double v = d.r[i] - alpha * d.ap[i];
                const double si = d.q[i] * v;
                d.sp[i] = make_double2(si, pi);
                rr += v * v;
                rs += v * si;
            }
        }
        mine[0] = block_reduce(rr, sh);
        mine[1] = block_reduce(rs, sh);
        if (!barrier_reduce(S, d.part + nb, nb, 2, mine, ++phase, red)) return;
        const double rnorm1 = red[0], prod3 = red[1];
        const int iters = it + 1;
        if (rnorm1 / rnorm0 <= tol || iters >= max_iters) {
            // converged: as jcg, the returned residual is the one before this
            // update (the copy r = r1 happens only when the loop goes on)
            if (i0 == 0) {
                S->iters = iters;
                S->done = 1;
            }
#pragma unroll
            for (int k = 0; k < K; k++)
                if (own[k]) {
                    d.x[i0 + k * stride] = x[k];
                    d.r[i0 + k * stride] = r[k];
                }
            return;
        }
        if (R > 0) {
#pragma unroll
            for (int k = 0; k < K; k++) r[k] = r[k] - alpha * ap[k];
        } else {
            for (int i = i0; i < d.n; i += stride) d.r[i] = d.r[i] - alpha * d.ap[i];
        }
        beta = prod3 / prod1;
        prod1 = prod3;
    }
}

// Results in the caller's precision: x (0 when nothing was solved), the
// returned residual, and the -999 marks reset to 0 after a solve.
__global__ void k_cg_finish(CgDev d, float* x_f, float* r_f) {
    const CgScalars* S = d.S;
    const bool trivial = S->trivial != 0;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.n) {
        x_f[i] = trivial ? 0.f : (float)d.x[i];
        if (r_f) r_f[i] = (float)d.r[i];
        if (!trivial && d.fix[i] == -999) d.fix[i] = 0;
    }
}

}  // namespace

struct gfsph_cg {
    int npoin = 0, nelem = 0, nnode = 0, ndofn = 0, n = 0;
    cudaStream_t stream = nullptr;
    int *first = nullptr, *len = nullptr, *col = nullptr, *fix = nullptr;
    double *val = nullptr, *diag = nullptr, *q = nullptr;
    double *x = nullptr, *r = nullptr, *p = nullptr, *ap = nullptr, *part = nullptr;
    double2* sp = nullptr;
    float *in_fixed = nullptr, *in_rhs = nullptr, *out_x = nullptr, *out_r = nullptr;  // caller precision
    CgScalars* S = nullptr;
    CgScalars* hS = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int nblocks = 0;      // one thread per dof (set-up and finish kernels)
    int coop_blocks = 0;  // blocks of the persistent kernel (all co-resident)
    bool regs = false;    // its rows fit kCgRows a thread
    double last_ms = 0.0; // device time of the last solve
    long long launches = 0;
};

namespace {

CgDev view(gfsph_cg* c) {
    CgDev d;
    d.n = c->n; d.first = c->first; d.len = c->len; d.col = c->col; d.val = c->val; d.diag = c->diag; d.q = c->q;
    d.fix = c->fix; d.x = c->x; d.r = c->r; d.sp = c->sp; d.ap = c->ap; d.p = c->p; d.part = c->part; d.S = c->S;
    return d;
}

template <class T>
int dal(T** p, size_t n) {
    return cudaMalloc((void**)p, std::max<size_t>(n, 1) * sizeof(T)) == cudaSuccess ? 0 : 1;
}

void cg_free(gfsph_cg* c) {
    void* ptrs[] = {c->first, c->len, c->col, c->fix, c->val, c->diag, c->q, c->x, c->r, c->sp, c->p, c->ap, c->part,
                    c->in_fixed, c->in_rhs, c->out_x, c->out_r, c->S};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (c->hS) cudaFreeHost(c->hS);
    if (c->ev0) cudaEventDestroy(c->ev0);
    if (c->ev1) cudaEventDestroy(c->ev1);
    if (c->stream) cudaStreamDestroy(c->stream);
}

// The kernels of one solve in stream st, with the right-hand side and the
// prescribed values (null: none) on the device and iffix in c->fix; the
// solution goes to c->out_x, the residual to out_r (or nowhere).
int enqueue_solve(gfsph_cg* c, const float* rhs, const float* fixed, float* out_r, float tol, cudaStream_t st) {
    CgScalars init{};
    init.tol = (double)tol;
    init.max_iters = (int)std::min<long long>(10LL * c->n, 0x7fffffffLL);  // miter = 10*ntotv
    *c->hS = init;
    if (cudaMemcpyAsync(c->S, c->hS, sizeof(CgScalars), cudaMemcpyHostToDevice, st) != cudaSuccess) return GFSPH_ERR_CUDA;
    CgDev d = view(c);
    const int nb = c->nblocks;
    cudaEventRecord(c->ev0, st);
    k_cg_init_x<<<nb, kCgThreads, 0, st>>>(d, fixed);
    k_cg_init_rest<<<nb, kCgThreads, 0, st>>>(d, rhs);
    void* args[] = {&d};
    const void* kernel = c->regs ? (const void*)k_cg_iterate<kCgRows> : (const void*)k_cg_iterate<0>;
    if (cudaLaunchCooperativeKernel(kernel, dim3(c->coop_blocks), dim3(kCgIterThreads), args, 0, st) != cudaSuccess)
        return GFSPH_ERR_CUDA;
    k_cg_finish<<<nb, kCgThreads, 0, st>>>(d, c->out_x, out_r);
    cudaEventRecord(c->ev1, st);
    c->launches += 4;
    if (cudaMemcpyAsync(c->hS, c->S, sizeof(CgScalars), cudaMemcpyDeviceToHost, st) != cudaSuccess) return GFSPH_ERR_CUDA;
    return GFSPH_OK;
}

// Waits for the solve (and the caller's copies after it).
int finish_solve(gfsph_cg* c, cudaStream_t st) {
    if (cudaStreamSynchronize(st) != cudaSuccess) return GFSPH_ERR_CUDA;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    c->last_ms = ms;
    if (c->hS->err) return GFSPH_ERR_CUDA;  // a grid barrier gave up: the result is incomplete
    return cudaGetLastError() == cudaSuccess ? GFSPH_OK : GFSPH_ERR_CUDA;
}

}  // namespace

// A solve without prescribed dofs from a right-hand side on the device, in the
// caller's stream, the solution to host memory x.
int cg_solve_on_device(gfsph_cg* c, const float* rhs, float* x, float tol, cudaStream_t st) {
    if (cudaMemsetAsync(c->fix, 0, c->n * sizeof(int), st) != cudaSuccess) return GFSPH_ERR_CUDA;
    int r = enqueue_solve(c, rhs, nullptr, nullptr, tol, st);
    if (r) return r;
    if (x && cudaMemcpyAsync(x, c->out_x, c->n * sizeof(float), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return GFSPH_ERR_CUDA;
    return finish_solve(c, st);
}

extern "C" {

int gfsph_cg_create(int npoin, int nelem, int nnode, int ndofn, const int* intmat, const float* gstif,
                    gfsph_cg** out) try {
    if (!out || !intmat || !gstif || npoin < 1 || nelem < 1 || nnode < 1 || ndofn < 1) return GFSPH_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return GFSPH_ERR_NO_DEVICE;
    const int nevab = nnode * ndofn;
    const long long ntot = (long long)npoin * ndofn;
    if (ntot > 0x3fffffffLL) return GFSPH_ERR_ARG;
    const int n = (int)ntot;
    // assemble sum_e gstif_e (FP64): the element rows around every row in
    // element order, each row's entries merged by column in that order
    for (long long k = 0; k < (long long)nelem * nnode; k++)
        if (intmat[k] < 1 || intmat[k] > npoin) return GFSPH_ERR_ARG;
    std::vector<int> node_ptr((size_t)npoin + 1, 0);
    for (long long k = 0; k < (long long)nelem * nnode; k++) node_ptr[intmat[k]]++;
    for (int p = 0; p < npoin; p++) node_ptr[p + 1] += node_ptr[p];
    std::vector<int> node_at((size_t)nelem * nnode);  // e * nnode + local node
    {
        std::vector<int> fill(node_ptr.begin(), node_ptr.end() - 1);
        for (long long k = 0; k < (long long)nelem * nnode; k++) node_at[fill[intmat[k] - 1]++] = (int)k;
    }
    struct Entry {
        int col;
        double v;
    };
    std::vector<Entry> row;
    std::vector<int> cols, len(n, 0), rowptr((size_t)n + 1, 0);
    std::vector<double> vals, diag(n, 0.0);
    for (int i = 0; i < n; i++) {
        const int na = i / ndofn, ia = i % ndofn;
        row.clear();
        for (int q = node_ptr[na]; q < node_ptr[na + 1]; q++) {
            const size_t e = (size_t)node_at[q] / nnode;
            const int ea = (node_at[q] % nnode) * ndofn + ia;
            for (int b = 0; b < nnode; b++)
                for (int ib = 0; ib < ndofn; ib++) {
                    const int col = (intmat[e * nnode + b] - 1) * ndofn + ib;
                    const double v = (double)gstif[e * nevab * nevab + (size_t)(b * ndofn + ib) * nevab + ea];
                    size_t k = row.size();
                    while (k > 0 && row[k - 1].col > col) k--;
                    if (k > 0 && row[k - 1].col == col) row[k - 1].v += v;
                    else row.insert(row.begin() + k, Entry{col, v});
                }
        }
        for (const Entry& t : row) {
            if (t.col == i) diag[i] = t.v;
            if (t.v == 0.0) continue;
            cols.push_back(t.col);
            vals.push_back(t.v);
            len[i]++;
        }
        rowptr[i + 1] = (int)cols.size();
    }
    // laid out by warps of 32 rows
    const size_t nwarp = ((size_t)n + 31) / 32;
    std::vector<int> first(nwarp);
    size_t total = 0;
    for (size_t w = 0; w < nwarp; w++) {
        int most = 0;
        for (size_t i = 32 * w; i < std::min((size_t)n, 32 * w + 32); i++) most = std::max(most, len[i]);
        if (total + 32 * (size_t)most > 0x7fffffffULL) return GFSPH_ERR_CAPACITY;
        first[w] = (int)total;
        total += 32 * (size_t)most;
    }
    std::vector<int> col(total, 0);
    std::vector<double> val(total, 0.0);
    for (int i = 0; i < n; i++)
        for (int k = 0; k < len[i]; k++) {
            const size_t at = (size_t)first[i >> 5] + 32 * (size_t)k + (i & 31);
            col[at] = cols[rowptr[i] + k];
            val[at] = vals[rowptr[i] + k];
        }
    gfsph_cg* c = new (std::nothrow) gfsph_cg();
    if (!c) return GFSPH_ERR_HOST;
    c->npoin = npoin; c->nelem = nelem; c->nnode = nnode; c->ndofn = ndofn; c->n = n;
    c->nblocks = (n + kCgThreads - 1) / kCgThreads;
    int st = 0;
    st |= dal(&c->first, nwarp); st |= dal(&c->len, n); st |= dal(&c->col, total); st |= dal(&c->val, total);
    st |= dal(&c->diag, n); st |= dal(&c->fix, n); st |= dal(&c->q, n);
    st |= dal(&c->x, n); st |= dal(&c->r, n); st |= dal(&c->sp, n); st |= dal(&c->p, n);
    st |= dal(&c->ap, n); st |= dal(&c->part, 3 * (size_t)c->nblocks);
    st |= dal(&c->in_fixed, n); st |= dal(&c->in_rhs, n); st |= dal(&c->out_x, n); st |= dal(&c->out_r, n);
    st |= dal(&c->S, 1);
    if (st || cudaMallocHost((void**)&c->hS, sizeof(CgScalars)) != cudaSuccess ||
        cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess) {
        cg_free(c);
        delete c;
        return GFSPH_ERR_CUDA;
    }
    // blocks of the persistent kernel: as many as can be resident at once
    // (a cooperative launch refuses more), at most one per kCgIterThreads dofs
    int dev = 0, nsm = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int want = (n + kCgIterThreads - 1) / kCgIterThreads;
    c->regs = n <= kCgRows * nsm * kCgIterThreads;
    if (c->regs) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg_iterate<kCgRows>, kCgIterThreads, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg_iterate<0>, kCgIterThreads, 0);
    c->coop_blocks = std::max(1, std::min(want, nsm * std::max(per_sm, 1)));
    cudaMemcpy(c->first, first.data(), nwarp * sizeof(int), cudaMemcpyHostToDevice);
    cudaMemcpy(c->len, len.data(), n * sizeof(int), cudaMemcpyHostToDevice);
    cudaMemcpy(c->col, col.data(), total * sizeof(int), cudaMemcpyHostToDevice);
    cudaMemcpy(c->val, val.data(), total * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(c->diag, diag.data(), n * sizeof(double), cudaMemcpyHostToDevice);
    if (cudaGetLastError() != cudaSuccess) { cg_free(c); delete c; return GFSPH_ERR_CUDA; }
    *out = c;
    return GFSPH_OK;
} catch (...) {  // a C++ exception never crosses the C ABI
    return GFSPH_ERR_HOST;
}

int gfsph_cg_destroy(gfsph_cg* c) try {
    if (!c) return GFSPH_ERR_ARG;
    cudaStreamSynchronize(c->stream);
    cg_free(c);
    delete c;
    return GFSPH_OK;
} catch (...) {  // a C++ exception never crosses the C ABI
    return GFSPH_ERR_HOST;
}

int gfsph_cg_solve(gfsph_cg* c, int* iffix, const float* fixed, float* rcg, float* ficg, float tol, int* iterations) try {
    if (!c || !iffix || !fixed || !rcg || !ficg) return GFSPH_ERR_ARG;
    const int n = c->n;
    cudaStream_t st = c->stream;
    if (cudaMemcpyAsync(c->fix, iffix, n * sizeof(int), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(c->in_fixed, fixed, n * sizeof(float), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(c->in_rhs, rcg, n * sizeof(float), cudaMemcpyHostToDevice, st) != cudaSuccess)
        return GFSPH_ERR_CUDA;
    int r = enqueue_solve(c, c->in_rhs, c->in_fixed, c->out_r, tol, st);
    if (r) return r;
    if (cudaMemcpyAsync(ficg, c->out_x, n * sizeof(float), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(rcg, c->out_r, n * sizeof(float), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(iffix, c->fix, n * sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return GFSPH_ERR_CUDA;
    r = finish_solve(c, st);
    if (r) return r;
    if (iterations) *iterations = c->hS->iters;
    return GFSPH_OK;
} catch (...) {  // a C++ exception never crosses the C ABI
    return GFSPH_ERR_HOST;
}

int gfsph_cg_device_ms(gfsph_cg* c, double* ms) try {
    if (!c || !ms) return GFSPH_ERR_ARG;
    *ms = c->last_ms;
    return GFSPH_OK;
} catch (...) {  // a C++ exception never crosses the C ABI
    return GFSPH_ERR_HOST;
}

int gfsph_solvegc2(int npoin, int nelem, int nnode, int ndofn, const int* intmat, int* iffix, const float* fixed,
                   const float* gstif, float* rcg, float* ficg, float tol, int* iterations) try {
    gfsph_cg* c = nullptr;
    int st = gfsph_cg_create(npoin, nelem, nnode, ndofn, intmat, gstif, &c);
    if (st) return st;
    st = gfsph_cg_solve(c, iffix, fixed, rcg, ficg, tol, iterations);
    gfsph_cg_destroy(c);
    return st;
} catch (...) {  // a C++ exception never crosses the C ABI
    return GFSPH_ERR_HOST;
}

long long gfsph_cg_launch_count(gfsph_cg* c) { return c ? c->launches : -1; }

}  // extern "C"
