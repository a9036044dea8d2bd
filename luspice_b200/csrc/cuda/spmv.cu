// Whole-GPU sparse matrix-vector products.
//
//  - spmv.h (src/spmv.h:23-57): fp64 CSR with a group of 4 lanes per row
//    (circuit matrices average 3-8 entries per row), fp64 accumulation.
//  - lusp_sell_*: SELL-C-sigma with C in {8, 16, 32}: rows sorted by length
//    inside windows of sigma rows, slices of C rows stored column-major; one
//    warp per slice, 32/C lanes per row.  Values fp64, fp32, or fp16 after
//    Ruiz equilibration (range-checked at creation), int32 indices, fp64
//    accumulation.  Padding credits nothing: the algorithmic bytes are
//    nnz*(value+index) + row pointers + x + y.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <new>
#include <numeric>
#include <vector>

#include "luspice_b200.h"
#include "spmv.h"
#include "engine_internal.h"

namespace {

constexpr int kCsrLanes = 4;

template <typename VT>
__global__ void __launch_bounds__(256)
csr_vector_kernel(int n, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                  const VT* __restrict__ values, const double* __restrict__ x,
                  double* __restrict__ y) {
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) / kCsrLanes;
    const int sub = threadIdx.x % kCsrLanes;
    double acc = 0.0;
    if (g < n) {
        // Four independent partial sums keep four loads per lane in flight
        // (long rows would otherwise wait one memory latency per entry).
        const int p1 = rowptr[g + 1];
        double a1 = 0.0, a2 = 0.0, a3 = 0.0;
        int p = rowptr[g] + sub;
        for (; p + 3 * kCsrLanes < p1; p += 4 * kCsrLanes) {
            const int c0 = colidx[p], c1 = colidx[p + kCsrLanes], c2 = colidx[p + 2 * kCsrLanes],
                      c3 = colidx[p + 3 * kCsrLanes];
            acc = fma((double)values[p], __ldg(x + c0), acc);
            a1 = fma((double)values[p + kCsrLanes], __ldg(x + c1), a1);
            a2 = fma((double)values[p + 2 * kCsrLanes], __ldg(x + c2), a2);
            a3 = fma((double)values[p + 3 * kCsrLanes], __ldg(x + c3), a3);
        }
        for (; p < p1; p += kCsrLanes) acc = fma((double)values[p], __ldg(x + colidx[p]), acc);
        acc = (acc + a1) + (a2 + a3);
    }
#pragma unroll
    for (int o = kCsrLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (g < n && sub == 0) y[g] = acc;
}

template <typename VT> __device__ __forceinline__ double ldv(const VT* p);
template <> __device__ __forceinline__ double ldv<double>(const double* p) { return __ldg(p); }
template <> __device__ __forceinline__ double ldv<float>(const float* p) { return (double)__ldg(p); }
template <> __device__ __forceinline__ double ldv<__half>(const __half* p) {
    return (double)__half2float(__ldg(p));
}

// Blocks [0, sell_blocks) take the slices, a warp each; the blocks after them
// take the long rows, LW warps per row (8: a block, or 1), lanes over its
// entries with four partial sums, fixed-order reductions.  WIDE: row numbers
// and up to eight entries per lane requested before the first is used; the
// other instances have no bound on resident blocks (one changes the order of
// their loads: a mesh of 1 M nodes 12.0 -> 16.1 us).  Which of them a product
// takes, and why, is said at sell_value.
constexpr int kWideBlocks = 4;      // resident blocks per SM of the wide instances
template <int C, bool WIDE, int LW, typename VT>
__global__ void __launch_bounds__(256, WIDE ? kWideBlocks : 0)
sell_kernel(int nslices, const int* __restrict__ ptr, const int* __restrict__ col,
            const VT* __restrict__ val, const int* __restrict__ perm,
            const double* __restrict__ x, double* __restrict__ y,
            const double* __restrict__ row_div, int sell_blocks, int nlong,
            const int* __restrict__ lrow, const int* __restrict__ lptr, const int* __restrict__ lcol,
            const VT* __restrict__ lval) {
    if ((int)blockIdx.x >= sell_blocks) {
        constexpr int T = 32 * LW;                                      // threads of a row
        __shared__ double part[8];
        const int w = (((int)blockIdx.x - sell_blocks) * 256 + (int)threadIdx.x) / T;
        if (w >= nlong) return;                                         // LW = 1: a whole warp
        const int p1 = lptr[w + 1];
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        int p = lptr[w] + (int)threadIdx.x % T;
        for (; p + 3 * T < p1; p += 4 * T) {
            const int c0 = lcol[p], c1 = lcol[p + T], c2 = lcol[p + 2 * T], c3 = lcol[p + 3 * T];
            a0 = fma(ldv<VT>(lval + p), __ldg(x + c0), a0);
            a1 = fma(ldv<VT>(lval + p + T), __ldg(x + c1), a1);
            a2 = fma(ldv<VT>(lval + p + 2 * T), __ldg(x + c2), a2);
            a3 = fma(ldv<VT>(lval + p + 3 * T), __ldg(x + c3), a3);
        }
        // At most three entries per thread are left.
        const bool b0 = p < p1, b1 = p + T < p1, b2 = p + 2 * T < p1;
        const int c0 = b0 ? lcol[p] : 0, c1 = b1 ? lcol[p + T] : 0, c2 = b2 ? lcol[p + 2 * T] : 0;
        if (b0) a0 = fma(ldv<VT>(lval + p), __ldg(x + c0), a0);
        if (b1) a1 = fma(ldv<VT>(lval + p + T), __ldg(x + c1), a1);
        if (b2) a2 = fma(ldv<VT>(lval + p + 2 * T), __ldg(x + c2), a2);
        double acc = (a0 + a1) + (a2 + a3);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (LW > 1) {
            if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
            __syncthreads();
            acc = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
        }
        if (threadIdx.x % T == 0) {
            const int row = lrow[w];
            y[row] = row_div ? acc / row_div[row] : acc;
        }
        return;
    }
    constexpr int G = 32 / C;
    const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (s >= nslices) return;
    const int lane = threadIdx.x & 31;
    const int r = lane % C, sub = lane / C;
    const int base = ptr[s];
    const int L = (ptr[s + 1] - base) / C;
    int row = -1;
    if (WIDE && sub == 0) row = perm[s * C + r];
    double acc = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (WIDE) {
        // The same sums as below: four interleaved partial sums over groups
        // of four, the rest into the first.
        for (int t = sub; t < L; t += 8 * G) {
            int c[8];
            double v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const bool in = t + q * G < L;
                const int e = base + (t + q * G) * C + r;
                c[q] = in ? col[e] : 0;
                v[q] = in ? ldv<VT>(val + e) : 0.0;
            }
#pragma unroll
            for (int h = 0; h < 8; h += 4) {
                if (t + (h + 3) * G < L) {
                    const double x0 = __ldg(x + c[h]), x1 = __ldg(x + c[h + 1]);
                    const double x2 = __ldg(x + c[h + 2]), x3 = __ldg(x + c[h + 3]);
                    acc = fma(v[h], x0, acc);
                    a1 = fma(v[h + 1], x1, a1);
                    a2 = fma(v[h + 2], x2, a2);
                    a3 = fma(v[h + 3], x3, a3);
                } else {
#pragma unroll
                    for (int q = h; q < h + 3; q++)
                        if (t + q * G < L) acc = fma(v[q], __ldg(x + c[q]), acc);
                }
            }
        }
    } else {
        int t = sub;
        for (; t + 3 * G < L; t += 4 * G) {
            const int e = base + t * C + r, d = G * C;
            const int c0 = col[e], c1 = col[e + d], c2 = col[e + 2 * d], c3 = col[e + 3 * d];
            acc = fma(ldv<VT>(val + e), __ldg(x + c0), acc);
            a1 = fma(ldv<VT>(val + e + d), __ldg(x + c1), a1);
            a2 = fma(ldv<VT>(val + e + 2 * d), __ldg(x + c2), a2);
            a3 = fma(ldv<VT>(val + e + 3 * d), __ldg(x + c3), a3);
        }
        for (; t < L; t += G) {
            const int e = base + t * C + r;
            acc = fma(ldv<VT>(val + e), __ldg(x + col[e]), acc);
        }
    }
    acc = (acc + a1) + (a2 + a3);
#pragma unroll
    for (int o = 16; o >= C; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (sub == 0) {
        if (!WIDE) row = perm[s * C + r];
        if (row >= 0) y[row] = row_div ? acc / row_div[row] : acc;
    }
}

// out = x / s elementwise (the column scaling undone on the input vector).
__global__ void unscale_kernel(int n, const double* __restrict__ x, const double* __restrict__ s,
                               double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = x[i] / s[i];
}

}  // namespace

struct SellObj {
    int n = 0, C = 32, sigma = 32, kind = 0, nslices = 0;
    long stored = 0, nnz = 0;
    int* d_ptr = nullptr;
    int* d_col = nullptr;
    void* d_val = nullptr;
    int* d_perm = nullptr;
    double* d_rs = nullptr;     // fp16: row scale
    double* d_cs = nullptr;     // fp16: column scale
    double* d_xs = nullptr;     // fp16: scaled x
    double smin = 0, smax = 0;
    // Rows much longer than the rest (supply nets) stay out of the slices
    // (one of them would set a whole slice's width): CSR.
    int nlong = 0;
    long long_stored = 0;       // entries of the long rows
    int* d_lrow = nullptr;      // [nlong] row
    int* d_lptr = nullptr;      // [nlong+1]
    int* d_lcol = nullptr;
    void* d_lval = nullptr;
};

template <int C, bool WIDE, int LW, typename VT>
static void sell_launch(const SellObj* S, int grid, int sell_blocks, const double* x, double* y, const double* rsc,
                        cudaStream_t st) {
    sell_kernel<C, WIDE, LW, VT><<<grid, 256, 0, st>>>(S->nslices, S->d_ptr, S->d_col, (const VT*)S->d_val, S->d_perm, x,
                                                       y, rsc, sell_blocks, S->nlong, S->d_lrow, S->d_lptr, S->d_lcol,
                                                       (const VT*)S->d_lval);
}

// The product's kernel (see sell_kernel).  B200, replayed graphs of 50 products
// of fp64 values, us.
//   Long rows: a block each while their blocks are resident at once (8 per SM)
//   or from 768 entries on, else a warp each, which shares the reduction's cost
//   among fewer lanes: 40,000 short rows with 100 rows of 300 entries 2.6 / 3.8
//   (block / warp), 1000 4.2 / 4.1, 2000 6.2 / 5.1, 4000 9.7 / 7.7, with 3000
//   of 700 11.8 / 10.4, 2000 of 1000 11.1 / 17.8.
//   Wide slices while every block is resident, so that a warp's latency is the
//   launch's: a mesh of 20,000 nodes 1.98 / 2.64 (wide / not), of 151,000
//   (4705 slices) 2.80 / 3.21; of 153,000 (4778) 3.44 / 3.25, of 1 M
//   13.6 / 12.0.  A long row's block counts: 140,000 short rows with 40 long
//   ones 3.3 / 3.7, with 100 4.1 / 3.7.  And for very long rows that are most of
//   the product, whose loads the 64 registers of the wide instances hold:
//   60,000 short rows with 800 of 10,000 entries 19.8 / 25.0, with 444 of 3000
//   7.8 / 7.7.
template <int C, typename VT>
static void sell_value(const SellObj* S, const double* x, double* y, const double* rsc, cudaStream_t st) {
    const int sms = lusp::sm_count(), sell_blocks = (int)(((long)S->nslices * 32 + 255) / 256);
    const bool block = S->nlong <= 8 * sms || S->long_stored >= 768L * S->nlong;
    const bool very = S->nlong > 0 && S->long_stored >= 4096L * S->nlong && 2 * S->long_stored >= S->stored;
    const int grid = sell_blocks + (block ? S->nlong : (S->nlong + 7) / 8);
    if (grid == 0) return;
    if (!block) sell_launch<C, false, 1, VT>(S, grid, sell_blocks, x, y, rsc, st);
    else if (grid <= kWideBlocks * sms || very) sell_launch<C, true, 8, VT>(S, grid, sell_blocks, x, y, rsc, st);
    else sell_launch<C, false, 8, VT>(S, grid, sell_blocks, x, y, rsc, st);
}

template <int C>
static void sell_kind(const SellObj* S, const double* x, double* y, const double* rsc, cudaStream_t st) {
    if (S->kind == 0) sell_value<C, double>(S, x, y, rsc, st);
    else if (S->kind == 1) sell_value<C, float>(S, x, y, rsc, st);
    else sell_value<C, __half>(S, x, y, rsc, st);
}

// Ruiz equilibration (max norm): alternately scale rows and columns by
// 1/sqrt(max |a|) until every row and column maximum is within tol of 1.
// Same iteration as the reference's preprocessing (bench/test_lu_gpu_f32.cu:
// 249-269), written over CSR.
void lusp_ruiz_csr(int n, const int* rowptr, const int* colidx, const double* vals, int sweeps,
                   double tol, std::vector<double>& rs, std::vector<double>& cs) {
    rs.assign(n, 1.0);
    cs.assign(n, 1.0);
    std::vector<double> cmax(n);
    for (int it = 0; it < sweeps; it++) {
        double dev = 0.0;
        for (int i = 0; i < n; i++) {
            double m = 0.0;
            for (int p = rowptr[i]; p < rowptr[i + 1]; p++) m = std::max(m, std::fabs(vals[p]) * rs[i] * cs[colidx[p]]);
            if (m > 0) { rs[i] /= std::sqrt(m); dev = std::max(dev, std::fabs(1.0 - m)); }
        }
        std::fill(cmax.begin(), cmax.end(), 0.0);
        for (int i = 0; i < n; i++)
            for (int p = rowptr[i]; p < rowptr[i + 1]; p++)
                cmax[colidx[p]] = std::max(cmax[colidx[p]], std::fabs(vals[p]) * rs[i] * cs[colidx[p]]);
        for (int j = 0; j < n; j++)
            if (cmax[j] > 0) { cs[j] /= std::sqrt(cmax[j]); dev = std::max(dev, std::fabs(1.0 - cmax[j])); }
        if (dev < tol) break;
    }
}

extern "C" {

int csr_alloc_device(const CSRMatrix* A, int** d_rowptr, int** d_colidx, double** d_values) {
    if (!A || !d_rowptr || !d_colidx || !d_values || A->n <= 0) return 1;
    const size_t nr = ((size_t)A->n + 1) * sizeof(int);
    const size_t nc = (size_t)std::max<long long>(A->nnz, 1) * sizeof(int);
    const size_t nv = (size_t)std::max<long long>(A->nnz, 1) * sizeof(double);
    *d_rowptr = nullptr;
    *d_colidx = nullptr;
    *d_values = nullptr;
    if (cudaMalloc((void**)d_rowptr, nr) != cudaSuccess) return 1;
    if (cudaMalloc((void**)d_colidx, nc) != cudaSuccess) return 1;
    if (cudaMalloc((void**)d_values, nv) != cudaSuccess) return 1;
    if (cudaMemcpy(*d_rowptr, A->rowptr, nr, cudaMemcpyHostToDevice) != cudaSuccess) return 1;
    if (A->nnz > 0) {
        if (cudaMemcpy(*d_colidx, A->colidx, (size_t)A->nnz * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) return 1;
        if (cudaMemcpy(*d_values, A->values, (size_t)A->nnz * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) return 1;
    }
    return 0;
}

void spmv_launch(int n, const int* d_rowptr, const int* d_colidx, const double* d_values,
                 const double* d_x, double* d_y, void* stream) {
    if (n <= 0) return;
    const long threads = (long)n * kCsrLanes;
    const int grid = (int)((threads + 255) / 256);
    csr_vector_kernel<double><<<grid, 256, 0, (cudaStream_t)stream>>>(n, d_rowptr, d_colidx, d_values, d_x, d_y);
}

int lusp_csr_spmv32(int n, const int* d_rowptr, const int* d_colidx, const float* d_values,
                    const double* d_x, double* d_y, void* stream) {
    if (n <= 0 || !d_rowptr || !d_colidx || !d_values || !d_x || !d_y) return LUSP_EARG;
    const long threads = (long)n * kCsrLanes;
    const int grid = (int)((threads + 255) / 256);
    csr_vector_kernel<float><<<grid, 256, 0, (cudaStream_t)stream>>>(n, d_rowptr, d_colidx, d_values, d_x, d_y);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? LUSP_OK : lusp::cuda_fail(e, "csr fp32 spmv launch");
}

int spmv_host(const CSRMatrix* A, const double* x, double* y, double* time_ms) {
    if (!A || !x || !y || A->n <= 0) return 1;
    int *dr = nullptr, *dc = nullptr;
    double *dv = nullptr, *dx = nullptr, *dy = nullptr;
    int rc = 1;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    const size_t nb = (size_t)A->n * sizeof(double);
    do {
        if (csr_alloc_device(A, &dr, &dc, &dv)) break;
        if (cudaMalloc((void**)&dx, nb) != cudaSuccess) break;
        if (cudaMalloc((void**)&dy, nb) != cudaSuccess) break;
        if (cudaMemcpy(dx, x, nb, cudaMemcpyHostToDevice) != cudaSuccess) break;
        spmv_launch(A->n, dr, dc, dv, dx, dy, 0);
        if (cudaDeviceSynchronize() != cudaSuccess) break;
        if (time_ms) {
            cudaEventCreate(&e0);
            cudaEventCreate(&e1);
            cudaEventRecord(e0, 0);
            spmv_launch(A->n, dr, dc, dv, dx, dy, 0);
            cudaEventRecord(e1, 0);
            cudaEventSynchronize(e1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            *time_ms = ms;
        }
        if (cudaGetLastError() != cudaSuccess) break;
        if (cudaMemcpy(y, dy, nb, cudaMemcpyDeviceToHost) != cudaSuccess) break;
        rc = 0;
    } while (0);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(dr);
    cudaFree(dc);
    cudaFree(dv);
    cudaFree(dx);
    cudaFree(dy);
    return rc;
}

int lusp_sell_create(int n, const int* rowptr, const int* colidx, const double* vals, int C,
                     int sigma, int value_kind, lusp_sell** out) {
    if (!out) return LUSP_EARG;
    *out = nullptr;
    if (n <= 0 || !rowptr || !colidx || !vals) return LUSP_EARG;
    if (C != 8 && C != 16 && C != 32) { lusp::set_error("sell_create: C must be 8, 16 or 32"); return LUSP_EARG; }
    if (value_kind < 0 || value_kind > 2) return LUSP_EARG;
    sigma = std::max(sigma, C);
    SellObj* S = nullptr;
    try {
        S = new SellObj();
        S->n = n;
        S->C = C;
        S->sigma = sigma;
        S->kind = value_kind;
        S->nnz = rowptr[n];
        std::vector<double> rs, cs;
        if (value_kind == 2) {
            lusp_ruiz_csr(n, rowptr, colidx, vals, 30, 1e-6, rs, cs);
            double mn = INFINITY, mx = 0.0;
            for (int i = 0; i < n; i++)
                for (int p = rowptr[i]; p < rowptr[i + 1]; p++) {
                    const double a = std::fabs(vals[p] * rs[i] * cs[colidx[p]]);
                    if (a == 0.0) continue;
                    mn = std::min(mn, a);
                    mx = std::max(mx, a);
                }
            S->smin = mn;
            S->smax = mx;
            // fp16 normal range: [2^-14, 65504].
            if (!(mn >= 6.103515625e-05) || !(mx <= 65504.0)) {
                lusp::set_error("sell_create: Ruiz-scaled values span [%.3e, %.3e], outside the fp16 normal range", mn, mx);
                delete S;
                return LUSP_EARG;
            }
        }
        std::vector<int> len(n), perm, lrows;
        for (int i = 0; i < n; i++) len[i] = rowptr[i + 1] - rowptr[i];
        // Rows longer than max(256, 8 x the mean row length) go to the long
        // list; the rest are sorted by length inside windows of sigma rows.
        const long thr = std::max<long>(256, 8 * ((rowptr[n] + n - 1) / n));
        for (int i = 0; i < n; i++) (len[i] > thr ? lrows : perm).push_back(i);
        const int nsh = (int)perm.size();
        for (int w0 = 0; w0 < nsh; w0 += sigma) {
            const int w1 = std::min(nsh, w0 + sigma);
            std::stable_sort(perm.begin() + w0, perm.begin() + w1, [&len](int a, int b) { return len[a] > len[b]; });
        }
        const int ns = (nsh + C - 1) / C;
        S->nslices = ns;
        std::vector<int> ptr(ns + 1, 0), hperm((size_t)ns * C, -1);
        for (int s = 0; s < ns; s++) {
            int ml = 0;
            for (int r = 0; r < C; r++) {
                const int k = s * C + r;
                if (k < nsh) { hperm[k] = perm[k]; ml = std::max(ml, len[perm[k]]); }
            }
            ptr[s + 1] = ptr[s] + ml * C;
        }
        const long total = ptr[ns];
        S->stored = total;
        std::vector<int> hcol(std::max<long>(total, 1), 0);
        std::vector<double> hval(std::max<long>(total, 1), 0.0);
        for (int s = 0; s < ns; s++)
            for (int r = 0; r < C; r++) {
                const int k = s * C + r;
                if (k >= nsh) continue;
                const int row = perm[k];
                const int L = (ptr[s + 1] - ptr[s]) / C;
                for (int t = 0; t < L; t++) {
                    const long e = ptr[s] + (long)t * C + r;
                    if (t < len[row]) {
                        const int p = rowptr[row] + t;
                        hcol[e] = colidx[p];
                        hval[e] = value_kind == 2 ? vals[p] * rs[row] * cs[colidx[p]] : vals[p];
                    } else {
                        hcol[e] = row < n ? row : 0;
                    }
                }
            }
        const size_t vsz = value_kind == 0 ? 8 : value_kind == 1 ? 4 : 2;
        cudaError_t e = cudaSuccess;
        e = cudaMalloc((void**)&S->d_ptr, (ns + 1) * sizeof(int));
        if (e == cudaSuccess) e = cudaMalloc((void**)&S->d_col, hcol.size() * sizeof(int));
        if (e == cudaSuccess) e = cudaMalloc(&S->d_val, hcol.size() * vsz);
        if (e == cudaSuccess) e = cudaMalloc((void**)&S->d_perm, hperm.size() * sizeof(int));
        if (e == cudaSuccess) e = cudaMemcpy(S->d_ptr, ptr.data(), (ns + 1) * sizeof(int), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(S->d_col, hcol.data(), hcol.size() * sizeof(int), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(S->d_perm, hperm.data(), hperm.size() * sizeof(int), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) {
            if (value_kind == 0) {
                e = cudaMemcpy(S->d_val, hval.data(), hval.size() * 8, cudaMemcpyHostToDevice);
            } else if (value_kind == 1) {
                std::vector<float> f(hval.size());
                for (size_t t = 0; t < f.size(); t++) f[t] = (float)hval[t];
                e = cudaMemcpy(S->d_val, f.data(), f.size() * 4, cudaMemcpyHostToDevice);
            } else {
                std::vector<__half> h(hval.size());
                for (size_t t = 0; t < h.size(); t++) h[t] = __double2half(hval[t]);
                e = cudaMemcpy(S->d_val, h.data(), h.size() * 2, cudaMemcpyHostToDevice);
            }
        }
        // Long rows: CSR in their original order, values as stored above.
        S->nlong = (int)lrows.size();
        if (e == cudaSuccess && S->nlong > 0) {
            std::vector<int> lptr(S->nlong + 1, 0), lcol;
            std::vector<double> lv;
            for (int t = 0; t < S->nlong; t++) {
                const int row = lrows[t];
                for (int p = rowptr[row]; p < rowptr[row + 1]; p++) {
                    lcol.push_back(colidx[p]);
                    lv.push_back(value_kind == 2 ? vals[p] * rs[row] * cs[colidx[p]] : vals[p]);
                }
                lptr[t + 1] = (int)lcol.size();
            }
            S->long_stored = (long)lcol.size();
            S->stored += S->long_stored;
            e = cudaMalloc((void**)&S->d_lrow, lrows.size() * sizeof(int));
            if (e == cudaSuccess) e = cudaMalloc((void**)&S->d_lptr, lptr.size() * sizeof(int));
            if (e == cudaSuccess) e = cudaMalloc((void**)&S->d_lcol, lcol.size() * sizeof(int));
            if (e == cudaSuccess) e = cudaMalloc(&S->d_lval, lv.size() * vsz);
            if (e == cudaSuccess) e = cudaMemcpy(S->d_lrow, lrows.data(), lrows.size() * sizeof(int), cudaMemcpyHostToDevice);
            if (e == cudaSuccess) e = cudaMemcpy(S->d_lptr, lptr.data(), lptr.size() * sizeof(int), cudaMemcpyHostToDevice);
            if (e == cudaSuccess) e = cudaMemcpy(S->d_lcol, lcol.data(), lcol.size() * sizeof(int), cudaMemcpyHostToDevice);
            if (e == cudaSuccess) {
                if (value_kind == 0) {
                    e = cudaMemcpy(S->d_lval, lv.data(), lv.size() * 8, cudaMemcpyHostToDevice);
                } else if (value_kind == 1) {
                    std::vector<float> f(lv.size());
                    for (size_t t = 0; t < f.size(); t++) f[t] = (float)lv[t];
                    e = cudaMemcpy(S->d_lval, f.data(), f.size() * 4, cudaMemcpyHostToDevice);
                } else {
                    std::vector<__half> h(lv.size());
                    for (size_t t = 0; t < h.size(); t++) h[t] = __double2half(lv[t]);
                    e = cudaMemcpy(S->d_lval, h.data(), h.size() * 2, cudaMemcpyHostToDevice);
                }
            }
        }
        if (e == cudaSuccess && value_kind == 2) {
            e = cudaMalloc((void**)&S->d_rs, n * sizeof(double));
            if (e == cudaSuccess) e = cudaMalloc((void**)&S->d_cs, n * sizeof(double));
            if (e == cudaSuccess) e = cudaMalloc((void**)&S->d_xs, n * sizeof(double));
            if (e == cudaSuccess) e = cudaMemcpy(S->d_rs, rs.data(), n * sizeof(double), cudaMemcpyHostToDevice);
            if (e == cudaSuccess) e = cudaMemcpy(S->d_cs, cs.data(), n * sizeof(double), cudaMemcpyHostToDevice);
        }
        if (e != cudaSuccess) {
            lusp_sell_destroy(reinterpret_cast<lusp_sell*>(S));
            return lusp::cuda_fail(e, "sell_create");
        }
    } catch (const std::bad_alloc&) {
        delete S;
        return LUSP_EALLOC;
    }
    *out = reinterpret_cast<lusp_sell*>(S);
    return LUSP_OK;
}

void lusp_sell_destroy(lusp_sell* hs) {
    SellObj* S = reinterpret_cast<SellObj*>(hs);
    if (!S) return;
    cudaFree(S->d_ptr);
    cudaFree(S->d_col);
    cudaFree(S->d_val);
    cudaFree(S->d_perm);
    cudaFree(S->d_rs);
    cudaFree(S->d_cs);
    cudaFree(S->d_xs);
    cudaFree(S->d_lrow);
    cudaFree(S->d_lptr);
    cudaFree(S->d_lcol);
    cudaFree(S->d_lval);
    delete S;
}

int lusp_sell_spmv(const lusp_sell* hs, const double* d_x, double* d_y, void* stream) {
    const SellObj* S = reinterpret_cast<const SellObj*>(hs);
    if (!S || !d_x || !d_y) return LUSP_EARG;
    cudaStream_t st = (cudaStream_t)stream;
    const double* xin = d_x;
    if (S->kind == 2) {
        // A x = Dr^-1 (Dr A Dc) (Dc^-1 x): the stored values are Dr A Dc.
        unscale_kernel<<<(S->n + 255) / 256, 256, 0, st>>>(S->n, d_x, S->d_cs, S->d_xs);
        xin = S->d_xs;
    }
    const double* rsc = S->kind == 2 ? S->d_rs : nullptr;
    if (S->C == 8) sell_kind<8>(S, xin, d_y, rsc, st);
    else if (S->C == 16) sell_kind<16>(S, xin, d_y, rsc, st);
    else sell_kind<32>(S, xin, d_y, rsc, st);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? LUSP_OK : lusp::cuda_fail(e, "sell spmv launch");
}

int lusp_sell_info(const lusp_sell* hs, long* stored, long* nnz, double* smin, double* smax) {
    const SellObj* S = reinterpret_cast<const SellObj*>(hs);
    if (!S) return LUSP_EARG;
    if (stored) *stored = S->stored;
    if (nnz) *nnz = S->nnz;
    if (smin) *smin = S->smin;
    if (smax) *smax = S->smax;
    return LUSP_OK;
}

}  // extern "C"
