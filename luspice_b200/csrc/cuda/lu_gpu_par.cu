// Single-block sparse LU with partial pivoting decided on the device, and
// its triangular solve: the kernels declared by lu_gpu_par.h.
//
// lu_factor_par_kernel: one CTA of 256 threads walks the columns in order.
// For column k the dense work vector x lives in shared memory (n doubles);
// the columns j < k that update it are discovered as a bitmap over pivot
// positions: A(:,k) seeds the bits of its pivoted rows, and every column
// applied sets the bits of the pivoted rows it touches (always at positions
// above the current one).  The lowest set bit is found with ballots, so the
// updates are applied in ascending pivot order, exactly the order of the
// single-thread reference kernel (src/lu_gpu.cu:64-77); exact zeros skip
// their column as there.  A second bitmap holds the touched rows: pivot
// search, U and L extraction walk it in row order (as a list, a lane per
// row), giving the same entry order as the single-thread kernel, and never
// look at the other rows.  Multiply and subtract are separately rounded.
//
// What bounds it: the serial chain of columns and of the dependencies inside
// one, each a few dependent loads and some hundred instructions of one warp.
// Circuit columns touch some tens of rows, so warp 0 walks them alone (no CTA
// barrier), the next column's input and the next dependency's pointers loaded
// ahead; the other warps join only for an update of more than kLongColumn
// rows.  The row permutation is kept in shared memory (16 bits: n is below
// 19,400 there).  B200, factor in ms against a CTA-wide scan of all n rows per
// column and a CTA-wide step per dependency: n = 989 circuit 7.26 -> 4.88 (a
// lane walking its word of the bitmap instead of the list: 6.85), n = 4050 grid
// 116 -> 79, dense n = 600 221 -> 192, band matrix n = 2000 with 120 diagonals
// on each side 303 -> 265.  The input's entries go in 32 at a time, in order: a
// lane looking for later duplicates of its entry took half the time of a dense
// matrix (n = 600: 410 ms).
#include <cuda_runtime.h>

#include "common.cuh"
#include "lu_gpu_par.h"

namespace {

constexpr int kThreads = 256;

// Rows of an update above which all warps share it: what one warp does in one
// step.  B200, factor in ms with 16 / 24 / 32 / 40 / 48 / 64: the n = 4050 grid
// (L columns of up to 146 rows) 80.0 / 79.6 / 79.4 / 80.4 / 81.7 / 84.1, band
// matrix n = 2000 with 60 diagonals on each side 119 / 119 / 119 / 119 / 119 /
// 133, an n = 4000 circuit with supply nets 71.9 / 71.8 / 71.7 / 72.4 / 79.4 /
// 82.7 (a CTA-wide step for every update: 117, 141, 108).
constexpr int kLongColumn = 32;
constexpr unsigned short kNone = 0xffffu;

// Inclusive prefix sum over a warp.
__device__ __forceinline__ int warp_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

}  // namespace

__global__ void __launch_bounds__(256)
lu_factor_par_kernel(int n, const int* Ap, const int* Ai, const double* Ax, const int* diagrow,
                     int* Lp, int* Li, double* Lx, long Lcap, int* Up, int* Ui, double* Ux,
                     long Ucap, int* pinv, int* xi, double* xg, int* lnnz, int* unnz,
                     int* singular_out) {
    (void)xg;
    if (blockDim.x != kThreads) {
        if (threadIdx.x == 0) *singular_out = -3;
        return;
    }
    extern __shared__ __align__(16) unsigned char lupar_smem[];
    __shared__ int s_beg, s_end, s_status;      // an update shared by all warps (s_beg < 0: none left)
    __shared__ double s_xr;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nwords = (n + 31) >> 5;
    double* x = (double*)lupar_smem;                                   // [n]
    unsigned* cand = (unsigned*)(x + n);                               // [nwords] dependencies, by pivot position
    unsigned* touched = cand + nwords;                                 // [nwords] rows of the column
    unsigned short* pos = (unsigned short*)(touched + nwords);         // [n] pivot position or kNone
    unsigned short* list = pos + n;                                    // [ncap] touched rows, ascending
    const int ncap = (int)((LU_PAR_SHARED_BYTES(n) - (size_t)((unsigned char*)list - lupar_smem)) / 2);
    int* rowat = xi;

    for (int i = tid; i < n; i += kThreads) {
        x[i] = 0.0;
        pinv[i] = -1;
        rowat[i] = -1;
        pos[i] = kNone;
    }
    for (int w = tid; w < 2 * nwords; w += kThreads) cand[w] = 0u;
    if (tid == 0) s_status = -1;
    __syncthreads();

    // x -= L(:,j) xr over entries [p0, p1), every stride-th from p0 + first.
    auto update = [&](int p0, int p1, double xr, int first, int stride) {
        for (int p = p0 + first; p < p1; p += stride) {
            const int i = Li[p];
            x[i] = __dsub_rn(x[i], __dmul_rn(Lx[p], xr));
            atomicOr(touched + (i >> 5), 1u << (i & 31));
            const int J = pos[i];
            if (J != kNone) atomicOr(cand + (J >> 5), 1u << (J & 31));
        }
    };

    long lnz = 0, unz = 0;
    if (warp == 0) {
        int status = -1;
        // Column k's input: bounds, diagonal row and this lane's first entry.
        int na0 = 0, na1 = 0, nck = 0, ni = -1;
        double nx = 0.0;
        int fb = 0, fe = 0, fd = 0;      // bounds and diagonal rows of 32 columns
        auto fetch = [&](int k) {
            if (k >= n) return;
            if ((k & 31) == 0 && k + lane < n) {
                fb = Ap[k + lane];
                fe = Ap[k + lane + 1];
                fd = diagrow[k + lane];
            }
            na0 = __shfl_sync(0xffffffffu, fb, k & 31);
            na1 = __shfl_sync(0xffffffffu, fe, k & 31);
            nck = __shfl_sync(0xffffffffu, fd, k & 31);
            ni = na0 + lane < na1 ? Ai[na0 + lane] : -1;
            nx = na0 + lane < na1 ? Ax[na0 + lane] : 0.0;
        };
        fetch(0);
        for (int k = 0; k < n; k++) {
            if (lane == 0) {
                Lp[k] = (int)lnz;
                Up[k] = (int)unz;
            }
            // 1. x = A(:,k) (assignment, the last duplicate wins) and seeds, 32
            //    entries at a time in order, the first of them loaded a column
            //    ahead: of equal rows in a group the last lane stores, and a
            //    later group stores over an earlier one.
            const int a0 = na0, a1 = na1, ck = nck, mi = ni;
            const double mx = nx;
            fetch(k + 1);
            auto seed = [&](int i, double v) {      // i < 0: no entry
                const unsigned same = __match_any_sync(0xffffffffu, i);
                if (i >= 0) {
                    if ((same >> lane) == 1u) x[i] = v;
                    atomicOr(touched + (i >> 5), 1u << (i & 31));
                    const int J = pos[i];
                    if (J != kNone) atomicOr(cand + (J >> 5), 1u << (J & 31));
                }
            };
            seed(mi, mx);
            for (int p = a0 + 32; p < a1; p += 32) {
                __syncwarp();
                const bool in = p + lane < a1;
                seed(in ? Ai[p + lane] : -1, in ? Ax[p + lane] : 0.0);
            }
            __syncwarp();
            // 2. Left-looking updates in ascending pivot position; the
            //    pointers of the next dependency known so far are loaded
            //    beside the current update.
            int pj = -1, pp0 = 0, pp1 = 0, prow = 0;
            for (int w0 = 0; w0 < nwords; w0 += 32) {
                const int w = w0 + lane;
                while (true) {
                    const unsigned bits = w < nwords ? cand[w] : 0u;
                    const unsigned any = __ballot_sync(0xffffffffu, bits != 0u);
                    if (!any) break;
                    const int src = __ffs(any) - 1;
                    const unsigned wb = __shfl_sync(0xffffffffu, bits, src);
                    const int j = ((w0 + src) << 5) + (__ffs(wb) - 1);
                    if (j != pj) {
                        pp0 = Lp[j];
                        pp1 = Lp[j + 1];
                        prow = rowat[j];
                    }
                    const int p0 = pp0 + 1, p1 = pp1;
                    const double xr = x[prow];
                    // The next set bit: in this word or the next non-empty one.
                    const unsigned rest = wb & (wb - 1u), more = any & (any - 1u);
                    const int nsrc = rest ? src : __ffs(more) - 1;
                    const unsigned nb = __shfl_sync(0xffffffffu, bits, nsrc < 0 ? 0 : nsrc);
                    pj = rest ? ((w0 + src) << 5) + (__ffs(rest) - 1)
                              : nsrc >= 0 ? ((w0 + nsrc) << 5) + (__ffs(nb) - 1) : -1;
                    if (pj >= 0) {
                        pp0 = Lp[pj];
                        pp1 = Lp[pj + 1];
                        prow = rowat[pj];
                    }
                    __syncwarp();
                    if (lane == src) cand[w] = rest;
                    __syncwarp();
                    if (xr != 0.0) {
                        if (p1 - p0 <= kLongColumn) {
                            update(p0, p1, xr, lane, 32);
                        } else {
                            if (lane == 0) {
                                s_beg = p0;
                                s_end = p1;
                                s_xr = xr;
                            }
                            __syncthreads();
                            update(p0, p1, xr, tid, kThreads);
                            __syncthreads();
                        }
                    }
                    __syncwarp();
                }
            }
            // 3. The touched rows as an ascending list, a lane per row from
            //    here on (columns that touch more rows than the list holds
            //    walk the bitmap, a lane per word).
            int rows = 0;
            for (int w0 = 0; w0 < nwords; w0 += 32) {
                const int w = w0 + lane;
                const unsigned bits = w < nwords ? touched[w] : 0u;
                const int inc = warp_scan(__popc(bits));
                int o = rows + inc - __popc(bits);
                rows += __shfl_sync(0xffffffffu, inc, 31);
                if (rows <= ncap)
                    for (unsigned b = bits; b; b &= b - 1u) list[o++] = (unsigned short)((w << 5) + __ffs(b) - 1);
            }
            __syncwarp();
            const bool listed = rows <= ncap;
            const unsigned below = (1u << lane) - 1u;
            // 4. Pivot search (largest |x|, smallest row on ties) and U(:,k),
            //    rows in ascending order.
            double bv = -1.0;
            int bi = -1;
            if (listed) {
                for (int t = 0; t < rows; t += 32) {
                    const int i = t + lane < rows ? list[t + lane] : -1;
                    const double v = i >= 0 ? x[i] : 0.0;
                    const int J = i >= 0 ? pos[i] : kNone;
                    const bool isU = J != kNone && v != 0.0;
                    if (i >= 0 && J == kNone && fabs(v) > bv) { bv = fabs(v); bi = i; }
                    const unsigned m = __ballot_sync(0xffffffffu, isU);
                    const int tot = __popc(m);
                    if (unz + tot > Ucap) {
                        status = -2;
                    } else if (isU) {
                        const long o = unz + __popc(m & below);
                        Ui[o] = J;
                        Ux[o] = v;
                    }
                    unz += tot;
                }
            } else {
                for (int w0 = 0; w0 < nwords; w0 += 32) {
                    const int w = w0 + lane;
                    const unsigned bits = w < nwords ? touched[w] : 0u;
                    int cnt = 0;
                    for (unsigned b = bits; b; b &= b - 1u) {
                        const int i = (w << 5) + __ffs(b) - 1;
                        const double v = x[i];
                        if (pos[i] == kNone) {
                            const double t = fabs(v);
                            if (t > bv) { bv = t; bi = i; }
                        } else if (v != 0.0) {
                            cnt++;
                        }
                    }
                    const int inc = warp_scan(cnt);
                    const int tot = __shfl_sync(0xffffffffu, inc, 31);
                    if (unz + tot > Ucap) {
                        status = -2;
                    } else {
                        long o = unz + inc - cnt;
                        for (unsigned b = bits; b && cnt > 0; b &= b - 1u) {
                            const int i = (w << 5) + __ffs(b) - 1;
                            const double v = x[i];
                            const int J = pos[i];
                            if (J != kNone && v != 0.0) {
                                Ui[o] = J;
                                Ux[o] = v;
                                o++;
                            }
                        }
                    }
                    unz += tot;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double v2 = __shfl_xor_sync(0xffffffffu, bv, o);
                const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
                if (v2 > bv || (v2 == bv && i2 >= 0 && (bi < 0 || i2 < bi))) { bv = v2; bi = i2; }
            }
            if (status != -1) break;
            if (bi == -1 || bv <= 0.0) { status = k; break; }
            if (pos[ck] == kNone && fabs(x[ck]) >= bv) bi = ck;
            if (unz + 1 > Ucap || lnz + 1 > Lcap) { status = -2; break; }
            const double pivot = x[bi], rpivot = __drcp_rn(pivot);
            __syncwarp();
            if (lane == 0) {
                Ui[unz] = k;
                Ux[unz] = pivot;
                pinv[bi] = k;
                pos[bi] = (unsigned short)k;
                rowat[k] = bi;
                Li[lnz] = bi;
                Lx[lnz] = 1.0;
            }
            __syncwarp();
            unz += 1;
            lnz += 1;
            // 5. L(:,k): unpivoted nonzero rows ascending, scaled by the
            //    pivot; the work vector and the bitmap are cleared on the way.
            if (listed) {
                for (int t = 0; t < rows; t += 32) {
                    const int i = t + lane < rows ? list[t + lane] : -1;
                    const double v = i >= 0 ? x[i] : 0.0;
                    const bool isL = i >= 0 && pos[i] == kNone && v != 0.0;
                    const unsigned m = __ballot_sync(0xffffffffu, isL);
                    const int tot = __popc(m);
                    if (lnz + tot > Lcap) {
                        status = -2;
                    } else if (isL) {
                        const long o = lnz + __popc(m & below);
                        Li[o] = i;
                        Lx[o] = lusp::div_by<false>(v, pivot, rpivot);
                    }
                    if (i >= 0) {
                        x[i] = 0.0;
                        touched[i >> 5] = 0u;
                    }
                    lnz += tot;
                }
            } else {
                for (int w0 = 0; w0 < nwords; w0 += 32) {
                    const int w = w0 + lane;
                    const unsigned bits = w < nwords ? touched[w] : 0u;
                    int cnt = 0;
                    for (unsigned b = bits; b; b &= b - 1u) {
                        const int i = (w << 5) + __ffs(b) - 1;
                        cnt += pos[i] == kNone && x[i] != 0.0;
                    }
                    const int inc = warp_scan(cnt);
                    const int tot = __shfl_sync(0xffffffffu, inc, 31);
                    const bool fits = lnz + tot <= Lcap;
                    if (!fits) status = -2;
                    long o = lnz + inc - cnt;
                    for (unsigned b = bits; b; b &= b - 1u) {
                        const int i = (w << 5) + __ffs(b) - 1;
                        const double v = x[i];
                        x[i] = 0.0;
                        if (fits && pos[i] == kNone && v != 0.0) {
                            Li[o] = i;
                            Lx[o] = lusp::div_by<false>(v, pivot, rpivot);
                            o++;
                        }
                    }
                    if (w < nwords) touched[w] = 0u;
                    lnz += tot;
                }
            }
            __syncwarp();
            if (status != -1) break;
            // The next column's reads see this one's entries and pointers.
            if (lane == 0) Lp[k + 1] = (int)lnz;
            __syncwarp();
        }
        if (lane == 0) {
            s_beg = -1;
            s_status = status;
            if (status == -1) {     // n = 0: written here alone
                Lp[n] = (int)lnz;
                Up[n] = (int)unz;
            }
        }
        __syncthreads();
        unz = __shfl_sync(0xffffffffu, unz, 0);
    } else {
        while (true) {
            __syncthreads();
            const int beg = s_beg;
            if (beg < 0) break;
            update(beg, s_end, s_xr, tid, kThreads);
            __syncthreads();
        }
    }
    if (s_status != -1) {
        if (tid == 0) *singular_out = s_status;
        return;
    }
    const int total = Lp[n];
    for (int p = tid; p < total; p += kThreads) Li[p] = pinv[Li[p]];
    __syncthreads();
    if (tid == 0) {
        *lnnz = (int)lnz;
        *unnz = (int)unz;
        *singular_out = -1;
    }
}

// One column sweep of trisolve over v (shared memory) by one warp.  UPPER:
// columns from the last down, v[k] = v[k] / diagonal (the column's last entry);
// else from the first up (the first entry), in both v[i] -= entry * v[k] for
// the column's other entries, separately rounded.  The pointers of 32 columns
// are loaded together, the diagonal and the first 32 CH entries of a column
// AHEAD columns ahead, so the chain of a column is the shared-memory round trip
// of v and the update; longer columns load 128 entries at a time.
template <bool UPPER, int CH, int AHEAD>
__device__ void trisolve_sweep(int n, const int* cp, const int* ci, const double* cx, double* v) {
    const int lane = threadIdx.x & 31;
    int pb = 0, pe = 0;                     // pointers of column (32 block + lane) in sweep order
    auto bounds = [&](int t, int& p0, int& p1) {   // t-th column of the sweep (t < n)
        if ((t & 31) == 0) {
            const int k = UPPER ? n - 1 - t - lane : t + lane;
            if (k >= 0 && k < n) {
                pb = cp[k];
                pe = cp[k + 1];
            }
        }
        p0 = __shfl_sync(0xffffffffu, pb, t & 31);
        p1 = __shfl_sync(0xffffffffu, pe, t & 31);
    };
    // Entries beside the diagonal: [p0 + 1, p1) of L, [p0, p1 - 1) of U.
    int p0[AHEAD], p1[AHEAD], i[AHEAD][CH];
    double e[AHEAD][CH], dg[AHEAD];
    auto fetch = [&](int t, int u) {
        bounds(t, p0[u], p1[u]);
        const int q = UPPER ? p0[u] + lane : p0[u] + 1 + lane, end = UPPER ? p1[u] - 1 : p1[u];
#pragma unroll
        for (int c = 0; c < CH; c++) {
            i[u][c] = q + 32 * c < end ? ci[q + 32 * c] : -1;
            e[u][c] = q + 32 * c < end ? cx[q + 32 * c] : 0.0;
        }
        dg[u] = cx[UPPER ? p1[u] - 1 : p0[u]];
    };
#pragma unroll
    for (int u = 0; u < AHEAD; u++)
        if (u < n) fetch(u, u);
    double rd = n > 0 ? __drcp_rn(dg[0]) : 1.0;
    for (int t0 = 0; t0 < n; t0 += AHEAD) {
#pragma unroll
        for (int u = 0; u < AHEAD; u++) {
            const int t = t0 + u;
            if (t >= n) break;
            const int k = UPPER ? n - 1 - t : t;
            const double d = dg[u], r = rd;
            const double vk = d == 1.0 ? v[k] : lusp::div_by<false>(v[k], d, r);
            __syncwarp();
            if (lane == 0) v[k] = vk;
#pragma unroll
            for (int c = 0; c < CH; c++)
                if (i[u][c] >= 0) v[i[u][c]] = __dsub_rn(v[i[u][c]], __dmul_rn(e[u][c], vk));
            const int end = UPPER ? p1[u] - 1 : p1[u];
            for (int q = (UPPER ? p0[u] : p0[u] + 1) + 32 * CH + lane; q - lane < end; q += 128) {
                int i4[4];
                double e4[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    i4[c] = q + 32 * c < end ? ci[q + 32 * c] : -1;
                    e4[c] = q + 32 * c < end ? cx[q + 32 * c] : 0.0;
                }
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (i4[c] >= 0) v[i4[c]] = __dsub_rn(v[i4[c]], __dmul_rn(e4[c], vk));
            }
            if (t + AHEAD < n) fetch(t + AHEAD, u);
            if (t + 1 < n && dg[(u + 1) % AHEAD] != 1.0) rd = __drcp_rn(dg[(u + 1) % AHEAD]);
            __syncwarp();
        }
    }
}

// The same sweep by the whole CTA for a vector in global memory: out[k] =
// in[k] / diagonal, in[i] -= entry * out[k].  A thread's first entry of the
// next column is loaded before the barrier that ends this one, the pointers a
// column earlier: n = 8000 grid 8320 -> 7470 us (B200; without the early loads
// 9120 beside the static shared memory of the small systems, which leaves less
// L1 for the vectors).
template <bool UPPER>
__device__ void trisolve_sweep_cta(int n, const int* cp, const int* ci, const double* cx, double* in, double* out) {
    const int tid = threadIdx.x, nt = blockDim.x;
    auto column = [&](int t) { return UPPER ? n - 1 - t : t; };
    int b0 = 0, b1 = 0, ni = -1;            // the next column: pointers, this thread's entry, diagonal
    double ne = 0.0, nd = 1.0;
    auto fetch = [&]() {
        const int q = UPPER ? b0 + tid : b0 + 1 + tid, end = UPPER ? b1 - 1 : b1;
        ni = q < end ? ci[q] : -1;
        ne = q < end ? cx[q] : 0.0;
        nd = cx[UPPER ? b1 - 1 : b0];
    };
    auto pointers = [&](int t, int& q0, int& q1) {
        q0 = cp[column(t)];
        q1 = cp[column(t) + 1];
    };
    int f0 = 0, f1 = 0;
    if (n > 0) pointers(0, b0, b1);
    if (n > 0) fetch();
    if (n > 1) pointers(1, f0, f1);
    for (int t = 0; t < n; t++) {
        const int k = column(t), p0 = b0, p1 = b1, i = ni;
        const double e = ne, d = nd, vk = d == 1.0 ? in[k] : __ddiv_rn(in[k], d);
        b0 = f0;
        b1 = f1;
        if (t + 1 < n) fetch();
        if (t + 2 < n) pointers(t + 2, f0, f1);
        if (tid == 0) out[k] = vk;
        if (i >= 0) in[i] = __dsub_rn(in[i], __dmul_rn(e, vk));
        const int end = UPPER ? p1 - 1 : p1;
        for (int q = (UPPER ? p0 : p0 + 1) + nt + tid; q < end; q += nt) {
            const int j = ci[q];
            in[j] = __dsub_rn(in[j], __dmul_rn(cx[q], vk));
        }
        __syncthreads();
    }
}

// Systems whose solve vector fits the kernel's static shared memory.  B200,
// us a solve against the whole CTA on a vector in global memory: n = 989 circuit
// 872 -> 514, n = 4050 grid 3961 -> 2713, dense n = 600 1429 -> 1265.
constexpr int kTriShared = 6000;
// Mean entries per column of L or U above which a sweep loads 128 entries of a
// column two columns ahead, else 32 entries four columns ahead.  B200, us a
// solve with 32 / 128: band matrices n = 2000 with 60 diagonals on each side
// 2285 / 1621, with 120 2980 / 2283, dense n = 200 248 / 217; n = 989 circuit
// (7 entries) 514 / 749, n = 4050 grid (28) 2712 / 3230.
constexpr int kTriLong = 48;

// pb = P b; L y = pb by columns (unit diagonal first); U z = y by columns
// (diagonal last); x = Q z.  Same operation sequence as splu.h:210-239, so
// the result is bitwise that of the host solve on the same factors.  Serial
// over columns; up to kTriShared unknowns one warp walks them on a vector in
// shared memory (a column costs its few dependent shared-memory accesses, no
// CTA barrier and no global round trip), larger systems with the whole CTA on
// the caller's work arrays.
__global__ void __launch_bounds__(256)
trisolve_par_kernel(int n, const int* Lp, const int* Li, const double* Lx, const int* Up,
                    const int* Ui, const double* Ux, const int* pinv, const int* q,
                    const double* b, double* x, int* work_i, double* work_d) {
    __shared__ double sv[kTriShared];
    const int tid = threadIdx.x, nt = blockDim.x;
    int* rowat = work_i;
    for (int i = tid; i < n; i += nt) rowat[i] = -1;
    __syncthreads();
    for (int i = tid; i < n; i += nt)
        if (pinv[i] >= 0) rowat[pinv[i]] = i;
    __syncthreads();
    if (n <= kTriShared) {
        for (int k = tid; k < n; k += nt) sv[k] = rowat[k] >= 0 ? b[rowat[k]] : 0.0;
        __syncthreads();
        if (tid < 32 && n > 0) {
            if (Lp[n] <= (long)kTriLong * n) trisolve_sweep<false, 1, 4>(n, Lp, Li, Lx, sv);
            else trisolve_sweep<false, 4, 2>(n, Lp, Li, Lx, sv);
            if (Up[n] <= (long)kTriLong * n) trisolve_sweep<true, 1, 4>(n, Up, Ui, Ux, sv);
            else trisolve_sweep<true, 4, 2>(n, Up, Ui, Ux, sv);
        }
        __syncthreads();
        for (int k = tid; k < n; k += nt) x[q ? q[k] : k] = sv[k];
        return;
    }
    double* pb = work_d;
    double* y = work_d + n;
    for (int k = tid; k < n; k += nt) pb[k] = rowat[k] >= 0 ? b[rowat[k]] : 0.0;
    __syncthreads();
    trisolve_sweep_cta<false>(n, Lp, Li, Lx, pb, y);
    // z overwrites pb (no longer needed).
    trisolve_sweep_cta<true>(n, Up, Ui, Ux, y, pb);
    for (int k = tid; k < n; k += nt) x[q ? q[k] : k] = pb[k];
}

extern "C" int lusp_lu_factor_par_launch(int n, const int* Ap, const int* Ai, const double* Ax,
                                         const int* diagrow, int* Lp, int* Li, double* Lx,
                                         long Lcap, int* Up, int* Ui, double* Ux, long Ucap,
                                         int* pinv, int* xi, double* xg, int* lnnz, int* unnz,
                                         int* singular_out, void* stream) {
    const size_t bytes = LU_PAR_SHARED_BYTES(n);
    cudaError_t e = cudaFuncSetAttribute(lu_factor_par_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    lu_factor_par_kernel<<<1, 256, bytes, (cudaStream_t)stream>>>(
        n, Ap, Ai, Ax, diagrow, Lp, Li, Lx, Lcap, Up, Ui, Ux, Ucap, pinv, xi, xg, lnnz, unnz,
        singular_out);
    return (int)cudaGetLastError();
}

extern "C" int lusp_trisolve_par_launch(int n, const int* Lp, const int* Li, const double* Lx,
                                        const int* Up, const int* Ui, const double* Ux,
                                        const int* pinv, const int* q, const double* b, double* x,
                                        int* work_i, double* work_d, void* stream) {
    trisolve_par_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(n, Lp, Li, Lx, Up, Ui, Ux, pinv, q, b,
                                                            x, work_i, work_d);
    return (int)cudaGetLastError();
}
