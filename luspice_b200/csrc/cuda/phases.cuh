// Per-CTA phases: refactorization of one system with frozen pivots, the
// level-scheduled triangular solves, SELL SpMV, Arnoldi and the GMRES-IR
// driver.  Every function here is called by all threads of the CTA.
#pragma once
#include <cooperative_groups.h>

#include <type_traits>

#include "engine.cuh"

namespace lusp {

// Shared-memory map of one CTA (byte offsets inside the dynamic region).
struct Smem {
    int* ctl;            // [0] claim counter, [1] status bits, [2] singular col,
                         // [3] wait-abort flag
    unsigned* ready;     // ready bits
    double* red;         // 40 doubles of reduction scratch
    char* uni;           // phase-specific area

    __device__ Smem(char* base, const SmemPlan& plan) {
        ctl = (int*)base;
        ready = (unsigned*)(base + 64);
        size_t off = 64 + (((size_t)plan.nwords * 4 + 15) & ~(size_t)15);
        red = (double*)(base + off);
        uni = base + off + 40 * sizeof(double);
    }
};

// Status bits that describe a solve (cleared when a new solve starts).
constexpr int kSolveBits = ST_STAGNATED | ST_NOT_CONVERGED | ST_NONFINITE | ST_WAIT_TIMEOUT | ST_FP16_OFF;

// Slot of row i among rows[lo, hi) (ascending), or -1.
__device__ __forceinline__ int find_slot(const int* rows, int lo, int hi, int i) {
    const int end = hi;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (rows[mid] < i) lo = mid + 1; else hi = mid;
    }
    return (lo < end && rows[lo] == i) ? lo : -1;
}

// Asynchronous global->shared copies (sm_80+ cp.async, L1-allocating):
// issued without waiting, completed by cp_async_wait_all().
__device__ __forceinline__ void cp_async_4(void* sdst, const void* gsrc) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_8(void* sdst, const void* gsrc) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_16(void* sdst, const void* gsrc) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_val(float* sdst, const float* gsrc) { cp_async_4(sdst, gsrc); }
__device__ __forceinline__ void cp_async_val(double* sdst, const double* gsrc) { cp_async_8(sdst, gsrc); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Orders this thread's memory operations for the other CTAs sharing a
// system: block scope for a lone CTA, cluster scope when the system's
// columns are spread over a thread-block cluster (release before publishing
// a ready bit, acquire after observing one).
__device__ __forceinline__ void share_fence(unsigned csize) {
    if (csize > 1) asm volatile("fence.acq_rel.cluster;\n" ::: "memory");
    else __threadfence_block();
}
// GPU scope: CTAs on any SM share the system (spread mode).  The release
// pattern (column values, then its ready bit) needs only a release fence
// before the relaxed atomic that sets the bit, and the acquire pattern (a
// ready bit read, then the column's values) only an acquire fence after the
// read; neither has to wait the way a full acq_rel or sequentially
// consistent fence does (grid refactor 1.68 -> 1.55 ms).
template <bool SPREAD>
__device__ __forceinline__ void share_release_t(unsigned csize) {
    if (SPREAD) asm volatile("fence.release.gpu;\n" ::: "memory");
    else share_fence(csize);
}
__device__ __forceinline__ void spread_acquire() { asm volatile("fence.acquire.gpu;\n" ::: "memory"); }

__device__ __forceinline__ int warp_claim(int* counter) {
    int idx = 0;
    if ((threadIdx.x & 31) == 0) idx = atomicAdd(counter, 1);
    return __shfl_sync(0xffffffffu, idx, 0);
}

// Pivot statistics of a CTA: warp reductions, then per-warp partials
// combined in order by thread 0.  first: overwrite the system's statistics
// (refactor kernel), else merge into them (dense trailing-block kernel).
// Status bits go through ctl[1], the singular column through ctl[2] (the
// CTA's own control words, or those of the cluster's rank 0).
__device__ void cta_store_pivot_stats(SysStats* st, Smem& sm, double minpiv, double minratio, double maxu,
                                      int bad, bool first, int* ctl) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    minpiv = warp_min(minpiv);
    minratio = warp_min(minratio);
    maxu = warp_max(maxu);
    bad = __reduce_or_sync(0xffffffffu, bad);
    __syncthreads();
    if (lane == 0) {
        sm.red[warp] = minpiv;
        atomicOr(&ctl[1], bad);
    }
    __syncthreads();
    double a = INFINITY;
    if (threadIdx.x == 0)
        for (int w = 0; w < nw; w++) a = fmin(a, sm.red[w]);
    __syncthreads();
    if (lane == 0) sm.red[warp] = minratio;
    __syncthreads();
    double b = INFINITY;
    if (threadIdx.x == 0)
        for (int w = 0; w < nw; w++) b = fmin(b, sm.red[w]);
    __syncthreads();
    if (lane == 0) sm.red[warp] = maxu;
    __syncthreads();
    if (threadIdx.x == 0) {
        double c = 0.0;
        for (int w = 0; w < nw; w++) c = fmax(c, sm.red[w]);
        const int c2 = *(volatile int*)&ctl[2];
        const int sc = c2 == 0x7fffffff ? -1 : c2;
        if (first) {
            st->min_abs_pivot = a;
            st->min_pivot_ratio = b;
            st->max_abs_u = c;
            st->status = *(volatile int*)&ctl[1];
            st->singular_col = sc;
            st->nres = 0;
            st->inner_iters = 0;
            st->outer_iters = 0;
        } else {
            st->min_abs_pivot = fmin(st->min_abs_pivot, a);
            st->min_pivot_ratio = fmin(st->min_pivot_ratio, b);
            st->max_abs_u = fmax(st->max_abs_u, c);
            st->status |= *(volatile int*)&ctl[1];
            if (sc >= 0 && (st->singular_col < 0 || sc < st->singular_col)) st->singular_col = sc;
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Dense trailing block of the refactorization (rows and columns [k0, n)).
// On entry W (fp64, block columns of 32: entry (r, c) at tail_index) holds
// the block after the updates from the columns before k0, in the entries of
// its pattern; the rest of W is undefined and read as 0.
//
// Left-looking by block columns of 32.  A CTA holds one block column in
// shared memory ([D][33] fp64), applies the finished panels before it, and
// factors it as the next panel.  An entry receives its updates in ascending
// order of the pivot column, each a separately rounded multiply and subtract
// with the stored (VT-rounded) multiplier and the fp64 U value, so the
// factor equals the column engine's bit for bit.  Pivot statistics as in the
// column engine.
//
// What bounds it: the chain panel -> update of the next block column ->
// next panel.  A thread keeps its row of the panel in registers, so a panel
// column reads only the pivot row from shared memory.  In the updates a lane
// keeps its column of the panel's U block in registers and the multipliers
// are broadcast from shared memory (one 16-byte load per two multiply-subtract
// pairs of a warp), which takes the load pipe about twice the fp64 pipe's time.  Warps other than the last stream
// their own rows of the panel (four rows of 256 bytes per copy group) with
// no CTA barrier; the last warp solves the next panel's 32 x 32 unit-lower
// block for U meanwhile.  CL: the two CTAs of a cluster take the block
// columns in turn; a finished panel is published through W (L2) and a
// counter in both CTAs' shared memory.
// B200, event times per launch: 50 systems with D = 320 (n = 4050 grid)
// 0.652 -> 0.438 ms, one system with D = 96 (n = 113 circuit) 155 -> 94 us,
// 768 systems with D up to 128 on lone CTAs 0.70 -> 0.27 ms, against a
// right-looking version with the panel in shared memory (a lane per row,
// 1.4-1.7 k cycles a column) and the trailing block in global memory.  The
// floor is the fp64 pipe: D^3 / 3 pairs at 32 per cycle and SM, 90 us for
// D = 320 on two SMs.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void named_sync(int id, int threads) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int threads) {
    __syncwarp();
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}
// Named barriers of the dense kernel: U block of a panel ready, rows of the
// next U block updated, and one for each four pivot rows of a panel.
constexpr int kBarU = 1, kBarRows = 2, kBarPivots = 3;
// Control word of Smem::ctl: panels finished (both CTAs of a cluster).
constexpr int kCtlPanels = 8;

// Bounded wait until the published panels reach `want` (every lane of a warp
// calls; the acquire orders the panel's reads after it).
__device__ __forceinline__ bool dense_wait_panel(int* ctl, int want, bool cluster) {
    const volatile int* done = ctl + kCtlPanels;
    const volatile int* ab = ctl + 3;
    bool ok = true;
    for (long long it = 0; *done < want; it++) {
        if (*ab || it > kSpinLimit) {
            atomicExch(ctl + 3, 1);
            ok = false;
            break;
        }
        __nanosleep(20);
    }
    ok = __all_sync(0xffffffffu, ok);
    share_fence(cluster ? 2u : 1u);
    return ok;
}

// Four rows (1 KB, contiguous) of a finished panel into shared memory, two
// 16-byte pieces per lane that bypass L1 (another SM may have written them).
__device__ __forceinline__ void dense_copy_rows(double* dst, const double* src, int rows) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int piece = lane + 32 * q;   // 16 pieces per row
        if ((piece >> 4) < rows) cp_async_16(dst + 2 * piece, src + 2 * piece);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// The phases below keep a row or a column of 32 fp64 values in registers;
// each is a call, so its registers are its own.  The substitutions are rolled
// loops over groups of four pivots whose update writes entry q to register
// q - 4: 4.8 k cycles for 32 columns (B200) with an eighth of the unrolled
// instructions; over single pivots 7.3 k (the loop's branches and the
// shared-memory latency are paid 32 times instead of 8).
//
// Forward substitution with the lower triangle at lk (row r at lk + pitch r),
// one column per lane in u.  EXACT: unit diagonal, separately rounded
// multiply and subtract (U rows of a panel); the solution of row r goes to
// out[33 r].  Else fma and a division by the diagonal (its reciprocal at
// lk + pitch r + 32): inverses, stored as VT to out[r * step].
template <bool EXACT, typename OT>
__device__ __forceinline__ void dense_substitute(const double* lk, int pitch, double (&u)[32], OT* out, int step) {
    auto sub = [](double a, double l, double x) { return EXACT ? __dsub_rn(a, __dmul_rn(l, x)) : fma(-l, x, a); };
#pragma unroll 1
    for (int c = 0; c < 32; c += 4) {
        const double* lc = lk + (size_t)c * pitch + c;   // L[c + i][c + k] at lc + pitch i + k
        auto fin = [&](int i) {
            if (!EXACT) u[i] = div_by(u[i], lc[(size_t)i * pitch + i], lk[(size_t)(c + i) * pitch + 32]);
        };
        fin(0);
#pragma unroll
        for (int i = 1; i < 4; i++) {
#pragma unroll
            for (int k = 0; k < i; k++) u[i] = sub(u[i], lc[(size_t)i * pitch + k], u[k]);
            fin(i);
        }
        const double u0 = u[0], u1 = u[1], u2 = u[2], u3 = u[3];
        out[(c + 0) * step] = ValTraits<OT>::to(u0);
        out[(c + 1) * step] = ValTraits<OT>::to(u1);
        out[(c + 2) * step] = ValTraits<OT>::to(u2);
        out[(c + 3) * step] = ValTraits<OT>::to(u3);
#pragma unroll
        for (int m = 4; m < 32; m += 4) {
            if (m < 32 - c) {
#pragma unroll
                for (int q = m; q < m + 4; q++) {
                    const double2 a = *(const double2*)(lc + (size_t)q * pitch);
                    const double2 b = *(const double2*)(lc + (size_t)q * pitch + 2);
                    u[q - 4] = sub(sub(sub(sub(u[q], a.x, u0), a.y, u1), b.x, u2), b.y, u3);
                }
            }
        }
    }
}

// u := L^-1 u for the unit-lower 32 x 32 block at lk (row r at lk + 32 r),
// one column per lane (u[r] at xk + 33 r).
__device__ __noinline__ void dense_solve_unit(const double* lk, double* xk) {
    double u[32];
#pragma unroll
    for (int r = 0; r < 32; r++) u[r] = xk[r * 33];
    dense_substitute<true>(lk, 32, u, xk, 33);
}

// Inverse of the 32 x 32 lower triangle at lk (row r at lk + 34 r, reciprocal
// diagonal at lk + 34 r + 32), a column per lane: element (r, lane) as VT at
// out[r * step].
template <typename VT>
__device__ __noinline__ void dense_block_inverse(const double* lk, VT* out, int step) {
    const int lane = threadIdx.x & 31;
    double u[32];
#pragma unroll
    for (int r = 0; r < 32; r++) u[r] = r == lane ? 1.0 : 0.0;
    dense_substitute<false>(lk, 34, u, out, step);
}

// Rows [rb, D) of the block column xs minus the panel rows src (row r at
// src + 32 r) times the panel's U block (column of this lane at xk + 33 c),
// four rows per group, groups warp, warp + nup, ...; my: this warp's stages.
// told: barrier kBarRows needs no arrival after this warp's groups below 8.
__device__ __noinline__ void dense_update_rows(double* xs, const double* xk, const double* src, double* my, int rb,
                                               int D, int nup, int stg, int nt, bool told) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ng = (D - rb + 3) >> 2;
    auto issue = [&](int g, int slot) {
        if (g < ng) dense_copy_rows(my + slot * 128, src + (size_t)(rb + 4 * g) * 32, D - rb - 4 * g);
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int t = 0; t < stg; t++) issue(warp + t * nup, t);
    named_sync(kBarU, nt);
    double u[32];
#pragma unroll
    for (int c = 0; c < 32; c++) u[c] = xk[c * 33];
    int slot = 0;
    for (int g = warp; g < ng; g += nup) {
        if (!told && g >= 8) {
            named_arrive(kBarRows, 32 * (min(8, nup) + 1));
            told = true;
        }
        if (stg >= 3) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
        else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncwarp();
        const double* l = my + slot * 128;
        const int row = rb + 4 * g;
        double a[4];
#pragma unroll
        for (int q = 0; q < 4; q++) a[q] = xs[(size_t)min(row + q, D - 1) * 33 + lane];
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const double2 lv = *(const double2*)(l + q * 32 + c);
                a[q] = __dsub_rn(a[q], __dmul_rn(lv.x, u[c]));
                a[q] = __dsub_rn(a[q], __dmul_rn(lv.y, u[c + 1]));
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (row + q < D) xs[(size_t)(row + q) * 33 + lane] = a[q];
        __syncwarp();
        issue(g + stg * nup, slot);
        slot = slot + 1 < stg ? slot + 1 : 0;
    }
    if (!told) named_arrive(kBarRows, 32 * (min(8, nup) + 1));
    cp_async_wait_all();
    __syncwarp();
}

// A panel of R rows (row r at xj + 33 r) and w columns.  Warp 0 factors the
// 32 pivot rows alone (a row per lane in registers, the pivot row exchanged
// through shared memory); the other warps (a row per lane, rows past the
// CTA's threads in later passes) follow four columns behind it, held only by
// one named barrier per four columns.  Their loop writes entry q to register
// q - 4, so it is rolled and the current columns are registers 0..3.  Bound by
// warp 0's chain (exchange, reciprocal 61, quotient 50, update 16 cycles a
// column, and its own update's issue): 320 rows and 32 columns 24 k cycles
// (B200, alone; in the kernel a panel and its publication take 35 k on average
// over a block of 320 and 48 k over one of 96); all warps in step, a barrier
// per column, 39 k; groups of four pivots eliminated redundantly by every lane
// 34 k (two dependent divisions per column instead of one).
// ud: the pivot rows, entry (r, 4 (r / 4) + q) at ud + 34 r + q, the pivot's
// reciprocal at ud + 34 r + 32.  vmax[c]: bits of the largest entry of column
// c below the pivot before scaling, over the entries above the pivot in
// magnitude (the others do not count for its ratio).  Ends with a CTA barrier.
template <typename VT>
__device__ __noinline__ void dense_panel(double* xj, double* ud, unsigned long long* vmax, int R, int w) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int pw = (min(R, nt) + 31) >> 5;
    auto scale = [](double v, double p, double rp) { return (double)ValTraits<VT>::to(div_by(v, p, rp)); };
    auto sub = [](double a, double l, double u) { return __dsub_rn(a, __dmul_rn(l, u)); };
    auto note = [&](int c, double v, double p) {
        if (fabs(v) > fabs(p)) atomicMax(vmax + c, (unsigned long long)__double_as_longlong(fabs(v)));
    };
    if (tid < 32) vmax[tid] = 0ull;
    __syncthreads();
    double x[32];
    if (warp == 0) {
        double* row = xj + (size_t)min(lane, R - 1) * 33;
#pragma unroll
        for (int c = 0; c < 32; c++) x[c] = lane < R ? row[c] : 0.0;
#pragma unroll
        for (int c = 0; c < 32; c++) {
            if (c < w) {
                constexpr int kAlign = ~3;
                double* uc = ud + c * 34 - (c & kAlign);   // entry (c, q) at uc + q
                if (lane == c) {
#pragma unroll
                    for (int q = c & kAlign; q < 32; q += 2) *(double2*)(uc + q) = make_double2(x[q], x[q + 1]);
                }
                const double p = __shfl_sync(0xffffffffu, x[c], c), rp = __drcp_rn(p);
                if (lane == 0) ud[c * 34 + 32] = rp;
                __syncwarp();
                if (lane > c) {
                    const double l = scale(x[c], p, rp);
                    note(c, x[c], p);
                    x[c] = l;
                    if (!(c & 1)) x[c + 1] = sub(x[c + 1], l, uc[c + 1]);
#pragma unroll
                    for (int q = (c + 2) & ~1; q < 32; q += 2) {
                        const double2 u = *(const double2*)(uc + q);
                        x[q] = sub(x[q], l, u.x);
                        x[q + 1] = sub(x[q + 1], l, u.y);
                    }
                }
            }
            if ((c & 3) == 3 && (c & ~3) < w && pw > 1) named_arrive(kBarPivots + (c >> 2), 32 * pw);
        }
        __syncwarp();
        if (lane < R) {
#pragma unroll
            for (int c = 0; c < 32; c++) row[c] = x[c];
        }
    }
    for (int r0 = warp * 32 + (warp == 0 ? nt : 0); r0 < R; r0 += nt) {
        const int r = r0 + lane;
        double* row = xj + (size_t)min(r, R - 1) * 33;
#pragma unroll
        for (int c = 0; c < 32; c++) x[c] = r < R ? row[c] : 0.0;
#pragma unroll 1
        for (int c = 0; c < w; c += 4) {
            const double* uc = ud + c * 34;
            if (r0 < nt) named_sync(kBarPivots + (c >> 2), 32 * pw);
            double v[4], l[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                v[k] = x[k];
                l[k] = scale(x[k], uc[k * 34 + k], uc[k * 34 + 32]);
#pragma unroll
                for (int q = k + 1; q < 4; q++) x[q] = sub(x[q], l[k], uc[k * 34 + q]);
            }
#pragma unroll
            for (int m = 4; m < 32; m += 4) {
                if (m < 32 - c) {
                    double y[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) y[q] = x[m + q];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const double2 e = *(const double2*)(uc + k * 34 + m);
                        const double2 f = *(const double2*)(uc + k * 34 + m + 2);
                        y[0] = sub(y[0], l[k], e.x);
                        y[1] = sub(y[1], l[k], e.y);
                        y[2] = sub(y[2], l[k], f.x);
                        y[3] = sub(y[3], l[k], f.y);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) x[m + q - 4] = y[q];
                }
            }
            if (r < R) {
#pragma unroll
                for (int k = 0; k < 4; k++) row[c + k] = l[k];
            }
            if (r < R) {
#pragma unroll
                for (int k = 0; k < 4; k++) note(c + k, v[k], uc[k * 34 + k]);
            }
        }
    }
    __syncthreads();
}

// The dense trailing block of one system (its own kernel: few warps, many
// registers each): factor, VT storage for the solves (column-major, unit L
// below the diagonal), inverses of its diagonal blocks, pivot statistics.
template <typename VT, bool CL = false>
__device__ void dense_phase(const SysDev& S, const SmemPlan& plan, char* smem_base, const SolveParams& prm) {
    namespace cgr = cooperative_groups;
    const PatternDev& P = *S.pat;
    if (P.dtail <= 0) return;
    Smem sm(smem_base, plan);
    const int rank = CL ? (int)cgr::this_cluster().block_rank() : 0;
    const int nranks = CL ? 2 : 1;
    const int D = P.dtail, ld = P.tail_ld, k0 = P.k0, nbk = ld >> 5;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int nup = nw - 1;                       // warps that update rows
    double* xs = (double*)sm.uni;                 // [drows][33] the block column
    double* ud = xs + (size_t)plan.drows * 33;     // [32][34] pivot rows of the panel
    double* lk = ud;                              // [32][32] panel diagonal block (update phase)
    double* ring = ud + 32 * 34;                  // [nup][dstg][4][32] panel rows in flight
    unsigned long long* vmax = (unsigned long long*)ring;   // [32] column maxima (panel phase)
    if (tid == 0) {
        sm.ctl[1] = 0;
        sm.ctl[2] = 0x7fffffff;
        sm.ctl[3] = 0;
        sm.ctl[kCtlPanels] = 0;
    }
    if (CL) cgr::this_cluster().sync();
    else __syncthreads();
    double* W = S.tailw;
    VT* T = (VT*)S.tail;
    double minpiv = INFINITY, minratio = INFINITY, maxu = 0.0;
    int bad = 0;
    long long c_panel = 0, c_update = 0, c_store = 0, tc = clock64();

    for (int j = rank; j < nbk; j += nranks) {
        const int w = min(32, D - 32 * j), R = D - 32 * j;
        double* Wj = W + (size_t)j * D * 32;
        // The block column from W, entries outside the pattern as 0.
        for (int r0 = warp * 4; r0 < D; r0 += nw * 4) {
            unsigned m[4];
            double v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) m[q] = r0 + q < D ? __ldg(P.tail_mask + (size_t)(r0 + q) * nbk + j) : 0u;
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = (m[q] >> lane) & 1u ? __ldcg(Wj + (size_t)(r0 + q) * 32 + lane) : 0.0;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (r0 + q < D) xs[(size_t)(r0 + q) * 33 + lane] = v[q];
        }
        __syncthreads();

        // Panels 0 .. j - 1 applied in order.
        if (warp == nup) {
            for (int k = 0; k < j; k++) {
                if (!dense_wait_panel(sm.ctl, k + 1, CL)) bad |= ST_WAIT_TIMEOUT;
                const double* src = W + (size_t)k * D * 32 + (size_t)(32 * k) * 32;
#pragma unroll 4
                for (int t = lane; t < 512; t += 32) cp_async_16(lk + 2 * t, src + 2 * t);
                // Rows of this U block updated by the panel before.
                if (k > 0) named_sync(kBarRows, 32 * (min(8, nup) + 1));
                cp_async_wait_all();
                __syncwarp();
                dense_solve_unit(lk, xs + (size_t)(32 * k) * 33 + lane);
                named_arrive(kBarU, nt);
            }
        } else {
            double* my = ring + (size_t)warp * plan.dstg * 128;
            for (int k = 0; k < j; k++) {
                if (!dense_wait_panel(sm.ctl, k + 1, CL)) bad |= ST_WAIT_TIMEOUT;
                dense_update_rows(xs, xs + (size_t)(32 * k) * 33 + lane, W + (size_t)k * D * 32, my, 32 * (k + 1), D,
                                  nup, plan.dstg, nt, k + 1 >= j || warp >= 8);
            }
        }
        __syncthreads();
        if (tid == 0) {
            const long long t2 = clock64();
            c_update += t2 - tc;
            tc = t2;
        }
        double* xj = xs + (size_t)(32 * j) * 33;
        dense_panel<VT>(xj, ud, vmax, R, w);
        // Publish the panel: its rows to W, then the counters.
        if (j + 1 < nbk) {
            for (int t = tid; t < R * 32; t += nt) {
                const int r = 32 * j + (t >> 5);
                Wj[(size_t)r * 32 + lane] = xs[(size_t)r * 33 + lane];
            }
            __syncthreads();
            if (tid == 0) {
                share_fence(CL ? 2u : 1u);
                *(volatile int*)(sm.ctl + kCtlPanels) = j + 1;
                if (CL) *(volatile int*)cgr::this_cluster().map_shared_rank(sm.ctl + kCtlPanels, rank ^ 1) = j + 1;
            }
        }
        if (tid == 0) {
            const long long t2 = clock64();
            c_panel += t2 - tc;
            tc = t2;
        }
        // Off the chain: statistics, VT storage, inverses.
        if (tid < w) {
            const int c = tid;
            const double piv = ud[c * 34 + (c & 3)];
            const double ap = fabs(piv);
            const double amax = __longlong_as_double((long long)vmax[c]);
            if (!(ap > 0.0) || !isfinite(piv)) {
                bad |= ST_SINGULAR;
                atomicMin(&sm.ctl[2], k0 + 32 * j + c);
            }
            minpiv = fmin(minpiv, ap);
            const double ratio = amax > ap ? ap / amax : 1.0;
            minratio = fmin(minratio, ratio);
            if (ratio < prm.pivot_tol) bad |= ST_PIVOT_WEAK;
        }
        for (int c = warp; c < w; c += nw) {
            const int col = 32 * j + c;
            for (int i = lane; i < ld; i += 32) {
                const double v = i < D ? xs[(size_t)i * 33 + c] : 0.0;
                if (i <= col) maxu = fmax(maxu, fabs(v));
                T[(size_t)col * ld + i] = ValTraits<VT>::to(v);
            }
        }
        __syncthreads();
        if (tid == 0) {
            const long long t2 = clock64();
            c_store += t2 - tc;
            tc = t2;
        }
    }
    // Inverses of the diagonal blocks, once every block column is stored: a
    // warp per block and factor, over both CTAs of a cluster.  The factors
    // are read as the solves read them (VT-rounded): unit L and, rows and
    // columns reversed, U are two lower triangles; the identity past a
    // partial block.  Element (i, c) of an inverse at c * 32 + i.
    if (CL) cgr::this_cluster().sync();
    const int ntile = plan.dinv;
    if (warp < ntile) {
        double* bs = xs + (size_t)warp * 32 * 34;   // [32][34], reciprocal diagonal in column 32
        for (int task = rank + nranks * warp; task < 2 * nbk; task += nranks * ntile) {
            const int j = task >> 1, up = task & 1, w = min(32, D - 32 * j);
            const VT* blk = T + (size_t)(32 * j) * ld + 32 * j;
            // Column by column (contiguous in T): lane = row.
            const int r = up ? 31 - lane : lane;
            double dg = 1.0;
#pragma unroll 8
            for (int cc = 0; cc < 32; cc++) {
                const bool in = lane < w && cc < w && (up || lane != cc);
                double v = lane == cc ? 1.0 : 0.0;
                if (in) v = ValTraits<VT>::load_cg(blk + (size_t)cc * ld + lane);
                const int c = up ? 31 - cc : cc;
                if (c <= r) bs[r * 34 + c] = v;
                if (c == r) dg = v;
            }
            bs[r * 34 + 32] = __drcp_rn(dg);
            __syncwarp();
            VT* inv = (VT*)S.tinv + (size_t)j * 2048 + up * 1024;
            if (!up) dense_block_inverse<VT>(bs, inv + lane * 32, 1);
            else dense_block_inverse<VT>(bs, inv + (31 - lane) * 32 + 31, -1);
            __syncwarp();
        }
    }
    // Statistics: rank 0 merges, then rank 1; the cluster barriers also keep
    // each CTA's shared memory alive until the other is done with it.
    for (int r = 0; r < nranks; r++) {
        if (rank == r) cta_store_pivot_stats(S.stats, sm, minpiv, minratio, maxu, bad, false, sm.ctl);
        if (CL) cgr::this_cluster().sync();
    }
    if (tid == 0 && rank == 0) {
        S.stats->cyc_tpanel = c_panel;
        S.stats->cyc_ttrsm = c_store;
        S.stats->cyc_tupdate = c_update;
    }
}

// ---------------------------------------------------------------------------
// Refactorization with the pivot order and pattern frozen.
//
// Column k (one warp): x = A(:,k) scattered into the column's own slots
// (duplicates summed in input order); for each U(:,k) row j ascending, once
// column j is ready: x[s] -= L(i,j) * x[j] for the strict-L entries (i, j),
// s = slot of row i in column k; U(:,k) = x[rows < k], U(k,k) = x[k], L(:,k) =
// x[rows > k] / U(k,k).  The work vector is fp64; multiply and subtract are
// separately rounded so the result is bitwise reproducible on the host.
// Values are stored as VT (fp32 for the mixed path, fp64 for the plain path):
// the strict-L part packed by columns (the later columns' gathers read it,
// published first), in the merged layout, and in the row-major copies used by
// the solves.
//
// The dependencies are applied in segments of consecutive columns of one
// supernode (PatternDev::seg): a lane keeps its rows' x in registers over the
// segment, the dependencies' own x are exchanged by shuffles, and only the
// first dependency's row slots are read.  The n = 4050 grid has 3.5
// dependencies per segment (23 k segments for 81 k dependencies of 41 rows),
// the n = 40,000 circuit more, analog circuits 1.4.  Staging every
// dependency's values and slots through shared memory took 250 instructions
// per dependency and filled 57 % of the issue slots; what bounds the refactor
// now is the chain of columns for few systems (a ready bit seen, the L values
// from L2, the update, the division, the release fence: ~7 k cycles a level
// on the grid against ~2 k for the bare round trips) and instructions per
// column for many.  B200, refactor kernel: 50 grids 1.54 -> 0.99 ms (fp64
// 1.59 -> 1.10), one grid 1.25 -> 0.81 ms, the n = 40,000 circuit 43.7 ->
// 17.4 ms, 50 circuits n = 989 263 -> 218 us, 768 uneven circuits 4.80 ->
// 4.13 ms.
//
// Shared memory per warp: the column's record, pivot minima, x[wcap] (fp64).
// ---------------------------------------------------------------------------
// One segment's update: dependencies [a, a + W) of a segment whose first
// dependency has slot u0 and its cnt strict-L rows packed from lp0, their
// slots at rel.  Row i of the update is dependency a itself (i = 0) or its
// strict-L row i - 1; it takes part in the steps t < i (dependency a + t),
// whose L value of row i > t is at pl[i], pl moving on by the column's length.
// An L value of a finished column.  LONE: written by this CTA, so the SM's own
// L1 has it; else past L1 (another SM may have written it).
template <bool LONE, typename VT>
__device__ __forceinline__ VT load_l(const VT* p) { return LONE ? *p : __ldcg(p); }

template <typename VT, bool TWO, bool LONE>
__device__ __forceinline__ void seg_rows(const VT* lcol, const unsigned short* rel, double* x, int u0, int a, int W,
                                         int lp0, int cnt) {
    const int lane = threadIdx.x & 31, R = cnt - a + 1;
    const int la = lane < R ? lane : -1;      // steps t < la update row lane
    const bool lb = TWO && lane + 32 < R;
    const VT* pl = lcol + (lp0 + a * cnt - ((a * (a - 1)) >> 1) - 1 + lane);
    int step = cnt - a - 1;
    const int sa = la > 0 ? (int)__ldg(rel + a + lane - 1) : u0 + a;
    const int sb = lb ? (int)__ldg(rel + a + lane + 31) : 0;
    double xa = 0.0, xb = 0.0;
    for (int t0 = 0; t0 < W; t0 += 4) {
        VT va[4], vb[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (t0 + q >= W) break;
            va[q] = t0 + q < la ? load_l<LONE>(pl) : VT(0);
            if (TWO) vb[q] = lb ? load_l<LONE>(pl + 32) : VT(0);
            pl += step;
            step--;
        }
        if (t0 == 0) {
            xa = x[sa];
            if (TWO) xb = x[sb];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (t0 + q >= W) break;
            const double xj = __shfl_sync(0xffffffffu, xa, t0 + q);
            if (xj != 0.0) {
                if (t0 + q < la) xa = __dsub_rn(xa, __dmul_rn((double)va[q], xj));
                if (lb) xb = __dsub_rn(xb, __dmul_rn((double)vb[q], xj));
            }
        }
    }
    if (la > 0) x[sa] = xa;
    if (lb) x[sb] = xb;
    if (!TWO) return;
    // Rows from 64 on, 64 at a time, with the dependencies' final x.
    for (int i0 = 64; i0 < R; i0 += 64) {
        const bool pa = i0 + lane < R, pb = i0 + lane + 32 < R;
        const VT* ph = lcol + (lp0 + a * cnt - ((a * (a - 1)) >> 1) - 1 + lane + i0);
        int hs = cnt - a - 1;
        const int ra = pa ? (int)__ldg(rel + a + i0 + lane - 1) : 0, rb = pb ? (int)__ldg(rel + a + i0 + lane + 31) : 0;
        double ya = x[ra], yb = x[rb];
        for (int t0 = 0; t0 < W; t0 += 4) {
            VT va[4], vb[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (t0 + q >= W) break;
                va[q] = pa ? load_l<LONE>(ph) : VT(0);
                vb[q] = pb ? load_l<LONE>(ph + 32) : VT(0);
                ph += hs;
                hs--;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (t0 + q >= W) break;
                const double xj = __shfl_sync(0xffffffffu, xa, t0 + q);
                if (xj != 0.0) {
                    if (pa) ya = __dsub_rn(ya, __dmul_rn((double)va[q], xj));
                    if (pb) yb = __dsub_rn(yb, __dmul_rn((double)vb[q], xj));
                }
            }
        }
        if (pa) x[ra] = ya;
        if (pb) x[rb] = yb;
    }
}

template <typename VT, bool LONE>
__device__ __forceinline__ void seg_update(const VT* lcol, const unsigned short* rel, double* x, int u0, int a, int W,
                                           int lp0, int cnt) {
    if (W == 1) {
        // One dependency: a multiply-subtract per row, two rows per lane in
        // flight.
        const int lane = threadIdx.x & 31, m = cnt - a;
        const VT* src = lcol + (lp0 + a * cnt - ((a * (a - 1)) >> 1));
        const double xj = x[u0 + a];
        if (xj != 0.0) {
            for (int e = lane; e < m; e += 64) {
                const bool two = e + 32 < m;
                const int s0 = (int)__ldg(rel + a + e), s1 = two ? (int)__ldg(rel + a + e + 32) : s0;
                const VT l0 = load_l<LONE>(src + e), l1 = two ? load_l<LONE>(src + e + 32) : VT(0);
                const double x0 = x[s0], x1 = x[s1];
                x[s0] = __dsub_rn(x0, __dmul_rn((double)l0, xj));
                if (two) x[s1] = __dsub_rn(x1, __dmul_rn((double)l1, xj));
            }
        }
    } else if (cnt - a < 32) {
        seg_rows<VT, false, LONE>(lcol, rel, x, u0, a, W, lp0, cnt);
    } else {
        seg_rows<VT, true, LONE>(lcol, rel, x, u0, a, W, lp0, cnt);
    }
    __syncwarp();
}

// Spread mode: the pivot statistics and cycle counters of one CTA merged
// into the system's sync area; the last CTA to finish writes the system's
// statistics (pivot minima through the bit patterns of non-negative doubles:
// a larger complement is a smaller value, so 0 means none yet).
__device__ void spread_finish(const SysDev& S, unsigned* sync, int group, double minpiv, double minratio,
                              double maxu, int bad, long long cw, long long cu, long long t_begin) {
    const int lane = threadIdx.x & 31;
    int* ctl = (int*)sync;
    unsigned long long* acc = (unsigned long long*)(sync + kSyncAcc);
    minpiv = warp_min(minpiv);
    minratio = warp_min(minratio);
    maxu = warp_max(maxu);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (lane == 0) {
        if (bad) atomicOr(&ctl[kSyncStatus], bad);
        if (minpiv < INFINITY) atomicMax(&acc[0], ~(unsigned long long)__double_as_longlong(minpiv));
        if (minratio < INFINITY) atomicMax(&acc[1], ~(unsigned long long)__double_as_longlong(minratio));
        atomicMax(&acc[2], (unsigned long long)__double_as_longlong(maxu));
        atomicAdd(&acc[3], (unsigned long long)cw);
        atomicAdd(&acc[4], (unsigned long long)cu);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&ctl[kSyncDone], 1) == group - 1) {
        __threadfence();
        const volatile unsigned long long* va = acc;
        const volatile int* vc = ctl;
        SysStats* st = S.stats;
        const unsigned long long a0 = va[0], a1 = va[1];
        st->min_abs_pivot = a0 ? __longlong_as_double((long long)~a0) : INFINITY;
        st->min_pivot_ratio = a1 ? __longlong_as_double((long long)~a1) : INFINITY;
        st->max_abs_u = __longlong_as_double((long long)va[2]);
        st->status = vc[kSyncStatus];
        const int sc = vc[kSyncSingular];
        st->singular_col = sc > 0 ? 0x7fffffff - sc : -1;
        st->nres = 0;
        st->inner_iters = 0;
        st->outer_iters = 0;
        st->cyc_wait = (long long)va[3];
        st->cyc_gather = 0;
        st->cyc_update = (long long)va[4];
        st->cyc_refactor = clock64() - t_begin;
    }
}

// Cycle split of the refactor (waits for dependency columns, updates) into
// SysStats::cyc_wait / cyc_update; cyc_gather is 0, since the L parts are read
// by the updates themselves.
// Reading the SM clock three times per dependency round costs ~3 % of the
// grid refactor, so the split is a build option (-DLUSP_REFACTOR_PHASE_CYCLES=1);
// without it both fields stay 0 (cyc_refactor is always written).
#ifndef LUSP_REFACTOR_PHASE_CYCLES
#define LUSP_REFACTOR_PHASE_CYCLES 0
#endif
__device__ __forceinline__ long long phase_clock() {
    if constexpr (LUSP_REFACTOR_PHASE_CYCLES != 0) return clock64();
    else return 0;
}

// A CTA's copy of its system's descriptors in shared memory: the column loop
// reads each pointer where it uses it (30 cycles) instead of holding some
// sixty registers of them or fetching them from global memory.
struct RefactorCtx {
    SysDev sys;
    PatternDev pat;
};

// Pause between two looks at the ready bits of a column's dependencies.
constexpr unsigned kPollSleep = 32;

// Bytes of a warp's column record and pivot minima, before its work vector.
constexpr int kWarpHead = 80;

// All threads; ends with a CTA barrier.
__device__ __forceinline__ void load_ctx(RefactorCtx& cx, const SysDev* sys) {
    static_assert(sizeof(SysDev) % 4 == 0 && sizeof(PatternDev) % 4 == 0, "copied as words");
    const int* pat = (const int*)sys->pat;
    for (int t = threadIdx.x; t < (int)(sizeof(SysDev) / 4); t += blockDim.x) ((int*)&cx.sys)[t] = ((const int*)sys)[t];
    for (int t = threadIdx.x; t < (int)(sizeof(PatternDev) / 4); t += blockDim.x) ((int*)&cx.pat)[t] = pat[t];
    __syncthreads();
}

// SPREAD: the system's columns are shared by `group` CTAs anywhere on the
// GPU (CTA `member` of them) through the sync area in global memory; else
// by the CTAs of this thread-block cluster through rank 0's shared memory.
// LONE: by this CTA alone, through its own shared memory.
template <typename VT, bool SPREAD = false, bool LONE = false>
__device__ void refactor_phase(const RefactorCtx& cx, const SmemPlan& plan, char* smem_base,
                               const SolveParams& prm, unsigned* sync = nullptr, int member = 0,
                               int group = 1) {
    const SysDev& S = cx.sys;
    const PatternDev& P = cx.pat;
    const int n = P.n;
    Smem sm(smem_base, plan);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // This warp's column record (16 ints), pivot minima and work vector.
    int* rec = (int*)(sm.uni + (size_t)warp * ((size_t)plan.wcap * 8 + kWarpHead));
    double* pmin = (double*)(rec + 16);
    double* wx = pmin + 2;
    if (lane == 0) pmin[0] = pmin[1] = INFINITY;
    const bool have_seg = P.seg != nullptr && prm.refactor_mode == 0;
    // The CTAs of a thread-block cluster share one system: the claim
    // counter, status, singular column, abort flag and ready bits live in
    // rank 0's shared memory (distributed shared memory for the others).
    namespace cgr = cooperative_groups;
    cgr::cluster_group cl = cgr::this_cluster();
    const unsigned crank = SPREAD ? (unsigned)member : LONE ? 0u : cl.block_rank();
    const unsigned csize = SPREAD ? (unsigned)group : LONE ? 1u : cl.num_blocks();
    unsigned* ready = SPREAD ? sync + kSyncReady : LONE ? sm.ready : cl.map_shared_rank(sm.ready, 0);
    int* ctl = SPREAD ? (int*)sync : LONE ? sm.ctl : cl.map_shared_rank(sm.ctl, 0);

    if (!SPREAD && crank == 0) {
        for (int t = threadIdx.x; t < (n + 31) / 32; t += blockDim.x) sm.ready[t] = 0u;
        if (threadIdx.x == 0) {
            sm.ctl[0] = 0;
            sm.ctl[1] = 0;
            sm.ctl[2] = 0x7fffffff;
            sm.ctl[3] = 0;
        }
    }
    double maxu = 0.0;
    int bad = 0;
    long long c_wait = 0, c_update = 0;
    const long long t_begin = clock64();
    if (!SPREAD) {
        if (crank == 0 && threadIdx.x == 0) {
            S.stats->cyc_wait = 0;
            S.stats->cyc_gather = 0;
            S.stats->cyc_update = 0;
        }
        if (LONE) __syncthreads();
        else cl.sync();
    }

    while (true) {
        const int idx = warp_claim(&ctl[0]);
        if (idx >= n) break;
        // The column's record, four 16-byte words into shared memory, then,
        // all in flight together: this lane's first input entry, its first
        // segment, the destination of its first slot, and the input value.
        // The later entries (columns longer than a warp) load as they are
        // reached.
        if (lane < 4) *(int4*)(rec + 4 * lane) = __ldg(P.crec + 4 * idx + lane);
        __syncwarp();
        const int len = rec[2], a0 = rec[4], a1 = rec[5], nseg = have_seg ? rec[13] : 0;
        const int ta = a0 + lane;
        const int adst = ta < a1 ? P.a_dst[ta] : -1;
        const int asrc = ta < a1 ? P.a_src[ta] : -1;
        const int aprev = (ta < a1 && ta > a0) ? P.a_dst[ta - 1] : -1;
        int4 sg = lane < nseg ? __ldg(P.seg + rec[12] + lane) : make_int4(0, 0, 0, 0);
        const int sdst0 = lane < len ? P.slot_dst[rec[1] + lane] : -1;
        const double av0 = asrc >= 0 ? S.a_val[asrc] : 0.0;
        double* x;
        if (len <= plan.wcap) {
            x = wx;
        } else if (S.scratch) {
            x = S.scratch + ((size_t)blockIdx.x * nw + warp) * P.max_col;
        } else {
            bad |= ST_CAPACITY;
            __syncwarp();
            if (lane == 0) set_ready(ready, rec[0]);
            continue;
        }
        for (int t = lane; t < len; t += 32) x[t] = 0.0;
        __syncwarp();
        // The factor of A + shift diag|A(i,i)|: the input's diagonal entry
        // (duplicates summed first) gains shift times its magnitude.
        const int adg = prm.shift != 0.0 ? rec[10] : -1;
        if (ta < a1 && (ta == a0 || aprev != adst)) {
            double s = av0;
            for (int u = ta + 1; u < a1 && P.a_dst[u] == adst; u++) s = __dadd_rn(s, S.a_val[P.a_src[u]]);
            if (adst == adg) s = __dadd_rn(s, __dmul_rn(prm.shift, fabs(s)));
            x[adst] = s;
        }
        for (int t = a0 + 32 + lane; t < a1; t += 32) {
            const int dst = P.a_dst[t];
            if (t == a0 || P.a_dst[t - 1] != dst) {
                double s = S.a_val[P.a_src[t]];
                for (int u = t + 1; u < a1 && P.a_dst[u] == dst; u++)
                    s = __dadd_rn(s, S.a_val[P.a_src[u]]);
                if (dst == adg) s = __dadd_rn(s, __dmul_rn(prm.shift, fabs(s)));
                x[dst] = s;
            }
        }
        __syncwarp();
        long long tc = phase_clock();
        // Apply the dependency columns in ascending order, 32 segments at a
        // time: each round takes the segments whose dependencies are all
        // complete, up to the first that is not, then the complete first part
        // of that one; it blocks only when nothing could be applied.
        const unsigned short* rel = P.rel + *(const long long*)(rec + 8);
        const VT* lcol = (const VT*)S.lcol;
        for (int s0 = 0; s0 < nseg; s0 += 32) {
            if (s0 > 0) sg = s0 + lane < nseg ? __ldg(P.seg + rec[12] + s0 + lane) : make_int4(0, 0, 0, 0);
            const int ns = min(32, nseg - s0);
            const int jj = sg.x, w = sg.y >> 16;
            int c = 0, off = 0;     // next segment of the window, its dependencies already applied
            long long spins = 0;    // looks since the last one that found work
            while (c < ns) {
                int r = 0;
                if (lane >= c && lane < ns) {
                    // Ready bits of columns jj .. jj + w - 1 (w <= 32).
                    const int sh = jj & 31;
                    const volatile unsigned* word = ready + (jj >> 5);
                    unsigned bits = word[0] >> sh;
                    if (sh + w > 32) bits |= word[1] << (32 - sh);
                    r = min(w, bits == 0xffffffffu ? 32 : __ffs(~bits) - 1);
                }
                // Acquire: each lane orders what follows after its own reads
                // of ready bits; the warp's ballot then orders the other
                // lanes' reads of those columns' values after them.
                if (SPREAD) spread_acquire();
                const unsigned full = __ballot_sync(0xffffffffu, lane >= c && lane < ns && r >= w) >> c;
                int run = full == 0xffffffffu ? 32 : __ffs(~full) - 1;
                int part = 0;        // applied part of the segment after the run
                bool late = false;
                if (c + run < ns) {
                    part = __shfl_sync(0xffffffffu, r, c + run);
                    if (run == 0 && part <= off) {
                        // Nothing to apply yet.  Spread mode: look again (the
                        // look is the poll: a wait for one bit and then a look
                        // would read the bits twice, 340 cycles each).  Else
                        // the bits are near: wait for the next dependency.
                        if (!SPREAD) {
                            const int jn = __shfl_sync(0xffffffffu, jj, c) + off;
                            if (__all_sync(0xffffffffu, wait_ready(ready, jn, &ctl[3]))) continue;
                        } else if (++spins <= kSpinLimit && ((spins & 31) || !*(const volatile int*)&ctl[3])) {
                            __nanosleep(kPollSleep);
                            continue;
                        }
                        if (SPREAD && spins > kSpinLimit) atomicExch(&ctl[3], 1);
                        spins = kSpinLimit;
                        bad |= ST_WAIT_TIMEOUT;
                        part = off + 1;
                        late = true;
                    }
                }
                if (!late) spins = 0;
                // Acquire (cluster): the dependency columns' values (written
                // by any CTA of the cluster) are read after their ready bits.
                if (!SPREAD) share_fence(csize);
                {
                    const long long t2 = phase_clock();
                    c_wait += t2 - tc;
                    tc = t2;
                }
                const int end = c + run + ((part > 0 && (run > 0 || part > off)) ? 1 : 0);
                for (int s = c; s < end; s++) {
                    const int y = __shfl_sync(0xffffffffu, sg.y, s), lp0 = __shfl_sync(0xffffffffu, sg.z, s);
                    const int cnt = __shfl_sync(0xffffffffu, sg.w, s);
                    const int a = s == c ? off : 0;
                    seg_update<VT, LONE>(lcol, rel, x, y & 0xffff, a, (s < c + run ? y >> 16 : part) - a, lp0, cnt);
                    if (s < c + run) rel += cnt;
                }
                if (run > 0) off = 0;
                if (part > off) off = part;
                c += run;
                if (late && off >= __shfl_sync(0xffffffffu, w, c)) {
                    rel += __shfl_sync(0xffffffffu, sg.w, c);
                    off = 0;
                    c++;
                }
                {
                    const long long t2 = phase_clock();
                    c_update += t2 - tc;
                    tc = t2;
                }
            }
        }
        // Without segments: one dependency at a time, its rows searched.
        for (int u = 0; !have_seg && u < rec[6]; u++) {
            const int* rows = P.ri + rec[1];
            const int j = rows[u];
            if (!__all_sync(0xffffffffu, wait_ready(ready, j, &ctl[3]))) bad |= ST_WAIT_TIMEOUT;
            if (SPREAD) spread_acquire();
            else share_fence(csize);
            const double xj = x[u];
            const int p0 = P.lp[j], cn = P.lp[j + 1] - p0;
            if (xj != 0.0) {
                for (int e = lane; e < cn; e += 32) {
                    const double l = (double)__ldcg(lcol + p0 + e);
                    const int s = find_slot(rows, u + 1, len, P.ri[P.dg[j] + 1 + e]);
                    if (s >= 0) x[s] = __dsub_rn(x[s], __dmul_rn(l, xj));
                    else bad |= ST_CAPACITY;
                }
            }
            __syncwarp();
        }
        const int k = rec[0], c0 = rec[1], d = rec[3];
        // A column of the dense trailing block applies only its dependencies
        // before k0 here (they come first: rows ascending; dsp of them).
        if (k >= P.k0) {
            // U rows before k0 are final; the rest goes to the dense block,
            // its pattern's entries (the dense kernel reads the others as 0;
            // destinations of four slots per lane loaded first).
            const int dsp = rec[6], k0 = P.k0, D = P.dtail;
            double* W = S.tailw;
            VT* uval = (VT*)S.uval;
            for (int t0 = lane; t0 < len; t0 += 128) {
                int dst[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int t = t0 + 32 * q;
                    dst[q] = t >= len ? 0 : t < dsp ? (t < 32 ? sdst0 : __ldg(P.slot_dst + c0 + t))
                                                    : __ldg(P.ri + c0 + t);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int t = t0 + 32 * q;
                    if (t >= len) break;
                    const double v = x[t];
                    if (t < dsp) {
                        maxu = fmax(maxu, fabs(v));
                        uval[dst[q]] = ValTraits<VT>::to(v);
                    } else {
                        W[tail_index(D, dst[q] - k0, k - k0)] = v;
                    }
                }
            }
            __syncwarp();
            continue;
        }
        const double piv = x[d], rpiv = __drcp_rn(piv);
        // The multipliers, published before anything else of the column.
        // amax: the largest |x| below the pivot that exceeds it (the others do
        // not count for its ratio).
        const double ap = fabs(piv);
        double amax = 0.0;
        VT* lk = (VT*)S.lcol + rec[14] - d - 1;
#pragma unroll 4
        for (int t = d + 1 + lane; t < len; t += 32) {
            const double v = x[t];
            const VT l = ValTraits<VT>::to(div_by<false>(v, piv, rpiv));
            lk[t] = l;
            x[t] = (double)l;
            if (fabs(v) > ap) amax = fmax(amax, fabs(v));
        }
        // Release: the column's values before its ready bit.
        share_release_t<SPREAD>(csize);
        __syncwarp();
        if (lane == 0) set_ready(ready, k);
        if (__any_sync(0xffffffffu, amax > 0.0)) amax = warp_max(amax);
        if (!(ap > 0.0) || !isfinite(piv)) {
            bad |= ST_SINGULAR;
            // The first singular column: a minimum (spread mode: the sync
            // area starts at 0, so the maximum of INT_MAX - k).
            if (lane == 0) {
                if (SPREAD) atomicMax(&ctl[kSyncSingular], 0x7fffffff - k);
                else atomicMin(&ctl[2], k);
            }
        }
        const double ratio = amax > ap ? ap / amax : 1.0;
        if (lane == 0) {
            pmin[0] = fmin(pmin[0], ap);
            pmin[1] = fmin(pmin[1], ratio);
        }
        if (ratio < prm.pivot_tol) bad |= ST_PIVOT_WEAK;
        // Each value is stored once where the solves read it (U rows, the
        // diagonal, L rows); the strict-L part also goes to the merged
        // columns.  The destinations of four slots per lane are loaded before
        // any of their stores (the loads could not move above the stores of
        // an earlier slot).
        VT* lu = (VT*)S.lu + c0;
        VT* lval = (VT*)S.lval;
        VT* uval = (VT*)S.uval;
        for (int t0 = lane; t0 < len; t0 += 128) {
            int dst[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int t = t0 + 32 * q;
                dst[q] = t < len ? (t < 32 ? sdst0 : __ldg(P.slot_dst + c0 + t)) : 0;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int t = t0 + 32 * q;
                if (t >= len) break;
                const double v = x[t];
                const VT sv = ValTraits<VT>::to(v);
                if (t <= d) maxu = fmax(maxu, fabs(v));
                if (t < d) uval[dst[q]] = sv;
                else if (t == d) {
                    ((VT*)S.udiag)[k] = sv;
                    ((VT*)S.udiag_bwd)[rec[7]] = ValTraits<VT>::to(rpiv);
                } else {
                    lu[t] = sv;
                    lval[dst[q]] = sv;
                }
            }
        }
        __syncwarp();
    }

    __syncwarp();
    const double minpiv = pmin[0], minratio = pmin[1];
    if (SPREAD) {
        spread_finish(S, sync, group, minpiv, minratio, maxu, bad, c_wait, c_update, t_begin);
        return;
    }
    if (lane == 0) {
        atomicAdd((unsigned long long*)&S.stats->cyc_wait, (unsigned long long)c_wait);
        atomicAdd((unsigned long long*)&S.stats->cyc_update, (unsigned long long)c_update);
    }
    if (threadIdx.x == 0) S.stats->cyc_refactor = clock64() - t_begin;
    // Statistics: rank 0 writes, the others merge, one after another; the
    // last cluster barrier also keeps rank 0's shared state alive until every
    // CTA of the cluster is done with it.
    if (LONE) {
        __syncthreads();
        cta_store_pivot_stats(S.stats, sm, minpiv, minratio, maxu, bad, true, ctl);
        return;
    }
    cl.sync();
    for (unsigned r = 0; r < csize; r++) {
        if (crank == r) cta_store_pivot_stats(S.stats, sm, minpiv, minratio, maxu, bad, r == 0, ctl);
        cl.sync();
    }
}

// ---------------------------------------------------------------------------
// Triangular solves of the dense trailing block (rows [k0, n), factor T in
// VT with leading dimension ld): 32-row blocks, the diagonal block by one
// warp through shuffles, the rest of the block's columns as one
// multiply-add per row and thread.  fp64 accumulation.
// ---------------------------------------------------------------------------
// sum_{c < w} row[c * stride] * y[c] for one 32-column block of a tail row
// (column-major factor): all loads issued before the multiply-adds.
template <typename VT>
__device__ __forceinline__ double tail_row_dot(const VT* row, size_t stride, const double* y, int w) {
    // Unconditional loads from clamped (in-bounds) addresses, so all 32 are
    // in flight before the first multiply-add.
    VT v[32];
#pragma unroll
    for (int c = 0; c < 32; c++) v[c] = row[(size_t)min(c, w - 1) * stride];
    double acc = 0.0;
#pragma unroll
    for (int c = 0; c < 32; c++) acc = fma(c < w ? (double)v[c] : 0.0, y[min(c, w - 1)], acc);
    return acc;
}

// The 32 factor values of one tail row's 32-column block (clamped
// addresses, all loads in flight), and their dot product with y.
template <typename VT>
__device__ __forceinline__ void tail_load_regs(const VT* row, size_t stride, int w, VT* v) {
#pragma unroll
    for (int c = 0; c < 32; c++) v[c] = row[(size_t)min(c, w - 1) * stride];
}
// tail_row_dot as a call (rows past the ones a thread preloads: D above the
// CTA size; keeps its 32 loads out of the caller's registers).
template <typename VT>
__device__ __noinline__ double tail_row_dot_call(const VT* row, size_t stride, const double* y, int w) {
    return tail_row_dot<VT>(row, stride, y, w);
}
template <typename VT>
__device__ __forceinline__ double tail_dot_regs(const VT* v, const double* y, int w) {
    double acc = 0.0;
#pragma unroll
    for (int c = 0; c < 32; c++) acc = fma(c < w ? (double)v[c] : 0.0, y[min(c, w - 1)], acc);
    return acc;
}

// y[k0..n) := L_tt^-1 y[k0..n) (unit lower; the tail rows' entries in the
// columns before k0 were applied by the forward sweep's last level).
template <typename VT>
__device__ __noinline__ void tail_forward(const PatternDev& P, const VT* T, const VT* Ti, double* y, SysStats* st) {
    const int k0 = P.k0, D = P.dtail, ld = P.tail_ld;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long c_diag = 0, c_gemv = 0;
    double* yt = y + k0;
    // Every thread loads 32 values before the diagonal block: warp 0 its
    // row of the block's inverse (L^-1, from the dense kernel), the other
    // warps their first row of the block's 32 columns below it (so those
    // loads overlap the diagonal product).
    const int nt = (int)blockDim.x - 32, t = (int)threadIdx.x - 32;
    for (int jb = 0; jb < D; jb += 32) {
        const int w = min(32, D - jb);
        const long long ta = clock64();
        const int i0 = jb + w + t;
        const bool pre = t >= 0 && i0 < D;
        VT v[32];
        if (warp == 0) tail_load_regs<VT>(Ti + (size_t)(jb >> 5) * 2048 + lane, 32, 32, v);
        else if (pre) tail_load_regs<VT>(T + (size_t)jb * ld + i0, ld, w, v);
        if (warp == 0) {
            // y_b := L_bb^-1 y_b: lane i's row of the inverse against the
            // block of y (all lanes read it before any writes).
            const double yr = lane < w ? tail_dot_regs<VT>(v, yt + jb, w) : 0.0;
            __syncwarp();
            if (lane < w) yt[jb + lane] = yr;
        }
        __syncthreads();
        const long long tb = clock64();
        if (pre) yt[i0] -= tail_dot_regs<VT>(v, yt + jb, w);
        for (int i = i0 + nt; t >= 0 && i < D; i += nt)
            yt[i] -= tail_row_dot_call<VT>(T + (size_t)jb * ld + i, ld, yt + jb, w);
        __syncthreads();
        const long long tc = clock64();
        c_diag += tb - ta;
        c_gemv += tc - tb;
    }
    if (threadIdx.x == 0) {
        st->cyc_tdiag += c_diag;
        st->cyc_tgemv += c_gemv;
    }
}

// y[k0..n) := U_tt^-1 y[k0..n) (upper with diagonal).
template <typename VT>
__device__ __noinline__ void tail_backward(const PatternDev& P, const VT* T, const VT* Ti, double* y, SysStats* st) {
    const int k0 = P.k0, D = P.dtail, ld = P.tail_ld;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long c_diag = 0, c_gemv = 0;
    double* yt = y + k0;
    // As tail_forward: warp 0 applies the block's U^-1, the other warps
    // update the rows above it, their first row loaded before that product.
    const int nt = (int)blockDim.x - 32, t = (int)threadIdx.x - 32;
    for (int jb = ((D - 1) / 32) * 32; jb >= 0; jb -= 32) {
        const int w = min(32, D - jb);
        const long long ta = clock64();
        const bool pre = t >= 0 && t < jb;
        VT v[32];
        if (warp == 0) tail_load_regs<VT>(Ti + (size_t)(jb >> 5) * 2048 + 1024 + lane, 32, 32, v);
        else if (pre) tail_load_regs<VT>(T + (size_t)jb * ld + t, ld, w, v);
        if (warp == 0) {
            const double yr = lane < w ? tail_dot_regs<VT>(v, yt + jb, w) : 0.0;
            __syncwarp();
            if (lane < w) yt[jb + lane] = yr;
        }
        __syncthreads();
        const long long tb = clock64();
        if (pre) yt[t] -= tail_dot_regs<VT>(v, yt + jb, w);
        for (int i = t + nt; t >= 0 && i < jb; i += nt)
            yt[i] -= tail_row_dot_call<VT>(T + (size_t)jb * ld + i, ld, yt + jb, w);
        __syncthreads();
        const long long tc = clock64();
        c_diag += tb - ta;
        c_gemv += tc - tb;
    }
    if (threadIdx.x == 0) {
        st->cyc_tdiag += c_diag;
        st->cyc_tgemv += c_gemv;
    }
}

// ---------------------------------------------------------------------------
// y := U^-1 L^-1 rhs in pivot-position space (level-scheduled, warp per row,
// factors read as VT, accumulation in fp64).  y may be shared or global
// memory; rhs must not alias y.
// ---------------------------------------------------------------------------
template <typename VT>
__device__ void cta_lu_apply(const PatternDev& P, const VT* lval, const VT* uval,
                             const VT* udiag, const VT* tail, const VT* tinv, const double* rhs, double* y,
                             Smem& sm, int& bad, SysStats* st) {
    const long long t0 = clock64();
    const int n = P.n, k0 = P.k0;
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = rhs[i];
    for (int t = threadIdx.x; t < (n + 31) / 32; t += blockDim.x) sm.ready[t] = 0u;
    if (threadIdx.x == 0) {
        sm.ctl[0] = 0;
        sm.ctl[3] = 0;
    }
    __syncthreads();
    volatile double* vy = y;
    while (true) {
        const int idx = warp_claim(&sm.ctl[0]);
        if (idx >= n) break;
        const int i = P.fwd_order[idx];
        const int p0 = P.lrp[idx], p1 = P.lrp[idx + 1];
        double acc = 0.0;
        for (int p = p0 + lane; p < p1; p += 32) {
            const int j = P.lci[p];
            const double v = ValTraits<VT>::load(lval + p);
            if (!wait_ready(sm.ready, j, &sm.ctl[3])) bad |= ST_WAIT_TIMEOUT;
            __threadfence_block();
            acc = fma(v, vy[j], acc);
        }
        acc = warp_sum(acc);
        if (lane == 0) {
            vy[i] = vy[i] - acc;
            __threadfence_block();
            set_ready(sm.ready, i);
        }
    }
    __syncthreads();
    const long long t1 = clock64();
    if (P.dtail > 0) {
        tail_forward<VT>(P, tail, tinv, y, st);
        tail_backward<VT>(P, tail, tinv, y, st);
    }
    const long long t2 = clock64();
    // Rows of the dense tail are complete before the sparse U sweep starts.
    for (int t = threadIdx.x; t < (n + 31) / 32; t += blockDim.x) {
        const int lo = t * 32;
        unsigned bits = 0u;
        for (int b = 0; b < 32; b++)
            if (lo + b >= k0 && lo + b < n) bits |= 1u << b;
        sm.ready[t] = bits;
    }
    if (threadIdx.x == 0) sm.ctl[0] = 0;
    __syncthreads();
    while (true) {
        const int idx = warp_claim(&sm.ctl[0]);
        if (idx >= k0) break;
        const int i = P.bwd_order[idx];
        const int p0 = P.urp[idx], p1 = P.urp[idx + 1];
        double acc = 0.0;
        for (int p = p0 + lane; p < p1; p += 32) {
            const int j = P.uci[p];
            const double v = ValTraits<VT>::load(uval + p);
            if (!wait_ready(sm.ready, j, &sm.ctl[3])) bad |= ST_WAIT_TIMEOUT;
            __threadfence_block();
            acc = fma(v, vy[j], acc);
        }
        acc = warp_sum(acc);
        if (lane == 0) {
            vy[i] = (vy[i] - acc) / ValTraits<VT>::load(udiag + i);
            __threadfence_block();
            set_ready(sm.ready, i);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && st) {
        st->cyc_lsolve += t1 - t0;
        st->cyc_tail += t2 - t1;
        st->cyc_usolve += clock64() - t2;
    }
}

// cp.async group control (sm_80+).
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// One triangular sweep, level-synchronous (one barrier per level).  Each
// level's entries (column positions, values and, for U, the diagonal of its
// rows in sweep order) are copied by cp.async into a ring of kStages
// shared-memory stages, kStages - 1 levels ahead of the level being
// computed, so a level's work reads shared memory only.  A level's rows are
// spread over groups of g lanes, g the power of two at or above its mean
// row length (1..32): wide levels of short rows run a row per thread,
// narrow levels of long rows a row per warp, or, for a level of a few very
// long rows, several warps per row whose partial sums are added in warp
// order (part: NT / 32 doubles of shared memory).  Levels larger than a
// stage read global memory directly.
// UPPER: y[i] = (y[i] - sum) / diag (U sweep), else y[i] -= sum.
constexpr int kStages = 4;

// Bulk asynchronous copies (TMA, untiled) with completion on an mbarrier in
// shared memory: 16-byte aligned addresses, sizes a multiple of 16 bytes.
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(unsigned long long* bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// The barriers' initialization, visible to the asynchronous proxy.
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
// Earlier generic-proxy accesses to shared memory ordered before later
// asynchronous-proxy (bulk copy) writes.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for phase `parity` of bar: false (and the status bit set)
// when it does not complete within kSpinLimit polls.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int* status) {
    for (long long it = 0; !mbar_try_wait(bar, parity); it++) {
        if (it > kSpinLimit) {
            if (status) atomicOr(status, ST_WAIT_TIMEOUT);
            return false;
        }
    }
    return true;
}

// sum over e = e0, e0 + g, ... < pe of val[e] * y[col[e]]: four partial
// sums, so a lane has four loads of y in flight when y lives in global
// memory (a row with fewer than four entries per lane keeps one sum).
template <typename VT>
__device__ __forceinline__ double row_dot(const VT* vv, const int* cc, const double* y, int e0, int pe, int g) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    int e = e0;
    for (; e + 3 * g < pe; e += 4 * g) {
        const int c0 = cc[e], c1 = cc[e + g], c2 = cc[e + 2 * g], c3 = cc[e + 3 * g];
        a0 = fma(ValTraits<VT>::load(vv + e), y[c0], a0);
        a1 = fma(ValTraits<VT>::load(vv + e + g), y[c1], a1);
        a2 = fma(ValTraits<VT>::load(vv + e + 2 * g), y[c2], a2);
        a3 = fma(ValTraits<VT>::load(vv + e + 3 * g), y[c3], a3);
    }
    for (; e < pe; e += g) a0 = fma(ValTraits<VT>::load(vv + e), y[cc[e]], a0);
    return (a0 + a1) + (a2 + a3);
}

__host__ __device__ inline size_t stage_bytes(int cap_e, int cap_r, int vsize) {
    return (size_t)(cap_e + 8) * (4 + vsize) + (size_t)(cap_r + 8) * vsize;
}

// The sweeps run on the first kSweepThreads threads (named barrier 1); the
// other warps of the CTA, if any, wait at the closing CTA barrier.
constexpr int kSweepThreads = 1024;

__device__ __forceinline__ void sweep_barrier(int nthreads) {
    asm volatile("bar.sync 1, %0;\n" ::"r"(nthreads) : "memory");
}

// The rows [r0, r1) of one level, 2^LG lanes per row (a compile-time group
// width, so the row reduction is unrolled), in rounds of NT / 2^LG rows.
template <typename VT, bool UPPER, bool GY, int LG>
__device__ __forceinline__ void sweep_rows(int r0, int r1, int NT, const int* order, const int* rp, const int* cc,
                                           const VT* vv, const VT* dd, int eb, int rb, double* y) {
    constexpr int g = 1 << LG;
    const int lig = threadIdx.x & (g - 1);
    const int warp = threadIdx.x >> 5;
    const int ngr = NT >> LG;
    for (int rbase = r0; rbase < r1; rbase += ngr) {
        if (rbase + ((warp * 32) >> LG) >= r1) break;   // nothing left for this warp
        const int r = rbase + ((int)threadIdx.x >> LG);
        double acc = 0.0, yi = 0.0, di = 1.0;
        int i = 0;
        if (r < r1) {
            // The row's own right-hand side and diagonal, loaded beside the
            // dot product instead of after its reduction (no other thread
            // writes y[i] in this level).
            if (lig == 0) {
                i = order[r];
                yi = y[i];
                if (UPPER) di = ValTraits<VT>::load(dd + (r - rb));
            }
            if (GY) {
                acc = row_dot<VT>(vv, cc, y, rp[r] - eb + lig, rp[r + 1] - eb, g);
            } else {
                // Two entries per lane in flight.
                const int pe = rp[r + 1] - eb;
                int e = rp[r] - eb + lig;
                double a1 = 0.0;
                for (; e + g < pe; e += 2 * g) {
                    const int c0 = cc[e], c1 = cc[e + g];
                    const double v0 = ValTraits<VT>::load(vv + e), v1 = ValTraits<VT>::load(vv + e + g);
                    acc = fma(v0, y[c0], acc);
                    a1 = fma(v1, y[c1], a1);
                }
                if (e < pe) acc = fma(ValTraits<VT>::load(vv + e), y[cc[e]], acc);
                acc += a1;
            }
        }
#pragma unroll
        for (int o = g >> 1; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, g);
        if (r < r1 && lig == 0) y[i] = UPPER ? (yi - acc) * di : yi - acc;
    }
}

// GY: y lives in global memory (large systems): levels of a few long rows
// (64 entries or more on average) get several warps per row, and long rows
// four partial sums per lane; with y in shared memory a lane keeps one sum
// and a row at most one warp.
template <typename VT, bool UPPER, bool GY>
__device__ __noinline__ void staged_sweep(int nlev, const int4* ld4, const int* lgl, const int* order, const int* rp,
                             const int* ci, const VT* val, const VT* dgo, double* y,
                             char* stage, int cap_e, int cap_r, double* part, int* status) {
    const int NT = min((int)blockDim.x, kSweepThreads);
    if ((int)threadIdx.x >= NT) {
        __syncthreads();
        return;
    }
    const int CE = cap_e + 8;
    const size_t sb = stage_bytes(cap_e, cap_r, sizeof(VT));
    const int warp = threadIdx.x >> 5;
    // Each staged level is three bulk copies (column indices, values and,
    // for U, the reciprocal diagonal: contiguous runs in sweep order, rounded
    // out to 16-byte boundaries; every array has slack past its end for the
    // rounding) issued by one thread, the last one (rows go to the lowest
    // warps), completing on the slot's mbarrier; every thread waits on that
    // barrier's phase before the level's CTA barrier.
    __shared__ unsigned long long mbar[kStages];
    const bool issuer = (int)threadIdx.x == NT - 1;
    auto staged = [&](const int4& d) { return d.w - d.z <= cap_e && d.y - d.x <= cap_r; };
    // Every level arrives on its slot's barrier (a level too large for a
    // stage with no bytes), so the k-th use of a slot is its phase k.
    auto issue = [&](int L) {
        if (!issuer || L >= nlev) return;
        const int4 d = ld4[L];
        if (!staged(d)) {
            mbar_expect_tx(&mbar[L % kStages], 0u);
            return;
        }
        char* base = stage + (size_t)(L % kStages) * sb;
        int* sc = (int*)base;
        VT* sv = (VT*)(base + (size_t)CE * 4);
        VT* sd = (VT*)(base + (size_t)CE * (4 + sizeof(VT)));
        const int a0 = d.z & ~3, n4 = ((d.w + 3) & ~3) - a0;
        const int b0 = d.x & ~3, m4 = UPPER ? ((d.y + 3) & ~3) - b0 : 0;
        unsigned long long* bar = &mbar[L % kStages];
        fence_proxy_async();
        mbar_expect_tx(bar, (unsigned)((size_t)n4 * (4 + sizeof(VT)) + (size_t)m4 * sizeof(VT)));
        if (n4 > 0) {
            bulk_g2s(sc, ci + a0, (unsigned)n4 * 4u, bar);
            bulk_g2s(sv, val + a0, (unsigned)(n4 * sizeof(VT)), bar);
        }
        if (UPPER && m4 > 0) bulk_g2s(sd, dgo + b0, (unsigned)(m4 * sizeof(VT)), bar);
    };
    if (threadIdx.x == 0) {
        for (int k = 0; k < kStages; k++) mbar_init(&mbar[k], 1);
        fence_mbar_init();
    }
    sweep_barrier(NT);
    for (int L = 0; L < kStages - 1; L++) issue(L);
    for (int L = 0; L < nlev; L++) {
        mbar_wait(&mbar[L % kStages], (unsigned)(L / kStages) & 1u, status);
        sweep_barrier(NT);
        issue(L + kStages - 1);
        const int4 d = ld4[L];
        const int r0 = d.x, r1 = d.y, nr = r1 - r0;
        const bool st = d.w - d.z <= cap_e && nr <= cap_r;
        char* base = stage + (size_t)(L % kStages) * sb;
        const int* cc = st ? (const int*)base : ci;
        const VT* vv = st ? (const VT*)(base + (size_t)CE * 4) : val;
        const VT* dd = st ? (const VT*)(base + (size_t)CE * (4 + sizeof(VT))) : dgo;
        const int eb = st ? (d.z & ~3) : 0, rb = st ? (r0 & ~3) : 0;
        const int lgd = lgl[L];
        if (lgd < 0) {
            // A run of narrow levels: one warp, its rows in level order (a
            // row's result is visible to the warp's next rows after the warp
            // barrier), no CTA barrier until the run ends.
            if (warp == 0) {
                const int lane = threadIdx.x & 31;
                for (int r = r0; r < r1; r++) {
                    // Four loads per lane in flight (a run too large for a
                    // stage reads global memory).
                    double acc = row_dot<VT>(vv, cc, y, rp[r] - eb + lane, rp[r + 1] - eb, 32);
                    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
                    if (lane == 0) {
                        const int i = order[r];
                        if (UPPER) y[i] = (y[i] - acc) * ValTraits<VT>::load(dd + (r - rb));
                        else y[i] = y[i] - acc;
                    }
                    __syncwarp();
                }
            }
            continue;
        }
        // Several warps per row only for rows long enough to pay for the two
        // extra barriers.
        if (GY && lgd > 5 && d.w - d.z >= 64 * nr) {
            // Threads per row: the largest power of two (32 .. 2^lgd) that
            // still gives every row of the level its own group in one pass.
            int gw = 32;
            while (gw * 2 <= (1 << lgd) && gw * 2 * nr <= NT) gw *= 2;
            if (gw > 32) {
                const int rpp = NT / gw, wpr = gw >> 5;
                const int lane = threadIdx.x & 31;
                for (int rp0 = r0; rp0 < r1; rp0 += rpp) {
                    const int r = rp0 + (int)threadIdx.x / gw;
                    const int lig = (int)threadIdx.x & (gw - 1);
                    double acc = 0.0;
                    if (r < r1) acc = row_dot<VT>(vv, cc, y, rp[r] - eb + lig, rp[r + 1] - eb, gw);
                    acc = warp_sum(acc);
                    if (lane == 0) part[warp] = acc;
                    sweep_barrier(NT);
                    if ((int)threadIdx.x < rpp) {
                        const int rr = rp0 + (int)threadIdx.x;
                        if (rr < r1) {
                            double sum = 0.0;
                            for (int w = 0; w < wpr; w++) sum += part[threadIdx.x * wpr + w];
                            const int i = order[rr];
                            if (UPPER) y[i] = (y[i] - sum) * ValTraits<VT>::load(dd + (rr - rb));
                            else y[i] = y[i] - sum;
                        }
                    }
                    sweep_barrier(NT);
                }
                continue;
            }
        }
        switch (min(lgd, 5)) {
            case 0: sweep_rows<VT, UPPER, GY, 0>(r0, r1, NT, order, rp, cc, vv, dd, eb, rb, y); break;
            case 1: sweep_rows<VT, UPPER, GY, 1>(r0, r1, NT, order, rp, cc, vv, dd, eb, rb, y); break;
            case 2: sweep_rows<VT, UPPER, GY, 2>(r0, r1, NT, order, rp, cc, vv, dd, eb, rb, y); break;
            case 3: sweep_rows<VT, UPPER, GY, 3>(r0, r1, NT, order, rp, cc, vv, dd, eb, rb, y); break;
            case 4: sweep_rows<VT, UPPER, GY, 4>(r0, r1, NT, order, rp, cc, vv, dd, eb, rb, y); break;
            default: sweep_rows<VT, UPPER, GY, 5>(r0, r1, NT, order, rp, cc, vv, dd, eb, rb, y); break;
        }
    }
    // Every staged level's copies were waited for; the barriers are free.
    sweep_barrier(NT);
    if (threadIdx.x == 0)
        for (int k = 0; k < kStages; k++) mbar_inval(&mbar[k]);
    __syncthreads();
}

// Shared-memory sweep descriptors of one system: [fwd level descriptors
// nfl x int4][bwd level descriptors nbl x int4][fwd lanes nfl][bwd lanes
// nbl][fwd_order n][fwd rp n+1][bwd_order n][bwd rp n+1].
__device__ __forceinline__ bool sweep_desc_fits(const PatternDev& P, const SmemPlan& plan) {
    return P.n <= plan.ycap && 4 * P.n + 5 * (P.nfwd_levels + P.nbwd_levels) + 4 <= plan.dcap &&
           (plan.sc_ent > 0 || plan.flow);
}

// Byte offset (16-byte aligned) of the sweep descriptors in the solve
// area: after the solve vector (ycap doubles) and the Hessenberg block.
__host__ __device__ inline size_t sweep_desc_offset(int ycap, int m) {
    const size_t b = ((size_t)ycap + (size_t)(m + 1) * m + 6 * (size_t)(m + 1)) * sizeof(double);
    return (b + 15) & ~(size_t)15;
}

__device__ __forceinline__ int* sweep_desc_base(const SmemPlan& plan, Smem& sm) {
    return (int*)(sm.uni + sweep_desc_offset(plan.ycap, plan.m));
}

struct SweepDesc {
    const int4 *f_ld, *b_ld;
    const int *f_lg, *b_lg, *f_ord, *f_rp, *b_ord, *b_rp;
    // The pattern's own arrays in global memory (systems whose solve vector
    // or descriptors do not fit shared memory).
    __device__ explicit SweepDesc(const PatternDev& P) {
        const int nfl = P.nfwd_levels, nbl = P.nbwd_levels;
        f_ld = (const int4*)P.fwd_ldesc;
        b_ld = (const int4*)P.bwd_ldesc;
        f_lg = P.fwd_ldesc + 4 * nfl;
        b_lg = P.bwd_ldesc + 4 * nbl;
        f_ord = P.fwd_order;
        f_rp = P.lrp;
        b_ord = P.bwd_order;
        b_rp = P.urp;
    }
    // The packed copy load_sweep_desc wrote to shared memory at d.
    __device__ SweepDesc(const PatternDev& P, const int* d) {
        const int n = P.n, nfl = P.nfwd_levels, nbl = P.nbwd_levels;
        f_ld = (const int4*)d;
        b_ld = f_ld + nfl;
        f_lg = (const int*)(b_ld + nbl);
        b_lg = f_lg + nfl;
        f_ord = b_lg + nbl;
        f_rp = f_ord + n;
        b_ord = f_rp + n + 1;
        b_rp = b_ord + n;
    }
};

__device__ void load_sweep_desc(const PatternDev& P, int* d) {
    const int n = P.n, nfl = P.nfwd_levels, nbl = P.nbwd_levels;
    const SweepDesc sd(P, d);
    int* f_ld = (int*)sd.f_ld;
    int* b_ld = (int*)sd.b_ld;
    int* f_lg = (int*)sd.f_lg;
    int* b_lg = (int*)sd.b_lg;
    int* f_ord = (int*)sd.f_ord;
    int* f_rp = (int*)sd.f_rp;
    int* b_ord = (int*)sd.b_ord;
    int* b_rp = (int*)sd.b_rp;
    for (int t = threadIdx.x; t < 4 * nfl; t += blockDim.x) f_ld[t] = P.fwd_ldesc[t];
    for (int t = threadIdx.x; t < 4 * nbl; t += blockDim.x) b_ld[t] = P.bwd_ldesc[t];
    for (int t = threadIdx.x; t < nfl; t += blockDim.x) f_lg[t] = P.fwd_ldesc[4 * nfl + t];
    for (int t = threadIdx.x; t < nbl; t += blockDim.x) b_lg[t] = P.bwd_ldesc[4 * nbl + t];
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        f_ord[t] = P.fwd_order[t];
        b_ord[t] = P.bwd_order[t];
    }
    for (int t = threadIdx.x; t <= n; t += blockDim.x) {
        f_rp[t] = P.lrp[t];
        b_rp[t] = P.urp[t];
    }
}

// Stage ring of the level-synchronous sweeps, after the descriptors.
__device__ __forceinline__ char* sweep_stage_base(const SmemPlan& plan, Smem& sm) {
    return (char*)(sweep_desc_base(plan, sm) + ((plan.dcap + 3) & ~3));
}

// y := U^-1 L^-1 rhs with the level-synchronous sweeps (descriptors sd in
// shared or global memory, stage ring at stage).  y may be global memory:
// the sweep barriers order its writes and reads inside the CTA.
template <typename VT>
__device__ void cta_lu_apply_levels(const SysDev& S, const PatternDev& P, const SmemPlan& plan,
                                    const double* rhs, double* y, const SweepDesc& sd, char* stage,
                                    double* part) {
    const int n = P.n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = rhs[i];
    __syncthreads();
    const long long t0 = clock64();
    const bool gy = P.n > plan.ycap;
    if (gy)
        staged_sweep<VT, false, true>(P.nfwd_levels, sd.f_ld, sd.f_lg, sd.f_ord, sd.f_rp, P.lci, (const VT*)S.lval,
                                      nullptr, y, stage, plan.sc_ent, plan.sc_rows, part, &S.stats->status);
    else
        staged_sweep<VT, false, false>(P.nfwd_levels, sd.f_ld, sd.f_lg, sd.f_ord, sd.f_rp, P.lci,
                                       (const VT*)S.lval, nullptr, y, stage, plan.sc_ent, plan.sc_rows, part, &S.stats->status);
    const long long t1 = clock64();
    if (P.dtail > 0) {
        tail_forward<VT>(P, (const VT*)S.tail, (const VT*)S.tinv, y, S.stats);
        tail_backward<VT>(P, (const VT*)S.tail, (const VT*)S.tinv, y, S.stats);
    }
    const long long t2 = clock64();
    if (gy)
        staged_sweep<VT, true, true>(P.nbwd_levels, sd.b_ld, sd.b_lg, sd.b_ord, sd.b_rp, P.uci, (const VT*)S.uval,
                                     (const VT*)S.udiag_bwd, y, stage, plan.sc_ent, plan.sc_rows, part, &S.stats->status);
    else
        staged_sweep<VT, true, false>(P.nbwd_levels, sd.b_ld, sd.b_lg, sd.b_ord, sd.b_rp, P.uci, (const VT*)S.uval,
                                      (const VT*)S.udiag_bwd, y, stage, plan.sc_ent, plan.sc_rows, part, &S.stats->status);
    if (threadIdx.x == 0) {
        S.stats->cyc_lsolve += t1 - t0;
        S.stats->cyc_tail += t2 - t1;
        S.stats->cyc_usolve += clock64() - t2;
    }
}

// ---------------------------------------------------------------------------
// Dataflow triangular sweeps with the solve vector in shared memory.  Warp w
// takes the rows w, w + NW, w + 2 NW, ... of a sweep order.  The order is
// level-sorted, so every dependency of a row comes before it; the smallest
// unfinished row therefore always has its dependencies done and its warp at
// it (a warp's earlier rows are smaller), and the sweep cannot deadlock.
// There is no CTA barrier inside a sweep and no ready flag: every output
// slot starts as a signalling-NaN bit pattern, which arithmetic never
// produces, a row's result is one 8-byte store, and a reader polls the value
// it needs.  Each warp stages its own rows in a private ring of
// kFlowSlots shared-memory slots, kFlowSlots - 1 rows ahead, by cp.async
// (column indices, values, the right-hand side and the reciprocal
// diagonal; a row's entries past kFlowCap are read from global memory, four
// chunks of 32 in flight), so a row waits only for its dependencies.
// ---------------------------------------------------------------------------
constexpr long long kFlowSentinel = 0x7ff00000deadbeefll;   // signalling NaN
constexpr int kFlowSlots = 3, kFlowCap = 128;

// One ring slot: kFlowCap column indices, kFlowCap values, the row's
// right-hand side (fp64) and its reciprocal diagonal (VT).
__host__ __device__ inline size_t flow_slot_bytes(int vsize) { return (size_t)kFlowCap * (4 + vsize) + 16; }
__host__ __device__ inline size_t flow_ring_bytes(int nwarps, int vsize) {
    return (size_t)nwarps * kFlowSlots * flow_slot_bytes(vsize);
}

// out[j] once written (bounded wait: after kSpinLimit polls, or at once when
// *abort is set, the wait gives up, sets ST_WAIT_TIMEOUT and returns the
// sentinel, a NaN).
__device__ __noinline__ double flow_wait(const double* out, int j, int* abort, int& bad) {
    const volatile long long* w = (const volatile long long*)out + j;
    const volatile int* ab = abort;
    long long v, it = 0;
    while ((v = *w) == kFlowSentinel) {
        if (++it > 32) {
            if (*ab) break;
            if (it > kSpinLimit) {
                atomicExch(abort, 1);
                break;
            }
            __nanosleep(32);
        }
    }
    if (v == kFlowSentinel) bad |= ST_WAIT_TIMEOUT;
    return __longlong_as_double(v);
}

__device__ __forceinline__ double flow_take(const double* out, int j, long long raw, int* abort, int& bad) {
    return raw != kFlowSentinel ? __longlong_as_double(raw) : flow_wait(out, j, abort, bad);
}

// Four entries per lane: sum into a[0..3] of v * out[j] (j < 0: none).
__device__ __forceinline__ void flow_acc4(const int* jj, const double* vv, const double* out, int* abort, int& bad,
                                          double* a) {
    const volatile long long* vo = (const volatile long long*)out;
    long long raw[4];
#pragma unroll
    for (int q = 0; q < 4; q++) raw[q] = jj[q] >= 0 ? vo[jj[q]] : 0ll;
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (jj[q] >= 0) a[q] = fma(vv[q], flow_take(out, jj[q], raw[q], abort, bad), a[q]);
}

// out[order[r]] := (rhs[order[r]] - sum_e val[e] out[ci[e]]) (* rdg[r] for
// U) over the rows r < nrows of a sweep order, entries e in [rp[r], rp[r+1]).
// ring: this CTA's staging area (flow_ring_bytes).  rhs may be global or
// shared memory.
template <typename VT, bool UPPER>
__device__ __noinline__ void flow_sweep(int nrows, const int* order, const int* rp, const int* ci, const VT* val,
                                        const VT* rdg, const double* rhs, double* out, char* ring, int* abort,
                                        int& bad) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const size_t sb = flow_slot_bytes(sizeof(VT));
    char* my = ring + (size_t)warp * kFlowSlots * sb;
    const bool rglob = __isGlobal(rhs);
    auto issue = [&](int k) {
        const int idx = warp + k * nw;
        if (idx < nrows) {
            const int b = rp[idx], m = min(rp[idx + 1] - b, kFlowCap);
            char* s = my + (size_t)(k % kFlowSlots) * sb;
            int* sc = (int*)s;
            VT* sv = (VT*)(s + (size_t)kFlowCap * 4);
            double* sx = (double*)(s + (size_t)kFlowCap * (4 + sizeof(VT)));
            for (int t = lane; t < m; t += 32) {
                cp_async_4(sc + t, ci + b + t);
                cp_async_val(sv + t, val + b + t);
            }
            if (lane == 0 && rglob) cp_async_8(sx, rhs + order[idx]);
            if (UPPER && lane == 1) cp_async_val((VT*)(sx + 1), rdg + idx);
        }
        cp_async_commit();
    };
    for (int k = 0; k < kFlowSlots - 1; k++) issue(k);
    for (int k = 0, idx = warp; idx < nrows; k++, idx += nw) {
        issue(k + kFlowSlots - 1);
        cp_async_wait_group<kFlowSlots - 1>();
        __syncwarp();
        const char* s = my + (size_t)(k % kFlowSlots) * sb;
        const int* sc = (const int*)s;
        const VT* sv = (const VT*)(s + (size_t)kFlowCap * 4);
        const double* sx = (const double*)(s + (size_t)kFlowCap * (4 + sizeof(VT)));
        const int i = order[idx], b = rp[idx], e = rp[idx + 1];
        const int m = min(e - b, kFlowCap);
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        for (int t0 = lane; t0 < m; t0 += 128) {
            int jj[4];
            double vv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int t = t0 + 32 * q;
                jj[q] = t < m ? sc[t] : -1;
                vv[q] = t < m ? ValTraits<VT>::load(sv + t) : 0.0;
            }
            flow_acc4(jj, vv, out, abort, bad, a);
        }
        for (int p0 = b + kFlowCap + lane; p0 < e; p0 += 128) {
            int jj[4];
            double vv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int p = p0 + 32 * q;
                jj[q] = p < e ? ci[p] : -1;
                vv[q] = p < e ? ValTraits<VT>::load(val + p) : 0.0;
            }
            flow_acc4(jj, vv, out, abort, bad, a);
        }
        const double acc = warp_sum((a[0] + a[1]) + (a[2] + a[3]));
        if (lane == 0) {
            const double r = (rglob ? sx[0] : rhs[i]) - acc;
            ((volatile double*)out)[i] = UPPER ? r * ValTraits<VT>::load((const VT*)(sx + 1)) : r;
        }
        __syncwarp();   // the slot is staged again by the next issue
    }
    cp_async_wait_all();
    __syncwarp();
}

// y := U^-1 L^-1 rhs with the dataflow sweeps: forward into y, the dense
// trailing block in place, backward into y2 (n doubles of shared memory),
// copied back to y.  ring: the staging area of flow_sweep.
template <typename VT>
__device__ void cta_lu_apply_flow(const SysDev& S, const PatternDev& P, const SweepDesc& sd, const double* rhs,
                                  double* y, double* y2, char* ring, Smem& sm, int& bad) {
    const int n = P.n, k0 = P.k0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) ((long long*)y)[i] = kFlowSentinel;
    if (threadIdx.x == 0) sm.ctl[3] = 0;
    __syncthreads();
    const long long t0 = clock64();
    flow_sweep<VT, false>(n, sd.f_ord, sd.f_rp, P.lci, (const VT*)S.lval, (const VT*)nullptr, rhs, y, ring,
                          &sm.ctl[3], bad);
    __syncthreads();
    const long long t1 = clock64();
    if (P.dtail > 0) {
        tail_forward<VT>(P, (const VT*)S.tail, (const VT*)S.tinv, y, S.stats);
        tail_backward<VT>(P, (const VT*)S.tail, (const VT*)S.tinv, y, S.stats);
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        ((long long*)y2)[i] = i < k0 ? kFlowSentinel : __double_as_longlong(y[i]);
    __syncthreads();
    const long long t2 = clock64();
    flow_sweep<VT, true>(k0, sd.b_ord, sd.b_rp, P.uci, (const VT*)S.uval, (const VT*)S.udiag_bwd, y, y2, ring,
                         &sm.ctl[3], bad);
    __syncthreads();
    for (int i = threadIdx.x; i < k0; i += blockDim.x) y[i] = y2[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        S.stats->cyc_lsolve += t1 - t0;
        S.stats->cyc_tail += t2 - t1;
        S.stats->cyc_usolve += clock64() - t2;
    }
}

// Second solve vector and staging ring of the dataflow sweeps, where the
// level sweeps' stage ring would be.
__device__ __forceinline__ double* flow_y2_base(const SmemPlan& plan, Smem& sm) {
    return (double*)sweep_stage_base(plan, sm);
}
__device__ __forceinline__ char* flow_ring_base(const SmemPlan& plan, Smem& sm) {
    return (char*)sweep_stage_base(plan, sm) + (((size_t)plan.ycap * 8 + 15) & ~(size_t)15);
}

// Dispatch: the dataflow sweeps of shared-memory solve vectors when the
// plan chose them (the second vector where the stage ring would be), else
// level-synchronous sweeps when the launch has a stage ring (sd != nullptr:
// descriptors in shared memory when they fit, else read from the pattern in
// global memory), else the per-row dataflow version over global memory.
template <typename VT>
__device__ __forceinline__ void lu_apply(const SysDev& S, const SmemPlan& plan, const double* rhs,
                                         double* y, Smem& sm, const SweepDesc* sd, int& bad) {
    const PatternDev& P = *S.pat;
    if (plan.flow && sd && P.n <= plan.ycap)
        cta_lu_apply_flow<VT>(S, P, *sd, rhs, y, flow_y2_base(plan, sm), flow_ring_base(plan, sm), sm, bad);
    else if (sd) cta_lu_apply_levels<VT>(S, P, plan, rhs, y, *sd, sweep_stage_base(plan, sm), sm.red);
    else cta_lu_apply<VT>(P, (const VT*)S.lval, (const VT*)S.uval, (const VT*)S.udiag, (const VT*)S.tail,
                          (const VT*)S.tinv, rhs, y, sm, bad, S.stats);
}

// The sweep descriptors of a solve: loaded into shared memory when they fit
// (returns the packed copy), else the pattern's global arrays when the
// launch has a stage ring, else none (dataflow sweeps).  Ends with a CTA
// barrier.
__device__ const SweepDesc* prepare_sweeps(const PatternDev& P, const SmemPlan& plan, Smem& sm, SweepDesc* buf) {
    const SweepDesc* sd = nullptr;
    if (sweep_desc_fits(P, plan)) {
        int* d = sweep_desc_base(plan, sm);
        load_sweep_desc(P, d);
        *buf = SweepDesc(P, d);
        sd = buf;
    } else if (plan.sc_ent > 0 || plan.flow) {
        *buf = SweepDesc(P);
        sd = buf;
    }
    __syncthreads();
    return sd;
}

// out = A x (RESID: out = bt - A x) with A in SELL-C-sigma, C = 32, values AT.
template <typename AT, bool RESID>
__device__ void cta_spmv(const PatternDev& P, const AT* vals, const double* xin,
                         const double* bt, double* out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int s = warp; s < P.nslices; s += nw) {
        const int base = P.sell_ptr[s];
        const int L = (P.sell_ptr[s + 1] - base) >> 5;
        // Four independent partial sums: four loads per lane in flight.
        double acc = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        int t = 0;
        for (; t + 3 < L; t += 4) {
            const int e = base + (t << 5) + lane;
            const int c0 = P.sell_col[e], c1 = P.sell_col[e + 32], c2 = P.sell_col[e + 64], c3 = P.sell_col[e + 96];
            acc = fma((double)vals[e], xin[c0], acc);
            a1 = fma((double)vals[e + 32], xin[c1], a1);
            a2 = fma((double)vals[e + 64], xin[c2], a2);
            a3 = fma((double)vals[e + 96], xin[c3], a3);
        }
        for (; t < L; t++) {
            const int e = base + (t << 5) + lane;
            acc = fma((double)vals[e], xin[P.sell_col[e]], acc);
        }
        acc = (acc + a1) + (a2 + a3);
        const int row = P.sell_perm[(s << 5) + lane];
        if (row >= 0) out[row] = RESID ? bt[row] - acc : acc;
    }
}

// ---------------------------------------------------------------------------
// fp16 inner products.  Ruiz equilibration of A (position space, SELL
// order) gives rs, cs with every row and column maximum of |rs_i a_ij cs_j|
// near 1; the scaled values are stored in fp16 only when every nonzero one
// lies in the fp16 normal range [2^-14, 65504], so no value underflows or
// overflows in storage (else the fp32 values are used and ST_FP16_OFF says
// so).  The scaling is the one lusp_sell_create applies (spmv.cu,
// lusp_ruiz_csr), operation for operation: row maxima of |a| rs_i cs_j,
// rs_i /= sqrt(max), then column maxima, cs_j /= sqrt(max), until every
// maximum is within 1e-6 of 1, at most kRuizSweeps sweeps.  The reference
// equilibrates the same way on the host (bench/test_lu_gpu_par.cu:237-260,
// 30 sweeps, early stop 1e-6).
// ---------------------------------------------------------------------------
constexpr int kRuizSweeps = 30;

// colmax: n doubles of global scratch.  Returns whether fp16 storage fits.
__device__ bool ruiz_sell16(const SysDev& S, const PatternDev& P, double* colmax, Smem& sm) {
    const int n = P.n;
    double* rs = S.rs;
    double* cs = S.cs;
    __half* h = (__half*)S.sell16;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        rs[i] = 1.0;
        cs[i] = 1.0;
    }
    __syncthreads();
    const int nq = 32 * P.nslices;
    for (int it = 0; it < kRuizSweeps; it++) {
        double dev = 0.0;
        // Rows: one thread per SELL row (a row's entries are one lane of its slice).
        for (int q = threadIdx.x; q < nq; q += blockDim.x) {
            const int r = P.sell_perm[q];
            if (r < 0) continue;
            const int base = P.sell_ptr[q >> 5], L = (P.sell_ptr[(q >> 5) + 1] - base) >> 5;
            const double rr = rs[r];
            double m = 0.0;
            for (int t = 0; t < L; t++) {
                const int e = base + (t << 5) + (q & 31);
                if (P.sell_src[e] >= 0) m = fmax(m, fabs(S.sell64[e]) * rr * cs[P.sell_col[e]]);
            }
            if (m > 0.0) {
                rs[r] = rr / sqrt(m);
                dev = fmax(dev, fabs(1.0 - m));
            }
        }
        for (int j = threadIdx.x; j < n; j += blockDim.x) colmax[j] = 0.0;
        __syncthreads();
        // Columns: maxima by atomic max on the bit patterns (non-negative).
        for (int q = threadIdx.x; q < nq; q += blockDim.x) {
            const int r = P.sell_perm[q];
            if (r < 0) continue;
            const int base = P.sell_ptr[q >> 5], L = (P.sell_ptr[(q >> 5) + 1] - base) >> 5;
            const double rr = rs[r];
            for (int t = 0; t < L; t++) {
                const int e = base + (t << 5) + (q & 31);
                if (P.sell_src[e] < 0) continue;
                const int c = P.sell_col[e];
                const double a = fabs(S.sell64[e]) * rr * cs[c];
                atomicMax((unsigned long long*)(colmax + c), (unsigned long long)__double_as_longlong(a));
            }
        }
        __syncthreads();
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const double m = colmax[j];
            if (m > 0.0) {
                cs[j] = cs[j] / sqrt(m);
                dev = fmax(dev, fabs(1.0 - m));
            }
        }
        dev = block_max(dev, sm.red);
        if (dev < 1e-6) break;
    }
    // fp16 values (padding 0) and the range of the scaled nonzeros.
    double mn = INFINITY, mx = 0.0;
    for (int q = threadIdx.x; q < nq; q += blockDim.x) {
        const int r = P.sell_perm[q];
        const int base = P.sell_ptr[q >> 5], L = (P.sell_ptr[(q >> 5) + 1] - base) >> 5;
        for (int t = 0; t < L; t++) {
            const int e = base + (t << 5) + (q & 31);
            double a = 0.0;
            if (r >= 0 && P.sell_src[e] >= 0) a = S.sell64[e] * rs[r] * cs[P.sell_col[e]];
            h[e] = __double2half(a);
            const double aa = fabs(a);
            if (aa != 0.0) {
                mn = fmin(mn, aa);
                mx = fmax(mx, aa);
            }
        }
    }
    mn = block_min(mn, sm.red);
    mx = block_max(mx, sm.red);
    return mn >= 6.103515625e-05 && mx <= 65504.0;
}

// out = A x with the fp16 values: out_r = (sum_c h_rc (x_c / cs_c)) / rs_r,
// fp64 accumulation; xc: n doubles of scratch.
__device__ void cta_spmv16(const PatternDev& P, const __half* vals, const double* rs, const double* cs,
                           const double* xin, double* xc, double* out) {
    for (int i = threadIdx.x; i < P.n; i += blockDim.x) xc[i] = xin[i] / cs[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int s = warp; s < P.nslices; s += nw) {
        const int base = P.sell_ptr[s];
        const int L = (P.sell_ptr[s + 1] - base) >> 5;
        double acc = 0.0, a1 = 0.0;
        int t = 0;
        for (; t + 1 < L; t += 2) {
            const int e = base + (t << 5) + lane;
            acc = fma((double)__half2float(vals[e]), xc[P.sell_col[e]], acc);
            a1 = fma((double)__half2float(vals[e + 32]), xc[P.sell_col[e + 32]], a1);
        }
        if (t < L) {
            const int e = base + (t << 5) + lane;
            acc = fma((double)__half2float(vals[e]), xc[P.sell_col[e]], acc);
        }
        const int row = P.sell_perm[(s << 5) + lane];
        if (row >= 0) out[row] = (acc + a1) / rs[row];
    }
}

__device__ __forceinline__ double cta_dot(const double* a, const double* b, int n, Smem& sm) {
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s = fma(a[i], b[i], s);
    return block_sum(s, sm.red);
}

// A in SELL order for the solve's products, from the system's input
// values: fp64 (outer residual, direct-solve residual) and, when the inner
// products use it, fp32.  Ends with a CTA barrier.
__device__ void build_sell_values(const SysDev& S, const PatternDev& P, bool f32) {
    const int total = P.sell_total, nt = blockDim.x;
    // Four entries per thread in flight (the value reads are gathers).
    for (int t0 = threadIdx.x; t0 < total; t0 += 4 * nt) {
        int src[4];
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) src[q] = t0 + q * nt < total ? P.sell_src[t0 + q * nt] : -1;
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = src[q] >= 0 ? S.a_val[src[q]] : 0.0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int t = t0 + q * nt;
            if (t < total) {
                S.sell64[t] = v[q];
                if (f32) S.sell32[t] = (float)v[q];
            }
        }
    }
    __syncthreads();
}

// Direct solve x = Q U^-1 L^-1 P b with the stored factors, then the fp64
// residual of the result.
template <typename VT>
__device__ void direct_phase(const SysDev& S, const SmemPlan& plan, char* smem_base) {
    const PatternDev& P = *S.pat;
    const int n = P.n;
    Smem sm(smem_base, plan);
    double* bt = S.work;
    double* xt = bt + n;
    double* r = xt + n;
    double* yg = r + 3 * n;
    double* y = (n <= plan.ycap) ? (double*)sm.uni : yg;
    int bad = 0;
    if (threadIdx.x == 0) S.stats->status &= ~kSolveBits;
    for (int i = threadIdx.x; i < n; i += blockDim.x) bt[i] = S.b[P.rowat[i]];
    build_sell_values(S, P, false);
    SweepDesc sdb(P);
    const SweepDesc* desc = prepare_sweeps(P, plan, sm, &sdb);
    const double nb = sqrt(cta_dot(bt, bt, n, sm));
    lu_apply<VT>(S, plan, bt, y, sm, desc, bad);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        xt[i] = y[i];
        S.x[P.q[i]] = y[i];
    }
    __syncthreads();
    cta_spmv<double, true>(P, S.sell64, xt, bt, r);
    __syncthreads();
    const double rn = sqrt(cta_dot(r, r, n, sm));
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && bad) atomicOr(&S.stats->status, bad);
    if (threadIdx.x == 0) {
        const double res = nb > 0 ? rn / nb : rn;
        S.stats->res[0] = res;
        S.stats->nres = 1;
        S.stats->outer_iters = 0;
        S.stats->inner_iters = 0;
        if (!isfinite(res)) atomicOr(&S.stats->status, (int)ST_NONFINITE);
    }
    __syncthreads();
}

// Arnoldi orthogonalization of w against the first j + 1 basis vectors
// (V_i at V + i n) for j < kFusedDots, every thread on every dot product.
// Both helpers are calls: inlined into the GMRES loop, their addresses stay
// live across the preconditioner application and the level sweeps it calls
// run out of registers (spill loads in every level step).
constexpr int kFusedDots = 3;

// d[i] = V_i . w (i <= j) and, when wsq is given, |w|^2 from one sweep over
// the vectors; all threads receive the sums.
__device__ __noinline__ void cgs_dots(const double* V, int n, int j, const double* w, double* d, double* wsq,
                                      Smem& sm) {
    double s[kFusedDots + 1];
#pragma unroll
    for (int i = 0; i <= kFusedDots; i++) s[i] = 0.0;
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const double we = w[e];
        if (wsq) s[kFusedDots] = fma(we, we, s[kFusedDots]);
#pragma unroll
        for (int i = 0; i < kFusedDots; i++)
            if (i <= j) s[i] = fma(V[(size_t)i * n + e], we, s[i]);
    }
    block_sum2(s[0], s[kFusedDots], sm.red);
    if (j >= 1) block_sum2(s[1], s[2], sm.red);
#pragma unroll
    for (int i = 0; i < kFusedDots; i++) d[i] = i <= j ? s[i] : 0.0;
    if (wsq) *wsq = s[kFusedDots];
}

// w -= sum_{i <= j} d[i] V_i; returns the new |w|^2 (all threads).
__device__ __noinline__ double cgs_update(const double* V, int n, int j, const double* d, double* w, Smem& sm) {
    double nrm = 0.0;
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        double acc = w[e];
#pragma unroll
        for (int i = 0; i < kFusedDots; i++)
            if (i <= j) acc = fma(-d[i], V[(size_t)i * n + e], acc);
        w[e] = acc;
        nrm = fma(acc, acc, nrm);
    }
    return block_sum(nrm, sm.red);
}

// ---------------------------------------------------------------------------
// GMRES-IR: restarted, right-preconditioned GMRES on P A Q with the stored
// factors as preconditioner (VT), inner products A z with AT values; outer
// residual b - A x, Arnoldi (classical Gram-Schmidt: for the first
// kFusedDots basis vectors a second pass only when the first cancels more
// than half of |w|^2, beyond them always two passes), Givens
// rotations, least-squares update and solution update in fp64.
// Workspace (doubles): bt, xt, r, z, w, yg (n each), V ((m+1) n), xprev (n).
// ---------------------------------------------------------------------------
template <typename VT, typename AT>
__device__ void gmres_phase(const SysDev& S, const SmemPlan& plan, char* smem_base,
                            const SolveParams& prm) {
    const PatternDev& P = *S.pat;
    const int n = P.n;
    const int m = prm.m;
    Smem sm(smem_base, plan);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double* bt = S.work;
    double* xt = bt + n;
    double* r = xt + n;
    double* z = r + n;
    double* w = z + n;
    double* yg = w + n;
    double* V = yg + n;
    double* xprev = V + (size_t)(m + 1) * n;   // iterate before the last correction
    double* Zb = xprev + n;                      // [m x n] preconditioned basis z_j = M^-1 v_j
    // Shared: y (optional) | H[(m+1) x m] | g, cs, sn, h, h2, yc
    double* ys = (double*)sm.uni;
    double* H = ys + plan.ycap;
    double* g = H + (size_t)(m + 1) * m;
    double* cs = g + (m + 1);
    double* sn = cs + m;
    double* h = sn + m;
    double* yc = h + (m + 1);
    double* y = (n <= plan.ycap) ? ys : yg;
    const VT* udiag = (const VT*)S.udiag;
    const VT* tail = (const VT*)S.tail;
    constexpr bool kHalf = std::is_same<AT, __half>::value;
    const void* ainner = sizeof(AT) == 8 ? (const void*)S.sell64 : (const void*)S.sell32;
    int bad = 0;
    int status = 0;
    int inner_total = 0, outer_done = 0, nres = 0;
    if (threadIdx.x == 0) S.stats->status &= ~kSolveBits;

    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        bt[i] = S.b[P.rowat[i]];
        xt[i] = 0.0;
    }
    build_sell_values(S, P, sizeof(AT) != 8);
    SweepDesc sdb(P);
    const SweepDesc* desc = prepare_sweeps(P, plan, sm, &sdb);
    bool use16 = false;
    if constexpr (kHalf) {
        // V holds nothing yet: its first n doubles serve the column maxima.
        use16 = ruiz_sell16(S, P, V, sm);
        if (!use16 && threadIdx.x == 0) atomicOr(&S.stats->status, (int)ST_FP16_OFF);
    }
    const double nb = sqrt(cta_dot(bt, bt, n, sm));
    if (!(nb > 0.0)) {
        for (int i = threadIdx.x; i < n; i += blockDim.x) S.x[i] = 0.0;
        if (threadIdx.x == 0) {
            S.stats->res[0] = 0.0;
            S.stats->nres = 1;
            if (!isfinite(nb)) atomicOr(&S.stats->status, (int)ST_NONFINITE);
        }
        __syncthreads();
        return;
    }
    double res_prev = INFINITY;
    // Forward-error estimate of the current iterate from the last two
    // corrections: contraction rho = |dx_k| / |dx_k-1|, remaining error
    // ~ |dx_k| rho / (1 - rho) relative to |x|.
    double dx_prev = 0.0, err_est = INFINITY;
    for (int outer = 0;; outer++) {
        if (outer == 0) {
            for (int i = threadIdx.x; i < n; i += blockDim.x) r[i] = bt[i];
        } else {
            cta_spmv<double, true>(P, S.sell64, xt, bt, r);
        }
        __syncthreads();
        const double beta = sqrt(cta_dot(r, r, n, sm));
        const double res = beta / nb;
        if (nres < 16) {
            if (threadIdx.x == 0) S.stats->res[nres] = res;
            nres++;
        }
        // A correction that made the residual worse (or non-finite) is
        // undone: the result is the best iterate, the status says why.
        if (outer > 0 && !(res <= res_prev)) {
            for (int i = threadIdx.x; i < n; i += blockDim.x) xt[i] = xprev[i];
            __syncthreads();
            status |= isfinite(res) ? ST_STAGNATED : ST_NONFINITE;
            break;
        }
        if (!isfinite(res)) { status |= ST_NONFINITE; break; }
        // Converged when the residual is small and the iterate has stopped
        // moving (or the residual is at fp64 round-off, nothing left to gain).
        if (res <= prm.rtol && (err_est <= prm.xtol || res <= 1e-15)) break;
        if (outer >= prm.max_outer) { status |= ST_NOT_CONVERGED; break; }
        if (outer > 0 && res > prm.stag_ratio * res_prev) { status |= ST_STAGNATED; break; }
        res_prev = res;
        const double inv_beta = 1.0 / beta;
        for (int i = threadIdx.x; i < n; i += blockDim.x) V[i] = r[i] * inv_beta;
        if (threadIdx.x == 0) {
            for (int t = 0; t <= m; t++) g[t] = 0.0;
            g[0] = beta;
        }
        // Inner solve: reduce the current residual by inner_rel (a cap at
        // rtol * |b| would stall the outer loop right above rtol).
        const double inner_stop = prm.inner_rel * beta;
        int jj = 0;
        for (int j = 0; j < m; j++) {
            const double* vj = V + (size_t)j * n;
            lu_apply<VT>(S, plan, vj, y, sm, desc, bad);
            // Keep z_j: the correction is then sum_i y_i z_i, without
            // another preconditioner application (flexible-GMRES layout).
            double* zj = Zb + (size_t)j * n;
            for (int e = threadIdx.x; e < n; e += blockDim.x) zj[e] = y[e];
            const long long tsp = clock64();
            if constexpr (kHalf) {
                // r is free inside the inner loop: it holds x / cs.
                if (use16) cta_spmv16(P, (const __half*)S.sell16, S.rs, S.cs, y, r, w);
                else cta_spmv<float, false>(P, S.sell32, y, nullptr, w);
            } else {
                cta_spmv<AT, false>(P, (const AT*)ainner, y, nullptr, w);
            }
            __syncthreads();
            if (threadIdx.x == 0) S.stats->cyc_spmv += clock64() - tsp;
            double wn0, hn;
            if (j < kFusedDots) {
                // Classical Gram-Schmidt against V_0..V_j, all threads on
                // every dot product: one sweep for the dots and |w|^2, one
                // for the update and the new |w|^2; the second pass only
                // when the first cancelled more than half of |w|^2 (Daniel,
                // Gragg, Kaufman and Stewart's reorthogonalization test).
                double d[kFusedDots];
                double wsq;
                cgs_dots(V, n, j, w, d, &wsq, sm);
                wn0 = sqrt(wsq);
                double hsq = cgs_update(V, n, j, d, w, sm);
                if (hsq < 0.5 * wsq) {
                    double d2[kFusedDots];
                    cgs_dots(V, n, j, w, d2, nullptr, sm);
                    hsq = cgs_update(V, n, j, d2, w, sm);
#pragma unroll
                    for (int i = 0; i < kFusedDots; i++) d[i] += d2[i];
                }
                if (threadIdx.x == 0) {
#pragma unroll
                    for (int i = 0; i < kFusedDots; i++)
                        if (i <= j) H[(size_t)i * m + j] = d[i];
                }
                hn = sqrt(hsq);
            } else {
                wn0 = sqrt(cta_dot(w, w, n, sm));
                for (int pass = 0; pass < 2; pass++) {
                    for (int i = warp; i <= j; i += nw) {
                        const double* vi = V + (size_t)i * n;
                        double s = 0.0;
                        for (int e = lane; e < n; e += 32) s = fma(vi[e], w[e], s);
                        s = warp_sum(s);
                        if (lane == 0) {
                            yc[i] = s;
                            if (pass == 0) h[i] = s;
                            else H[(size_t)i * m + j] = h[i] + s;
                        }
                    }
                    __syncthreads();
                    for (int e = threadIdx.x; e < n; e += blockDim.x) {
                        double acc = w[e];
                        for (int i = 0; i <= j; i++) acc = fma(-yc[i], V[(size_t)i * n + e], acc);
                        w[e] = acc;
                    }
                    __syncthreads();
                }
                hn = sqrt(cta_dot(w, w, n, sm));
            }
            inner_total++;
            jj = j + 1;
            const bool breakdown = !(hn > 1e-14 * wn0) || hn == 0.0;
            if (threadIdx.x == 0) {
                for (int i = 0; i < j; i++) {
                    const double t1 = H[(size_t)i * m + j], t2 = H[(size_t)(i + 1) * m + j];
                    H[(size_t)i * m + j] = cs[i] * t1 + sn[i] * t2;
                    H[(size_t)(i + 1) * m + j] = -sn[i] * t1 + cs[i] * t2;
                }
                const double a = H[(size_t)j * m + j];
                const double bb = breakdown ? 0.0 : hn;
                const double rr = sqrt(a * a + bb * bb);
                const double c = rr > 0.0 ? a / rr : 1.0;
                const double s_ = rr > 0.0 ? bb / rr : 0.0;
                cs[j] = c;
                sn[j] = s_;
                H[(size_t)j * m + j] = rr;
                g[j + 1] = -s_ * g[j];
                g[j] = c * g[j];
                sm.red[34] = g[j + 1];
            }
            __syncthreads();
            const double gres = fabs(sm.red[34]);
            if (breakdown || gres <= inner_stop || !isfinite(gres)) break;
            const double inv_hn = 1.0 / hn;
            double* vn = V + (size_t)(j + 1) * n;
            for (int e = threadIdx.x; e < n; e += blockDim.x) vn[e] = w[e] * inv_hn;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            for (int i = jj - 1; i >= 0; i--) {
                double s = g[i];
                for (int t = i + 1; t < jj; t++) s -= H[(size_t)i * m + t] * yc[t];
                const double dgv = H[(size_t)i * m + i];
                yc[i] = dgv != 0.0 ? s / dgv : 0.0;
            }
        }
        __syncthreads();
        // The correction sum_i y_i z_i, applied as it is formed.
        double sy = 0.0, sx = 0.0;
        for (int e = threadIdx.x; e < n; e += blockDim.x) {
            double acc = 0.0;
            for (int i = 0; i < jj; i++) acc = fma(yc[i], Zb[(size_t)i * n + e], acc);
            const double xo = xt[e];
            xprev[e] = xo;
            const double xn = xo + acc;
            xt[e] = xn;
            sy = fma(acc, acc, sy);
            sx = fma(xn, xn, sx);
        }
        block_sum2(sy, sx, sm.red);
        const double ny = sqrt(sy);
        const double nx = sqrt(sx);
        const double dx = nx > 0.0 ? ny / nx : ny;
        if (dx_prev > 0.0) {
            const double rho = fmin(dx / dx_prev, 0.99);
            err_est = dx * rho / (1.0 - rho);
        }
        dx_prev = dx;
        outer_done++;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) S.x[P.q[i]] = xt[i];
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (lane == 0 && bad) atomicOr(&S.stats->status, bad);
    if (threadIdx.x == 0) {
        if (status) atomicOr(&S.stats->status, status);
        S.stats->nres = nres < 16 ? nres : 16;
        S.stats->inner_iters = inner_total;
        S.stats->outer_iters = outer_done;
    }
    __syncthreads();
}

}  // namespace lusp
