// solve_core.cuh -- blocked triangular sweeps on right-hand sides held in
// shared memory, shared by getrs (lu_blocked.cu, lu_vbatched.cu), the
// iterative-refinement correction solves (ir.cu) and the Cholesky solves
// (chol_core.cuh).
//
// One CTA holds NR right-hand sides (column c at sB + c * ldx) and runs a
// sweep over the 32-row diagonal blocks of a triangular factor, ascending or
// descending.  Per block:
//   D  the diagonal block is solved from a copy in shared memory (staged by
//      cp.async while the previous block's update runs: the copy is free again
//      after D's barrier), the right-hand sides spread over the CTA's warps;
//   U  the rows that remain are updated, one warp task per (32 rows, CG
//      columns), each lane one row with its 32 coefficients in registers (FP64:
//      the first task's are loaded before D).
// What bounds it: FP64, the FP64 pipe -- a warp instruction holds its
// scheduler's share of it for 64 cycles whatever its lanes do, so D runs on
// several warps (one warp can use a quarter of the pipe), two columns to a
// warp, and U does no work for columns that are not there; FP32, instruction
// issue and the latency of D (see Diag).
// Measured before and after: at getrs_kernel (lu_blocked.cu).
//
// Every element receives its updates in the order of the CPU oracle
// (oracle/lu_oracle.c, getrs), so results are bit-identical to it.
#pragma once
#include "common.cuh"

namespace mlu {

// Column stride of the right-hand sides in shared memory: a multiple of 16
// bytes, so that a sweep reads consecutive solved values with 16-byte loads.
template <typename T>
__host__ __device__ constexpr int solve_ldx(int n)
{
    const int v = (int)(16 / sizeof(T)), l = (n + v - 1) & ~(v - 1);
    return l % 32 == 0 ? l + v : l;              // columns start in different banks
}

// This thread's warp, turned by a hash of the block index: the few warps that
// solve a diagonal block would otherwise be the same ones, on the same of the
// SM's four schedulers, in every CTA.
__device__ __forceinline__ int turned_warp(int block, int nw)
{
    return (int)(((threadIdx.x >> 5) + ((unsigned)block * 0x9E3779B1u >> 27)) % (unsigned)nw);
}

// The staged diagonal block.  FP64: D[row][column], row stride 33.  FP32: the
// coefficients of one step contiguous, in rows of 36 that are read 16 bytes at
// a time, and the reciprocals of the diagonal.
template <typename T> struct Diag;
template <> struct Diag<double> {
    static constexpr int LD = 33;
    double d[32 * LD];
};
template <> struct Diag<float> {
    static constexpr int LD = 36;
    float d[32 * LD];
    float r[32];
};

// Block [t0, t0 + tb) of the factor by cp.async, all threads.  Rows and columns
// past tb are set to zero.
template <typename T, bool CT>
__device__ __forceinline__ void stage_diag(int n, const T *A, int lda, int t0, int tb, Diag<T> &D)
{
    constexpr int LD = Diag<T>::LD;
    for (int e = threadIdx.x; e < 32 * 32; e += blockDim.x) {
        const int r = e & 31, c = e >> 5;
        T *dst = D.d + (sizeof(T) == 4 && !CT ? c * LD + r : r * LD + c);
        const bool in = r < tb && c < tb && MLU_BC2(t0 + r, t0 + c, n, n, 801);
        cp_async_elem<sizeof(T)>(dst, in ? A + t0 + r + (size_t)(t0 + c) * lda : A, in);
    }
    cp_async_commit();
}

// The coefficients of row i (a row of the factor) for LW columns t0 .. of the
// block, of which tb exist: c(i, t) = A(i, t), or A(t, i) with CT.  Columns past
// tb read as zero.  `vec`: 16-byte loads along t are aligned (CT).
template <typename T, bool CT, int LW>
__device__ __forceinline__ void load_coefs(T (&l)[LW], int n, const T *A, int lda, int i, int t0, int tb, bool vec)
{
    if (tb > 0 && (!MLU_BC2(i, t0, n, n, 802) || !MLU_BC2(i, t0 + min(tb, LW) - 1, n, n, 803))) tb = 0;
    const T *p = CT ? A + (size_t)i * lda + t0 : A + i + (size_t)t0 * lda;
    const size_t step = CT ? 1 : lda;
    if (tb < LW) {
#pragma unroll
        for (int t = 0; t < LW; t++) l[t] = t < tb ? p[t * step] : T(0);
    } else if (CT && vec) {
        if constexpr (sizeof(T) == 8) {
#pragma unroll
            for (int t = 0; t < LW; t += 2) {
                const double2 v = *reinterpret_cast<const double2 *>(p + t);
                l[t] = v.x;
                l[t + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int t = 0; t < LW; t += 4) {
                const float4 v = *reinterpret_cast<const float4 *>(p + t);
                l[t] = v.x;
                l[t + 1] = v.y;
                l[t + 2] = v.z;
                l[t + 3] = v.w;
            }
        }
    } else {
#pragma unroll
        for (int t = 0; t < LW; t++) l[t] = p[t * step];
    }
}

// Consecutive solved values, 16 bytes at a time.  Volatile, so that the
// compiler re-reads them per task instead of keeping them in registers.
__device__ __forceinline__ void lds16(const double *p, double (&v)[2])
{
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n"
                 : "=d"(v[0]), "=d"(v[1]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void lds16(const float *p, float (&v)[4])
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}

// acc[c] = fma(-l_t, x_ct, acc[c]) over LW columns t of the block, of which tb
// exist, ascending or descending; x: the solved values of column 0.
template <typename T, int CG, bool ASC, int LW>
__device__ __forceinline__ void update_row(T (&acc)[CG], const T (&l)[LW], const T *x, int ldx, int tb)
{
    constexpr int V = 16 / sizeof(T);
    if (tb >= LW) {
#pragma unroll
        for (int b = 0; b < LW / V; b++) {
            const int t = (ASC ? b : LW / V - 1 - b) * V;
#pragma unroll
            for (int c = 0; c < CG; c++) {
                T v[V];
                lds16(x + c * ldx + t, v);
#pragma unroll
                for (int u = 0; u < V; u++) {
                    const int k = ASC ? u : V - 1 - u;
                    acc[c] = Prec<T>::fma_(-l[t + k], v[k], acc[c]);
                }
            }
        }
    } else {
#pragma unroll
        for (int b = 0; b < LW; b++) {
            const int t = ASC ? b : LW - 1 - b;
            if (t < tb) {
#pragma unroll
                for (int c = 0; c < CG; c++) acc[c] = Prec<T>::fma_(-l[t], x[c * ldx + t], acc[c]);
            }
        }
    }
}

// FP64, one column (x: its block) by one warp, lane = row: xt = y_t (times the
// reciprocal of the diagonal when not UNIT), then y_i = fma(-c(i, t), xt, y_i)
// for the rows that follow.
template <bool CT, bool ASC, bool UNIT>
__device__ __forceinline__ void diag_rows(const double *D, double *x, int tb)
{
    constexpr int LD = Diag<double>::LD;
    const int lane = threadIdx.x & 31;
    const bool v = lane < tb;
    double y = v ? x[lane] : 0.0, dl = 1.0, rl = 1.0;
    bool plain = true;                         // no diagonal entry needs the division
    if (!UNIT) {
        if (v) dl = D[lane * LD + lane];
        rl = recip(dl);
        plain = !__any_sync(FULL, v && !Prec<double>::normal_or_special(dl));
    }
#pragma unroll 8
    for (int s = 0; s < tb; s++) {
        const int t = ASC ? s : tb - 1 - s;
        const double l = CT ? D[t * LD + lane] : D[lane * LD + t];
        double xt = shfl(y, t);
        if (!UNIT) {
            const double r = shfl(rl, t);
            if (plain) xt = xt * r;
            else xt = rscale(xt, shfl(dl, t), r);
            if (lane == t) y = xt;
        }
        if (ASC ? lane > t : lane < t) y = fma(-l, xt, y);
    }
    if (v) x[lane] = y;
}

// FP64, two columns (x and x + cstep) of a full block by one warp: half a warp
// per column and 16 rows at a time, so that the triangles waste half as many
// lanes: 48 (80 when not UNIT) FP64 warp instructions for both columns instead
// of 64 (128).  False when a diagonal entry needs the division.
template <bool CT, bool ASC, bool UNIT>
__device__ __forceinline__ bool diag_rows_pair(const double *D, double *x, int cstep)
{
    constexpr int LD = Diag<double>::LD;
    const int lane = threadIdx.x & 31, r = lane & 15, h = lane & 16;
    auto coef = [&](int i, int t) { return CT ? D[t * LD + i] : D[i * LD + t]; };
    double rl = 1.0;
    if (!UNIT) {
        const double dl = D[lane * LD + lane];
        rl = recip(dl);
        if (__any_sync(FULL, !Prec<double>::normal_or_special(dl))) return false;
    }
    double *xc = x + (h ? cstep : 0);
    double y[2] = {xc[r], xc[16 + r]};         // rows r and 16 + r of this lane's column
#pragma unroll
    for (int s = 0; s < 2; s++) {
        constexpr int F = ASC ? 0 : 1;         // the half solved first
        const int b = s == 0 ? F : 1 - F, o = 16 * b;
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const int t = ASC ? q : 15 - q;
            double xt = __shfl_sync(FULL, y[b], h + t);
            if (!UNIT) {
                xt = xt * shfl(rl, o + t);
                if (r == t) y[b] = xt;
            }
            if (ASC ? r > t : r < t) y[b] = fma(-coef(o + r, o + t), xt, y[b]);
        }
        if (s == 0) {
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const int t = ASC ? q : 15 - q;
                const double xt = __shfl_sync(FULL, y[F], h + t);
                y[1 - F] = fma(-coef(16 * (1 - F) + r, 16 * F + t), xt, y[1 - F]);
            }
        }
    }
    xc[r] = y[0];
    xc[16 + r] = y[1];
    return true;
}

// FP32: the diagonal block for the nr columns (x: the block of column 0) by one
// warp.  Two triangles of 16 rows, lane = column, in registers with the
// coefficients broadcast from shared memory -- no shuffle is on the chain of 32
// steps -- and between them the 16 x 16 square, all lanes.  About 450 warp
// instructions and 650 cycles for up to eight columns; a step-by-step solve with
// lane = row costs 360 instructions a column and 900 cycles.  A partial block is
// a full one with zero coefficients and right-hand sides (and a diagonal of one)
// past tb: those steps change no value.
template <bool ASC, bool UNIT>
__device__ __forceinline__ void diag_cols(Diag<float> &D, float *x, int ldx, int nr, int tb)
{
    constexpr int LD = Diag<float>::LD;
    const int lane = threadIdx.x & 31;
    float *xc = x + (size_t)min(lane, nr - 1) * ldx;
    if (!UNIT) {
        const float dl = lane < tb ? D.d[lane * LD + lane] : 1.f;
        D.r[lane] = recip(dl);
        const bool plain = !__any_sync(FULL, lane < tb && !Prec<float>::normal_or_special(dl));
        if (!plain) {                            // some row needs the division
            __syncwarp();
            if (lane < nr)
                for (int s = 0; s < tb; s++) {
                    const int t = ASC ? s : tb - 1 - s;
                    const float xt = rscale(xc[t], D.d[t * LD + t], D.r[t]);
                    xc[t] = xt;
                    for (int i = ASC ? t + 1 : 0; i < (ASC ? tb : t); i++) xc[i] = fmaf(-D.d[t * LD + i], xt, xc[i]);
                }
            return;
        }
        __syncwarp();
    }
#pragma unroll
    for (int s = 0; s < 2; s++) {
        const int o = 16 * ((s == 0) == ASC ? 0 : 1), o2 = 16 - o;   // this triangle's rows, the other's
        if (o >= tb) continue;                   // a block of at most 16 rows: its second half is empty
        if (lane < nr) {
            float y[16];
#pragma unroll
            for (int i = 0; i < 16; i++) y[i] = o + i < tb ? xc[o + i] : 0.f;
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const int t = ASC ? k : 15 - k;
                if (!UNIT) y[t] = y[t] * D.r[o + t];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (ASC ? 4 * q + 3 > t : 4 * q < t) {
                        const float4 v = *reinterpret_cast<const float4 *>(D.d + (o + t) * LD + o + 4 * q);
                        const float l[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            if (ASC ? 4 * q + u > t : 4 * q + u < t) y[4 * q + u] = fmaf(-l[u], y[t], y[4 * q + u]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (o + i < tb) xc[o + i] = y[i];
        }
        if (s == 0 && tb > 16) {
            __syncwarp();
            const int ts = min(16, tb - o);       // columns of the square (the rest are zero)
            for (int e = lane; e < 16 * nr; e += 32) {
                const int r = o2 + (e & 15);
                float *xe = x + (size_t)(e >> 4) * ldx;
                if (r >= tb || ts <= 0) continue;
                float acc = xe[r];
                if (ts == 16) {
#pragma unroll
                    for (int k = 0; k < 16; k++) {
                        const int t = o + (ASC ? k : 15 - k);
                        acc = fmaf(-D.d[t * LD + r], xe[t], acc);
                    }
                } else {
                    for (int k = 0; k < ts; k++) {
                        const int t = o + (ASC ? k : ts - 1 - k);
                        acc = fmaf(-D.d[t * LD + r], xe[t], acc);
                    }
                }
                xe[r] = acc;
            }
            __syncwarp();
        }
    }
}

// One sweep over a triangular factor for the nr columns of sB.  CT: the
// coefficient of row i and column t is A(t, i).  ASC: blocks ascending (rows
// below updated), else descending.  CG: columns per update task; FP32: columns
// nr .. rounded up to CG must exist in sB (their values are not used).  LW:
// coefficients a lane holds at a time (16 where registers are short).  D: room
// for one diagonal block.
// All threads call it; ends with a barrier.  sB must be visible to all threads
// (the caller's barrier) when it starts.
template <typename T, int CG, bool CT, bool ASC, bool UNIT, int LW>
__device__ __forceinline__ void tri_sweep(int n, const T *A, int lda, T *sB, int ldx, int nr, Diag<T> &D)
{
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int warp = turned_warp(blockIdx.x + gridDim.x * blockIdx.y, nw);
    const int nb = (n + 31) >> 5, ng = (nr + CG - 1) / CG;
    const bool vec = CT && ((uintptr_t)A & 15) == 0 && ((size_t)lda * sizeof(T) & 15) == 0;
    constexpr int H0 = ASC ? 0 : 32 - LW;            // the half (or all) of a block's columns used first
    {
        const int t0 = ASC ? 0 : 32 * (nb - 1);
        stage_diag<T, CT>(n, A, lda, t0, min(32, n - t0), D);
    }
    for (int s = 0; s < nb; s++) {
        const int t0 = 32 * (ASC ? s : nb - 1 - s), tb = min(32, n - t0);
        const int rbase = ASC ? t0 + 32 : 0, rend = ASC ? n : t0;
        const int ntask = rend > rbase ? ((rend - rbase + 31) >> 5) * ng : 0;
        T l[LW];
        // (FP32: warp 0, which does D, takes its tasks last)
        const int w0 = sizeof(T) == 8 ? warp : (warp == 0 ? nw : warp) - 1;
        int i = rbase + 32 * (ng == 1 ? w0 : w0 / ng) + lane;
        // the first task's coefficients are in flight during D: in the warps that do
        // not take part in it and, where there are registers for it (FP64), in all
        const bool early = (sizeof(T) == 8 && LW == 32) || (sizeof(T) == 4 && warp > 0);
        if (early && w0 < ntask) load_coefs<T, CT, LW>(l, n, A, lda, min(i, rend - 1), t0 + H0, tb - H0, vec);
        cp_async_wait<0>();
        __syncthreads();                          // the diagonal block, and the previous update
        T *x = sB + t0;
        if constexpr (sizeof(T) == 8) {
            // pairs of columns first, then one by one what is left
            int c = 0;
            if (tb == 32)
                for (; c + 1 < nr; c += 2)
                    if ((c >> 1) % nw == warp && !diag_rows_pair<CT, ASC, UNIT>(D.d, x + c * ldx, ldx)) {
                        diag_rows<CT, ASC, UNIT>(D.d, x + c * ldx, tb);
                        diag_rows<CT, ASC, UNIT>(D.d, x + (c + 1) * ldx, tb);
                    }
            for (; c < nr; c++)
                if (c % nw == warp) diag_rows<CT, ASC, UNIT>(D.d, x + c * ldx, tb);
        } else if (warp == 0) {
            diag_cols<ASC, UNIT>(D, x, ldx, nr, tb);
        }
        if (!early && w0 < ntask) load_coefs<T, CT, LW>(l, n, A, lda, min(i, rend - 1), t0 + H0, tb - H0, vec);
        __syncthreads();
        if (s + 1 < nb) {
            const int u0 = 32 * (ASC ? s + 1 : nb - 2 - s);
            stage_diag<T, CT>(n, A, lda, u0, min(32, n - u0), D);
        }
        for (int task = w0; task < ntask;) {
            const int c0 = ng == 1 ? 0 : (task % ng) * CG;
            const T *xs = sB + (size_t)c0 * ldx + t0;
            T *xr = sB + (size_t)c0 * ldx + i;
            T acc[CG];
#pragma unroll
            for (int q = 0; q < CG; q++) acc[q] = i < rend && c0 + q < nr ? xr[(size_t)q * ldx] : T(0);
#pragma unroll
            for (int h = 0; h < 32 / LW; h++) {
                const int o = ASC ? h * LW : 32 - LW - h * LW;
                if (h > 0) load_coefs<T, CT, LW>(l, n, A, lda, min(i, rend - 1), t0 + o, tb - o, vec);
                if (CG > 1 && sizeof(T) == 8 && c0 + 1 >= nr) {
                    T one[1] = {acc[0]};           // a last odd column alone
                    update_row<T, 1, ASC, LW>(one, l, xs + o, ldx, tb - o);
                    acc[0] = one[0];
                } else {
                    update_row<T, CG, ASC, LW>(acc, l, xs + o, ldx, tb - o);
                }
            }
            if (i < rend) {
#pragma unroll
                for (int q = 0; q < CG; q++)
                    if (c0 + q < nr && MLU_BC2(i, c0 + q, n, nr, 807)) xr[(size_t)q * ldx] = acc[q];
            }
            task += nw;
            if (task < ntask) {
                i = rbase + 32 * (ng == 1 ? task : task / ng) + lane;
                load_coefs<T, CT, LW>(l, n, A, lda, min(i, rend - 1), t0 + H0, tb - H0, vec);
            }
        }
    }
    __syncthreads();
}

// op(A) X = B with the LU factors in A, interchanges applied by the caller:
// L then U, or (TRANS) U^T then L^T.
template <typename T, bool TRANS, int CG, int LW = 32>
__device__ __forceinline__ void solve_smem(int n, const T *A, int lda, T *sB, int ldx, int nr, Diag<T> &D)
{
    tri_sweep<T, CG, TRANS, true, !TRANS, LW>(n, A, lda, sB, ldx, nr, D);
    tri_sweep<T, CG, TRANS, false, TRANS, LW>(n, A, lda, sB, ldx, nr, D);
}

// Columns per update task of NR right-hand sides: FP64 two (more tasks than warps matters more than
// re-reading coefficients), FP32 up to eight (the coefficients are what it loads).
template <typename T, int NR>
__host__ __device__ constexpr int solve_cg() { return sizeof(T) == 8 ? (NR < 2 ? NR : 2) : (NR < 8 ? NR : 8); }

// The row that the sequential interchanges k = 0..n-1 (targets piv[k], 1-based)
// bring to row `tau`, found by running the transpositions backwards.
__device__ __forceinline__ int resolve_row(int tau, const int *piv, int n)
{
#pragma unroll 4
    for (int k = n - 1; k >= 0; k--) {
        const int p = piv[k] - 1;
        tau = tau == k ? p : (tau == p ? k : tau);
    }
    return tau;
}

// The sequential interchanges k = 0..n-1 (targets piv[k], 1-based) applied to the nr
// columns of sB, or (UNDO) undone, 32 interchanges at a time: a warp resolves where the
// values of the 32 rows and of their targets come from by running the block's
// transpositions backwards, then gathers and scatters its columns at once.  n / 32
// blocks of about 300 instructions, so linear in n (every row resolved through all n
// interchanges is quadratic; a call with that / with this, FP32: n = 1000, 20 matrices of
// eight right-hand sides 298 / 228 us, n = 9000, one of one, 16.5 / 9.8 ms).
template <bool UNDO, typename T>
__device__ __forceinline__ void swap_rows(int n, const int *piv, T *sB, int ldx, int nr)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (warp >= nr) return;
    const int nb = (n + 31) >> 5;
    int next = lane + 32 * (UNDO ? nb - 1 : 0);
    next = next < n ? piv[next] - 1 : next;
    for (int s = 0; s < nb; s++) {
        const int k0 = 32 * (UNDO ? nb - 1 - s : s), w = min(32, n - k0);
        const int p = next;                      // (lanes past w: themselves)
        if (s + 1 < nb) {
            const int k = lane + 32 * (UNDO ? nb - 2 - s : s + 1);
            next = k < n ? piv[k] - 1 : k;
        }
        int from = k0 + lane, far = p;           // sources of row k0 + lane and of row p
#pragma unroll 8
        for (int q = 0; q < w; q++) {
            const int a = k0 + (UNDO ? q : w - 1 - q), t = __shfl_sync(FULL, p, UNDO ? q : w - 1 - q);
            from = from == a ? t : (from == t ? a : from);
            far = far == a ? t : (far == t ? a : far);
        }
        const bool top = lane < w, out = top && (unsigned)(p - k0) >= 32u;
        for (int c = warp; c < nr; c += nw) {
            T *x = sB + (size_t)c * ldx;
            T u = T(0), v = T(0);
            if (top && MLU_BC2(from, c, n, nr, 804)) u = x[from];
            if (out && MLU_BC2(far, c, n, nr, 805)) v = x[far];
            __syncwarp();
            if (top) x[k0 + lane] = u;
            if (out && MLU_BC2(p, c, n, nr, 806)) x[p] = v;   // (interchanges with one target: the same value)
            __syncwarp();
        }
    }
}

// Right-hand sides into shared memory with the interchanges piv applied, or (SCATTER)
// the transposed solve's result back with them undone.  piv: this matrix's ipiv (null:
// no interchanges).  Columns nr .. nc-1 of sB are set to zero.
template <typename T, bool SCATTER>
__device__ __forceinline__ void move_rhs(int n, const int *piv, T *B, int ldb, T *sB, int ldx, int nr, int nc)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    if (SCATTER && piv != nullptr) {
        swap_rows<true>(n, piv, sB, ldx, nr);
        __syncthreads();
    }
    for (int i = tid; i < n; i += nt) {
#pragma unroll 4
        for (int c = 0; c < (SCATTER ? nr : nc); c++) {
            if (SCATTER) B[i + (size_t)c * ldb] = sB[c * ldx + i];
            else sB[c * ldx + i] = c < nr ? B[i + (size_t)c * ldb] : T(0);
        }
    }
    if (!SCATTER && piv != nullptr) {
        __syncthreads();
        swap_rows<false>(n, piv, sB, ldx, nr);
    }
}

}  // namespace mlu
