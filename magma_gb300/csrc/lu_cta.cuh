// lu_cta.cuh -- the whole LU factorisation of one matrix of at most 256 rows
// and columns by one CTA, shared by the variable-size kernel (lu_vbatched.cu)
// and the fixed-size path (lu_blocked.cu).
//
// Restates the same steps as lu_core.cuh (panel, interchanges, U12, trailing
// update) with the same floating-point operations in the same order, arranged
// for what bounds FP64 work on this part: a warp FMA holds the SM's FP64 pipe
// for 16 cycles (one scheduler's share for 64) however many of its lanes work,
// so every phase is laid out to fill its lanes and to keep warps of all four
// schedulers busy, and the serial parts of one matrix run beside the updates
// of the other CTAs of the SM (three of 256 threads, seven of 128, fourteen of 64):
//   panel   CTA_NB columns in registers, a row per thread, rows in place; one
//           barrier per column; the reciprocal on the integer pipes (recip);
//   columns one thread per column outside the panel and per right-hand side:
//           the panel's interchanges (the row map after the panel gives them:
//           a top row comes from row slot[q], the row a pivot left receives an
//           original top row, nothing else moves) and, right of the panel, U12
//           in registers -- no barrier;
//   update  A22 -= L21 U12 by 4 x 4 (2 x 2) elements per thread, L21 and U12
//           from shared memory, the blocks dealt out to lanes in one sequence,
//           so that no lane is idle but in the last group of 32.
// Panels are 16 columns wide: A22 goes through registers once per 16 steps,
// which the caches serve beside the FP64 pipe, and the panel and U12 (63 KB
// together at order 256, 16 at order 64) leave room for those CTAs.
#pragma once
#include "common.cuh"

namespace mlu {

constexpr int CTA_NB = 16;
constexpr int CTA_MAX_N = 256;

// Row strides in shared memory, multiples of four elements (a 4 x 4 block reads up
// to there): of the panel, and of U12 after a first panel of nb columns or more, whose
// place also holds the panel's U rows while it is factored.  No more than that:
// the CTAs per SM depend on it.
__host__ __device__ constexpr int cta_ldp(int m) { return (m + 3) & ~3; }
__host__ __device__ constexpr int cta_ldu(int n, int nb) { return n - nb > CTA_NB ? (n - nb + 3) & ~3 : CTA_NB; }
template <typename T>
__host__ __device__ constexpr size_t cta_lu_smem(int max_m, int max_n, int nb)
{
    return (size_t)CTA_NB * (cta_ldp(max_m) + cta_ldu(max_n, nb)) * sizeof(T);
}

// Shared state of one panel.  Each 32-row block (one warp) publishes its best
// candidate of the current column, double-buffered: |v| as a 63-bit key (NaN by
// idamax's rule), its position (ties go to the smaller) and what remains of its
// row, the current column first.  NCH: 32-row blocks, at most.
template <typename T, int NCH> struct CtaPanel {
    T rest[2][NCH][CTA_NB];
    T rcp[2][NCH];           // reciprocal of rest[..][0] (not valid where recip_special)
    unsigned hi[2][NCH], lo[2][NCH], pos[2][NCH];
    int ipiv[CTA_NB];        // position chosen at each column
    int slot[CTA_NB];        // top row q comes from this row
    int dst[CTA_NB];         // original top row i goes to this row (-1: it stays in the top block)
};

// One step's update of a panel row and the search of the next column.  a[j - 1] =
// fma(-l, u_j, a[j]) for 1 <= j < REM (u_j at rest[j]): shifted, so that the current
// column stays a[0]; then the warp's best candidate of that column, published with
// its reciprocal for step k + 1.  Straight-line: the search and the reciprocal are
// integer instructions on the new a[0] alone, which is computed first, and issue
// between the other FMAs, 64 cycles apart on the FP64 pipe.  REM <= 1: no update
// (before the first step).  Rows already chosen as pivots go through the motions.
template <int REM, typename T, int NCH>
__device__ __forceinline__ void cta_step(T (&a)[CTA_NB], T l, const T *rest, CtaPanel<T, NCH> &s, int buf, int chunk,
                                         bool live, int pos, int k)
{
    if (REM > 1) a[0] = Prec<T>::fma_(-l, rest[1], a[1]);
    unsigned long long mag = Prec<T>::absbits(a[0]);
    if (Prec<T>::isnan_(a[0])) mag = pos == k ? 0x7fffffffffffffffull : 0ull;
    const unsigned long long key = live ? mag | 0x8000000000000000ull : 0ull;
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mhi = __reduce_max_sync(FULL, hi);
    const unsigned mlo = __reduce_max_sync(FULL, hi == mhi ? lo : 0u);
    const unsigned mp = __reduce_min_sync(FULL, live && hi == mhi && lo == mlo ? (unsigned)pos : 0xffffffffu);
    const bool win = live && (unsigned)pos == mp;
    const T r = recip_plain(a[0]);                       // (the winner's is used)
#pragma unroll
    for (int j = 2; j < REM; j++) a[j - 1] = Prec<T>::fma_(-l, rest[j], a[j]);
    if (win) {
        s.hi[buf][chunk] = mhi;
        s.lo[buf][chunk] = mlo;
        s.pos[buf][chunk] = mp;
        s.rcp[buf][chunk] = r;
#pragma unroll
        for (int j = 0; j < (REM > 1 ? REM - 1 : CTA_NB); j++) s.rest[buf][chunk][j] = a[j];
    }
    if (mhi == 0u && (threadIdx.x & 31) == 0) s.hi[buf][chunk] = 0u;   // no row left in this block
}

// ... with rem columns remaining at the step: a jump to the code for that many,
// rounded up to even.  Guards (j < rem) would be turned into predicates, and an
// FP64 instruction that is predicated off takes its full 16 cycles of the pipe
// (panel of 64 rows, twelve CTAs per SM: 153,000 cycles with guards).
template <typename T, int NCH>
__device__ __forceinline__ void cta_step(T (&a)[CTA_NB], T l, const T *rest, CtaPanel<T, NCH> &s, int buf, int chunk,
                                         bool live, int pos, int k, int rem)
{
    static_assert(CTA_NB == 16, "cases");
    switch ((rem + 1) >> 1) {
    case 1: cta_step<2>(a, l, rest, s, buf, chunk, live, pos, k); break;
    case 2: cta_step<4>(a, l, rest, s, buf, chunk, live, pos, k); break;
    case 3: cta_step<6>(a, l, rest, s, buf, chunk, live, pos, k); break;
    case 4: cta_step<8>(a, l, rest, s, buf, chunk, live, pos, k); break;
    case 5: cta_step<10>(a, l, rest, s, buf, chunk, live, pos, k); break;
    case 6: cta_step<12>(a, l, rest, s, buf, chunk, live, pos, k); break;
    case 7: cta_step<14>(a, l, rest, s, buf, chunk, live, pos, k); break;
    default: cta_step<16>(a, l, rest, s, buf, chunk, live, pos, k); break;
    }
}

// Panel of pm rows (pm <= blockDim.x <= 256) and ib <= CTA_NB columns at Ap, row
// `i` (a permutation of the thread index by whole warps) per thread.  On return
// sP[j * ldp + i] and Ap hold it in pivoted order, s.ipiv / slot / dst are set
// (visible to all threads) and the return value is the 1-based column of the
// first zero pivot, or 0, in every thread with a row.  top: room for the panel's U rows.
//
// A row's remaining columns sit in its thread's registers with the current one
// first, so that the column loop stays a loop.  A column that is done leaves for
// sP, in physical row order until the end.
template <typename T, int NCH>
__device__ __forceinline__ int cta_panel(int pm, int ib, T *Ap, int lda, T *sP, int ldp, T *top, CtaPanel<T, NCH> &s, int i)
{
    const int lane = i & 31, chunk = i >> 5;
    const int nch = (pm + 31) >> 5;                      // 32-row blocks
    const bool row = i < pm;
    bool live = row;
    int pos = i, info = 0;
    T a[CTA_NB];
#pragma unroll
    for (int j = 0; j < CTA_NB; j++) a[j] = row && j < ib ? Ap[i + (size_t)j * lda] : T(0);
    if (chunk < nch) cta_step<1>(a, T(0), (const T *)nullptr, s, 0, chunk, live, pos, 0);
#pragma unroll 1
    for (int k = 0; k < ib; k++) {
        const int buf = k & 1;
        if (nch > 1) __syncthreads();
        else __syncwarp();
        if (chunk >= nch) continue;
        int gw = 0;
        if (nch > 1) {
            const unsigned h = lane < nch ? s.hi[buf][lane] : 0u;
            const unsigned mh = __reduce_max_sync(FULL, h);
            unsigned eq = __ballot_sync(FULL, lane < nch && h == mh);
            if (eq & (eq - 1)) {                         // the upper halves tie: the lower, then the positions
                const bool c = (eq >> lane) & 1;
                const unsigned l = c ? s.lo[buf][lane] : 0u;
                const unsigned ml = __reduce_max_sync(FULL, l);
                const unsigned p = c && l == ml ? s.pos[buf][lane] : 0xffffffffu;
                const unsigned mp = __reduce_min_sync(FULL, p);
                eq = __ballot_sync(FULL, c && p == mp);
            }
            gw = __ffs(eq) - 1;
        }
        const T *rest = s.rest[buf][gw];
        const unsigned gpos = s.pos[buf][gw];
        const T piv = rest[0];
        T r = s.rcp[buf][gw];
        const bool nz = Prec<T>::nonzero(piv);
        if (!nz && info == 0) info = k + 1;
        if (i == 0) s.ipiv[k] = (int)gpos;
        if (chunk == 0 && lane < ib - k) top[k * CTA_NB + k + lane] = rest[lane];
        if (pos == (int)gpos) {
            live = false;                                // the pivot row is U row k
            pos = k;
        } else if (pos == k) {
            pos = (int)gpos;
        }
        T l = a[0] * r;
        if (recip_special(piv)) l = nz ? rscale(a[0], piv, recip(piv)) : a[0];
        if (row) sP[k * ldp + i] = l;                    // (rows already chosen: never read)
        if (k + 1 < ib) cta_step(a, l, rest, s, buf ^ 1, chunk, live, pos, k + 1, ib - k);
    }
    // pivoted order: every row to its position, in shared memory and in A.  A row's
    // L entries are its own stores (no barrier needed to read them back); a top row
    // goes on with its U entries.
    const int nl = pos < ib ? pos : ib;
    if (row && MLU_BC2(pos, 0, pm, 1, 701)) {
#pragma unroll
        for (int j = 0; j < CTA_NB; j++)
            if (j < nl) a[j] = sP[j * ldp + i];
        if (pos < ib) s.slot[pos] = i;
        if (i < ib) s.dst[i] = pos >= ib ? pos : -1;
    }
    __syncthreads();
    if (row && MLU_BC2(pos, 0, pm, 1, 704)) {
#pragma unroll
        for (int j = 0; j < CTA_NB; j++)
            if (j < ib) {
                const T v = j < nl ? a[j] : top[pos * CTA_NB + j];
                sP[j * ldp + pos] = v;
                Ap[pos + (size_t)j * lda] = v;
            }
    }
    __syncthreads();
    return info;
}

// M consecutive values from shared memory, 16 bytes at a time where they fill
// them (p aligned to M elements, at most 16 bytes).
template <int M>
__device__ __forceinline__ void cta_lds(double (&v)[M], const double *p)
{
#pragma unroll
    for (int a = 0; a < M; a += 2) {
        const double2 x = *reinterpret_cast<const double2 *>(p + a);
        v[a] = x.x;
        v[a + 1] = x.y;
    }
}
__device__ __forceinline__ void cta_lds(float (&v)[4], const float *p)
{
    const float4 x = *reinterpret_cast<const float4 *>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
__device__ __forceinline__ void cta_lds(float (&v)[2], const float *p)
{
    const float2 x = *reinterpret_cast<const float2 *>(p);
    v[0] = x.x, v[1] = x.y;
}

// The panel's interchanges on column `col` (pointer to its row j0, pm rows), and with
// SOLVE U12 = L11^{-1} A12 for it, also stored to sU (stride ldu).  FULL: ib is CTA_NB.
template <bool SOLVE, bool FULL, typename T, int NCH>
__device__ __forceinline__ void cta_column(T *col, int pm, int ib, const T *sP, int ldp, const CtaPanel<T, NCH> &s, T *sU, int ldu)
{
    T v[CTA_NB];
    const volatile int *slot = s.slot, *dst = s.dst;     // re-read: registers are short here
#pragma unroll
    for (int q = 0; q < CTA_NB; q++)
        if (FULL || q < ib) v[q] = MLU_BC2(slot[q], 0, pm, 1, 702) ? col[slot[q]] : T(0);
#pragma unroll
    for (int q0 = 0; q0 < CTA_NB; q0 += 4) {             // the rows the pivots left
        T w[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            if ((FULL || q0 + q < ib) && dst[q0 + q] >= 0) w[q] = col[q0 + q];
#pragma unroll
        for (int q = 0; q < 4; q++)
            if ((FULL || q0 + q < ib) && dst[q0 + q] >= 0 && MLU_BC2(dst[q0 + q], 0, pm, 1, 703)) col[dst[q0 + q]] = w[q];
    }
    if (SOLVE) {
#pragma unroll
        for (int t = 0; t < CTA_NB; t++)
            if (FULL || t < ib) {
                const T *l = sP + t * ldp;
#pragma unroll
                for (int q0 = (t + 1) & ~1; q0 < CTA_NB; q0 += 2) {
                    T lq[2];
                    cta_lds(lq, l + q0);
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int q = q0 + u;
                        if (q > t && (FULL || q < ib)) v[q] = Prec<T>::fma_(-lq[u], v[t], v[q]);
                    }
                }
            }
    }
#pragma unroll
    for (int q = 0; q < CTA_NB; q++)
        if (FULL || q < ib) {
            col[q] = v[q];
            if (SOLVE && MLU_BC2(q, 0, CTA_NB, ldu, 708)) sU[q * ldu] = v[q];
        }
}

// A22 -= L21 U12 for the rm x rn block at A22: M x M elements per thread, L21 at
// sL (column k at sL + k * ldp), U12 at sU.  ib is a multiple of eight.
template <typename T, int M>
__device__ __forceinline__ void cta_update(T *A22, int lda, int rm, int rn, int ib, const T *sL, int ldp, const T *sU,
                                           int ldu, int vtid)
{
    const int nr = (rm + M - 1) / M, items = nr * ((rn + M - 1) / M);
    for (int it = vtid; it < items; it += blockDim.x) {
        const int c = it / nr * M, r = (it - it / nr * nr) * M;
        T *p = A22 + r + (size_t)c * lda;
        T acc[M][M];                                     // [column][row]
#pragma unroll
        for (int b = 0; b < M; b++)
#pragma unroll
            for (int a = 0; a < M; a++)
                acc[b][a] = (r + a < rm && c + b < rn && MLU_BC2(r + a, c + b, rm, rn, 705)) ? p[a + (size_t)b * lda] : T(0);
        // (a block reads L21 and U12 up to its fourth row and column)
        if (!MLU_BC2(r + M - 1, c + M - 1, ldp - ib, ldu, 706)) continue;
        for (int k0 = 0; k0 < ib; k0 += 8) {
#pragma unroll 2
            for (int k = 0; k < 8; k++) {
                T l[M], u[M];
                cta_lds(l, sL + (k0 + k) * ldp + r);
                cta_lds(u, sU + (k0 + k) * ldu + c);
#pragma unroll
                for (int b = 0; b < M; b++)
#pragma unroll
                    for (int a = 0; a < M; a++) acc[b][a] = Prec<T>::fma_(-l[a], u[b], acc[b][a]);
            }
        }
#pragma unroll
        for (int b = 0; b < M; b++)
#pragma unroll
            for (int a = 0; a < M; a++)
                if (r + a < rm && c + b < rn && MLU_BC2(r + a, c + b, rm, rn, 707)) p[a + (size_t)b * lda] = acc[b][a];
    }
}

// A turn for matrix k: hashed, because the CTAs that share an SM start with
// indices a multiple of the number of SMs (8 * 19) apart.
__device__ __forceinline__ int cta_rot(int k) { return (int)((unsigned)k * 0x9E3779B1u >> 29); }

// The factorisation of the m x n matrix at A (m, n <= blockDim.x), and the
// interchanges applied to its nrhs right-hand sides.  smem: cta_lu_smem bytes for
// the row strides ldp >= cta_ldp(m), ldu >= cta_ldu(n, nb).  nb: panel width, 8 or 16;
// small: 2 x 2 elements per thread in every update.  `rot` turns the assignment of rows and columns to warps, so that the short panels and steps
// of different matrices do not all load the same scheduler (cta_rot).  Sets *info_out to the
// first zero pivot (1-based) or 0; ends with a barrier.
template <typename T, int NCH>
__device__ __forceinline__ void cta_lu(int m, int n, T *A, int lda, int *ipiv, int nrhs, T *B, int ldb,
                                      unsigned char *smem, int ldp, int ldu, CtaPanel<T, NCH> &s, int nb, bool small, int rot, int *info_out)
{
    T *sP = reinterpret_cast<T *>(smem), *sU = sP + CTA_NB * ldp;
    const int tid = threadIdx.x, nt = blockDim.x, mn = min(m, n);
    for (int j0 = 0, step = rot; j0 < mn; j0 += nb, step++) {
        const int ib = min(nb, mn - j0);
        T *Ap = A + j0 + (size_t)j0 * lda;
        const int vtid = (tid + 32 * (step & 7)) & (nt - 1);   // nt is a power of two
        const int il = cta_panel<T>(m - j0, ib, Ap, lda, sP, ldp, sU, s, vtid);
        // every thread with a row knows il: the one with row 0 keeps the first
        if (vtid == 0) {
            if (step == rot) *info_out = il;             // (the panel's barriers order these writes)
            else if (il != 0 && *info_out == 0) *info_out = j0 + il;
        }
        if (tid < ib) ipiv[j0 + tid] = j0 + s.ipiv[tid] + 1;
        const int rm = m - j0 - ib, rn = n - j0 - ib;
        // columns right of the panel, then the right-hand sides and those left of it
        for (int c = vtid; c < rn + nrhs + j0; c += nt) {
            if (c < rn) {
                T *col = Ap + (size_t)(ib + c) * lda;
                if (ib == CTA_NB) cta_column<true, true>(col, m - j0, ib, sP, ldp, s, sU + c, ldu);
                else cta_column<true, false>(col, m - j0, ib, sP, ldp, s, sU + c, ldu);
            } else {
                T *col = c < rn + nrhs ? B + j0 + (size_t)(c - rn) * ldb : A + j0 + (size_t)(c - rn - nrhs) * lda;
                cta_column<false, false>(col, m - j0, ib, sP, ldp, s, (T *)nullptr, 0);
            }
        }
        __syncthreads();
        if (rm > 0 && rn > 0) {
            T *A22 = Ap + ib + (size_t)ib * lda;
            // 4 x 4 elements per thread, or 2 x 2 where its rounds waste less
            const int n4 = ((rm + 3) >> 2) * ((rn + 3) >> 2), n2 = ((rm + 1) >> 1) * ((rn + 1) >> 1);
            if (small || 4 * ((n2 + nt - 1) / nt) < 16 * ((n4 + nt - 1) / nt))
                cta_update<T, 2>(A22, lda, rm, rn, ib, sP + ib, ldp, sU, ldu, vtid);
            else
                cta_update<T, 4>(A22, lda, rm, rn, ib, sP + ib, ldp, sU, ldu, vtid);
        }
        __syncthreads();
    }
    if (mn <= 0 && tid == 0) *info_out = 0;
}

}  // namespace mlu
