// lu_small.cu -- warp-per-matrix LU factor / solve for n <= 32.
//
// Replaces, for one warp per matrix instead of one CTA per matrix:
//   magma_dgesv_batched_small           magmablas/zgesv_batched_small.cu:49-162,376-493
//   magma_dgetrf_batched_smallsq_noshfl magmablas/zgetrf_batched_smallsq_noshfl.cu:40-285
//   the n <= 32 part of magma_dgetrs_batched  src/zgetrs_batched.cpp:86-181
//
// Layout: lane i of the warp holds row i of the matrix (n values in
// registers) and row i of the right-hand sides.  Rows never move during the
// elimination ("lazy" interchange, as the reference kernels do); each lane
// tracks the row's position in LAPACK's current row order, which is what the
// pivot search breaks ties on and where the row is written at the end.
//
// Pivot search runs on the integer pipes: |a| as an unsigned 63-bit key,
// reduced with redux.sync on the two 32-bit halves, ties to the smallest
// current position.  NaN follows idamax's strict '>' scan: a NaN at the
// current diagonal position wins, any other NaN never does.
//
// FP64 keeps the matrix in shared memory instead (small_gesv_packed_kernel): an
// FP64 warp instruction takes 16 cycles of the SM's FP64 pipe whatever its lanes
// do, so the trailing elements of a step are spread over all 32 lanes.
#include "common.cuh"
#include "trace.cuh"

namespace mlu {

constexpr int SMALL_WARPS = 4;   // matrices per CTA (solve kernel, packed factor kernel)
constexpr int GESV_WARPS = 8;    // matrices per CTA (register factor kernel)

// FP32: lane = row in registers.
template <typename T, int N, int NRHS>
__global__ void __launch_bounds__(GESV_WARPS * 32, NRHS > 4 ? 2 : 3)
small_gesv_kernel(int n, int nrhs, T **dA_array, int ldda, int **ipiv_array, T **dB_array,
                  int lddb, int *info_array, int batch)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int mat = blockIdx.x * GESV_WARPS + warp;
    if (mat >= batch) return;

    T *A = dA_array[mat];
    const bool row_valid = lane < n;

    T a[N];
#pragma unroll
    for (int j = 0; j < N; j++)
        a[j] = (row_valid && j < n) ? A[lane + (size_t)j * ldda] : T(0);

    constexpr int NB = NRHS > 0 ? NRHS : 1;
    T b[NB];
    T *B = nullptr;
    if (NRHS > 0) {
        B = dB_array[mat];
#pragma unroll
        for (int c = 0; c < NB; c++)
            b[c] = (row_valid && c < nrhs) ? B[lane + (size_t)c * lddb] : T(0);
    }

    unsigned pos = lane;      // position in LAPACK's current row order
    bool active = row_valid;  // not yet chosen as a pivot row
    int info = 0;
    int my_ipiv = 0;
    T my_rcp = T(0);          // reciprocal of this row's pivot, once it is one

#pragma unroll
    for (int k = 0; k < N; k++) {
        if (k >= n) break;
        const T v = a[k];
        unsigned long long key = 0ull;
        if (active) {
            unsigned long long mag = Prec<T>::absbits(v);
            if (Prec<T>::isnan_(v)) mag = (pos == (unsigned)k) ? 0x7fffffffffffffffull : 0ull;
            key = mag | 0x8000000000000000ull;
        }
        const unsigned ppos = warp_argmax_key(key, active ? pos : 0xffffffffu);
        const int plane = __ffs(__ballot_sync(FULL, active && pos == ppos)) - 1;
        const T piv = shfl(v, plane);
        const bool nz = Prec<T>::nonzero(piv);
        if (!nz && info == 0) info = k + 1;
        const T r = recip(piv);
        if (lane == k) my_ipiv = (int)ppos + 1;
        const bool was_k = (pos == (unsigned)k);
        if (lane == plane) { pos = k; active = false; my_rcp = r; }
        else if (was_k) pos = ppos;

        const T l = (active && nz) ? rscale(v, piv, r) : v;
        if (active) a[k] = l;
#pragma unroll
        for (int j = k + 1; j < N; j++) {
            if (j < n) {
                const T u = shfl(a[j], plane);
                if (active) a[j] = Prec<T>::fma_(-l, u, a[j]);
            }
        }
        if (NRHS > 0) {
#pragma unroll
            for (int c = 0; c < NB; c++) {
                if (c < nrhs) {
                    const T u = shfl(b[c], plane);
                    if (active) b[c] = Prec<T>::fma_(-l, u, b[c]);
                }
            }
        }
    }

    if (NRHS > 0) {
        // U x = y, column-oriented, multiplying by the stored pivot reciprocals.
#pragma unroll
        for (int t = N - 1; t >= 0; t--) {
            if (t >= n) continue;
            const int tl = __ffs(__ballot_sync(FULL, row_valid && pos == (unsigned)t)) - 1;
            const T d = shfl(a[t], tl);
            const T rr = shfl(my_rcp, tl);
#pragma unroll
            for (int c = 0; c < NB; c++) {
                if (c < nrhs) {
                    const T x = rscale(shfl(b[c], tl), d, rr);
                    if (lane == tl) b[c] = x;
                    else if (row_valid && pos < (unsigned)t) b[c] = Prec<T>::fma_(-a[t], x, b[c]);
                }
            }
        }
    }

    if (row_valid) {
#pragma unroll
        for (int j = 0; j < N; j++)
            if (j < n) A[pos + (size_t)j * ldda] = a[j];
        ipiv_array[mat][lane] = my_ipiv;
        if (NRHS > 0) {
#pragma unroll
            for (int c = 0; c < NB; c++)
                if (c < nrhs) B[pos + (size_t)c * lddb] = b[c];
        }
    }
    if (lane == 0) info_array[mat] = info;
}

// e / d for 0 <= e < 1536 and 1 <= d <= 48: (e * small_magic(d)) >> 20.  The magic
// number is at least 2^20 / d and less than 2 above it, so that e times its excess
// stays below 2^20 / d.
__device__ __forceinline__ unsigned small_magic(int d) { return (unsigned)__fdividef(1048576.f, (float)d) + 1u; }
__device__ __forceinline__ int small_div(int e, unsigned magic) { return (int)(((unsigned)e * magic) >> 20); }

// FP64, one warp per matrix: the matrix and its right-hand sides sit row-major in
// shared memory (row stride ld odd, right-hand sides in columns n ..), rows are
// interchanged physically, and the update of step k spreads its (n-1-k) x
// (n-1-k+nrhs) elements over all lanes.  Bound by the FP64 pipe: at n = 32 and
// one right-hand side 356 update FMAs, 31 scalings and 64 solve instructions per
// matrix (365 would be the bare minimum); the pipe is busy 77 % of the time with
// the 24 warps that shared memory has room for, the rest is the chain search -
// reciprocal - scaling of each step.  No barrier: every warp computes its own
// reciprocals on the integer pipes (10,000 matrices: 420 us with one FP64 division
// shared by eight warps in lockstep, 326 us now; n = 16: 189 -> 70 us).
__host__ __device__ constexpr int small_ld(int n, int nrhs) { return (n + nrhs) | 1; }
// Elements of shared memory per matrix: the rows and the pivot reciprocals (in the
// padding column where there is one).
__host__ __device__ constexpr int small_elems(int n, int nrhs)
{
    return n * small_ld(n, nrhs) + ((n + nrhs) & 1 ? n : 0);
}

template <typename T>
__global__ void __launch_bounds__(SMALL_WARPS * 32)
small_gesv_packed_kernel(int n, int nrhs, T **dA_array, int ldda, int **ipiv_array, T **dB_array,
                         int lddb, int *info_array, int batch)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int mat = blockIdx.x * SMALL_WARPS + warp;
    if (mat >= batch) return;
    const int ld = small_ld(n, nrhs), cols = n + nrhs;
    T *sA = reinterpret_cast<T *>(smem_raw) + (size_t)warp * small_elems(n, nrhs), *sR = (cols & 1) ? sA + n * ld : sA + cols;
    const int rs = (cols & 1) ? 1 : ld;              // sR[k * rs]: the reciprocal of pivot k
    T *A = dA_array[mat];
    T *B = nrhs > 0 ? dB_array[mat] : nullptr;
    const unsigned mn = small_magic(n);
#pragma unroll 8
    for (int e = lane; e < n * n; e += 32) {
        const int j = small_div(e, mn), i = e - j * n;
        sA[i * ld + j] = A[i + (size_t)j * ldda];
    }
#pragma unroll 4
    for (int e = lane; e < n * nrhs; e += 32) {
        const int c = small_div(e, mn), i = e - c * n;
        sA[i * ld + n + c] = B[i + (size_t)c * lddb];
    }
    __syncwarp();
    int info = 0, my_ipiv = 0;
    bool plain = true;                               // no pivot needs the division
    for (int k = 0; k < n; k++) {
        const bool cand = lane >= k && lane < n;
        T *vp = sA + min(lane, n - 1) * ld + k;      // this lane's entry of column k
        const T v = *vp;
        unsigned long long key = 0ull;
        if (cand) {
            unsigned long long mag = Prec<T>::absbits(v);
            if (Prec<T>::isnan_(v)) mag = (lane == k) ? 0x7fffffffffffffffull : 0ull;
            key = mag | 0x8000000000000000ull;
        }
        const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
        const unsigned mhi = __reduce_max_sync(FULL, hi);
        unsigned win = __ballot_sync(FULL, cand && hi == mhi);
        if (win & (win - 1)) {                       // upper halves tie
            const unsigned mlo = __reduce_max_sync(FULL, hi == mhi ? lo : 0u);
            win = __ballot_sync(FULL, cand && hi == mhi && lo == mlo);
        }
        const int p = __ffs(win) - 1;                // the smallest position among equals
        const T piv = shfl(v, p);
        const bool nz = Prec<T>::nonzero(piv);
        if (!nz && info == 0) info = k + 1;
        if (p != k && MLU_BC2(p, 0, n, 1, 601)) {    // whole rows k and p
            for (int c = lane; c < cols; c += 32) {
                const T x = sA[k * ld + c];
                sA[k * ld + c] = sA[p * ld + c];
                sA[p * ld + c] = x;
            }
        }
        if (lane == k) my_ipiv = p + 1;
        plain = plain && Prec<T>::normal_or_special(piv);
        const T r = recip(piv);
        if (lane == 0) sR[k * rs] = r;
        __syncwarp();
        if (cand && lane > k && nz) *vp = rscale(*vp, piv, r);
        __syncwarp();
        const int w = n - 1 - k, wc = w + nrhs;
        if (w > 0) {
            // element e: row k+1 + e / wc, column k+1 + e % wc
            const unsigned mw = small_magic(wc);
            const T *uk = sA + k * ld + k + 1;       // the pivot row right of the pivot
            T *base = sA + (k + 1) * ld + k;         // row k+1, column k (the multipliers)
            const int total = w * wc;
            int e = lane;
            // four elements at a time, their loads ahead of their stores
            for (int e0 = 0; e0 + 128 <= total; e0 += 128, e += 128) {
                T *d[4], l[4], u[4], a[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int i = small_div(e + 32 * q, mw), j = e + 32 * q - i * wc;
                    T *row = base + i * ld;
                    l[q] = row[0];
                    u[q] = uk[j];
                    d[q] = row + 1 + j;
                    a[q] = *d[q];
                }
#pragma unroll
                for (int q = 0; q < 4; q++) *d[q] = Prec<T>::fma_(-l[q], u[q], a[q]);
            }
            // (not unrolled: guarded copies would be predicated, and an FP64
            // instruction that is predicated off takes its time in the pipe)
#pragma unroll 1
            for (; e < total; e += 32) {
                const int i = small_div(e, mw), j = e - i * wc;
                T *row = base + i * ld;
                row[1 + j] = Prec<T>::fma_(-row[0], uk[j], row[1 + j]);
            }
        }
        __syncwarp();
    }
    if (nrhs > 0) {
        // U x = y, multiplying by the pivot reciprocals
        if (nrhs == 1) {                             // lane = row, y in registers
            const T *row = sA + min(lane, n - 1) * ld;
            T y = row[n];
            if (plain) {
#pragma unroll 4
                for (int t = n - 1; t >= 0; t--) {
                    const T x = shfl(y, t) * sR[t * rs], z = Prec<T>::fma_(-row[t], x, y);
                    y = lane == t ? x : lane < t ? z : y;
                }
            } else {
#pragma unroll 1
                for (int t = n - 1; t >= 0; t--) {
                    const T x = rscale(shfl(y, t), sA[t * ld + t], sR[t * rs]), z = Prec<T>::fma_(-row[t], x, y);
                    y = lane == t ? x : lane < t ? z : y;
                }
            }
            if (lane < n) sA[lane * ld + n] = y;
        } else {
            const unsigned mr = small_magic(nrhs);
            for (int t = n - 1; t >= 0; t--) {
                const T r = sR[t * rs], d = sA[t * ld + t];
                T *xt = sA + t * ld + n;
                if (lane < nrhs) xt[lane] = plain ? xt[lane] * r : rscale(xt[lane], d, r);
                __syncwarp();
#pragma unroll 1
                for (int e = lane; e < t * nrhs; e += 32) {
                    const int i = small_div(e, mr), c = e - i * nrhs;
                    T *y = sA + i * ld + n + c;
                    *y = Prec<T>::fma_(-sA[i * ld + t], xt[c], *y);
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
#pragma unroll 8
    for (int e = lane; e < n * n; e += 32) {
        const int j = small_div(e, mn), i = e - j * n;
        A[i + (size_t)j * ldda] = sA[i * ld + j];
    }
#pragma unroll 4
    for (int e = lane; e < n * nrhs; e += 32) {
        const int c = small_div(e, mn), i = e - c * n;
        B[i + (size_t)c * lddb] = sA[i * ld + n + c];
    }
    if (lane < n) ipiv_array[mat][lane] = my_ipiv;
    if (lane == 0) info_array[mat] = info;
}

// Solve with existing factors, n <= 32.  NoTrans: lane i holds row i of LU.
// Trans: lane i holds column i of LU, so that U(t,i) and L(t,i) are static
// register indices.  RHS columns [blockIdx.y*NRHS, +NRHS).
template <typename T, int N, int NRHS, bool TRANS>
__global__ void __launch_bounds__(SMALL_WARPS * 32)
small_getrs_kernel(int n, int nrhs, T **dA_array, int ldda, int **ipiv_array, T **dB_array,
                   int lddb, int batch)
{
    const int lane = threadIdx.x & 31;
    const int mat = blockIdx.x * SMALL_WARPS + (threadIdx.x >> 5);
    if (mat >= batch) return;
    const int c0 = blockIdx.y * NRHS;
    const T *A = dA_array[mat];
    const int *ipiv = ipiv_array[mat];
    T *B = dB_array[mat] + (size_t)c0 * lddb;
    const int nr = min(NRHS, nrhs - c0);
    const bool valid = lane < n;

    T a[N];
#pragma unroll
    for (int j = 0; j < N; j++) {
        if (TRANS) a[j] = (valid && j < n) ? A[j + (size_t)lane * ldda] : T(0);
        else       a[j] = (valid && j < n) ? A[lane + (size_t)j * ldda] : T(0);
    }
    T b[NRHS];
#pragma unroll
    for (int c = 0; c < NRHS; c++) b[c] = (valid && c < nr) ? B[lane + (size_t)c * lddb] : T(0);
    const int my_piv = valid ? ipiv[lane] - 1 : lane;

    if (!TRANS) {
        // B <- P B, sequential interchanges k = 0..n-1
#pragma unroll
        for (int k = 0; k < N; k++) {
            if (k >= n) break;
            const int p = shfl(my_piv, k);
            if (p != k) {
#pragma unroll
                for (int c = 0; c < NRHS; c++) {
                    const T vk = shfl(b[c], k), vp = shfl(b[c], p);
                    if (lane == k) b[c] = vp;
                    if (lane == p) b[c] = vk;
                }
            }
        }
        // L y = b (unit lower)
#pragma unroll
        for (int t = 0; t < N; t++) {
            if (t >= n) break;
#pragma unroll
            for (int c = 0; c < NRHS; c++) {
                const T y = shfl(b[c], t);
                if (lane > t) b[c] = Prec<T>::fma_(-a[t], y, b[c]);
            }
        }
        // U x = y
#pragma unroll
        for (int t = N - 1; t >= 0; t--) {
            if (t >= n) continue;
            const T d = shfl(a[t], t);
            const T r = T(1) / d;
#pragma unroll
            for (int c = 0; c < NRHS; c++) {
                const T x = rscale(shfl(b[c], t), d, r);
                if (lane == t) b[c] = x;
                else if (lane < t) b[c] = Prec<T>::fma_(-a[t], x, b[c]);
            }
        }
    } else {
        // U^T y = b: lane i holds column i, so a[t] = U(t,i) for t <= i.
#pragma unroll
        for (int t = 0; t < N; t++) {
            if (t >= n) break;
            const T d = shfl(a[t], t);
            const T r = T(1) / d;
#pragma unroll
            for (int c = 0; c < NRHS; c++) {
                const T x = rscale(shfl(b[c], t), d, r);
                if (lane == t) b[c] = x;
                else if (lane > t) b[c] = Prec<T>::fma_(-a[t], x, b[c]);
            }
        }
        // L^T x = y: a[t] = L(t,i) for t > i.
#pragma unroll
        for (int t = N - 1; t >= 0; t--) {
            if (t >= n) continue;
#pragma unroll
            for (int c = 0; c < NRHS; c++) {
                const T x = shfl(b[c], t);
                if (lane < t) b[c] = Prec<T>::fma_(-a[t], x, b[c]);
            }
        }
        // B <- P^T B, interchanges in reverse order
#pragma unroll
        for (int k = N - 1; k >= 0; k--) {
            if (k >= n) continue;
            const int p = shfl(my_piv, k);
            if (p != k) {
#pragma unroll
                for (int c = 0; c < NRHS; c++) {
                    const T vk = shfl(b[c], k), vp = shfl(b[c], p);
                    if (lane == k) b[c] = vp;
                    if (lane == p) b[c] = vk;
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < NRHS; c++)
        if (valid && c < nr) B[lane + (size_t)c * lddb] = b[c];
}

template <typename T, int N, int NRHS>
static void launch_small_gesv(int n, int nrhs, T **dA, int ldda, int **ipiv, T **dB, int lddb,
                              int *info, int batch, cudaStream_t s)
{
    MLU_LAUNCH(mlu::KC_SMALL_GESV, s, small_gesv_kernel<T, N, NRHS><<<mlu_ceildiv(batch, GESV_WARPS), GESV_WARPS * 32, 0, s>>>(
        n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch));
}

template <typename T, int N>
static void dispatch_nrhs(int n, int nrhs, T **dA, int ldda, int **ipiv, T **dB, int lddb,
                          int *info, int batch, cudaStream_t s)
{
    if (nrhs == 0)      launch_small_gesv<T, N, 0>(n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch, s);
    else if (nrhs == 1) launch_small_gesv<T, N, 1>(n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch, s);
    else if (nrhs <= 4) launch_small_gesv<T, N, 4>(n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch, s);
    else                launch_small_gesv<T, N, 16>(n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch, s);
}

// Fused factor (+ solve when nrhs > 0) for n <= 32, nrhs <= 16.
template <typename T>
magma_int_t small_gesv(int n, int nrhs, T **dA, int ldda, int **ipiv, T **dB, int lddb, int *info,
                       int batch, magma_queue_t q)
{
    if (n > 32 || n < 1 || nrhs > 16) return MAGMA_ERR;   // -100: not applicable
    if (batch <= 0) return MAGMA_SUCCESS;
    cudaStream_t s = q->stream;
    if constexpr (sizeof(T) == 8) {
        const size_t smem = (size_t)SMALL_WARPS * small_elems(n, nrhs) * sizeof(T);   // at most 52 KB
        static size_t dyn_cache[MLU_MAX_DEVICES];
        mlu_device_cached(dyn_cache, [] { return mlu_allow_dynamic_smem(small_gesv_packed_kernel<T>); });
        MLU_LAUNCH(mlu::KC_SMALL_GESV, s, small_gesv_packed_kernel<T><<<mlu_ceildiv(batch, SMALL_WARPS), SMALL_WARPS * 32, smem, s>>>(
            n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch));
    } else {
        if (n <= 8)       dispatch_nrhs<T, 8>(n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch, s);
        else if (n <= 16) dispatch_nrhs<T, 16>(n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch, s);
        else              dispatch_nrhs<T, 32>(n, nrhs, dA, ldda, ipiv, dB, lddb, info, batch, s);
    }
    MLU_CHECK_LAUNCH();
    return MAGMA_SUCCESS;
}

template <typename T, int N, bool TRANS>
static void launch_small_getrs(int n, int nrhs, T **dA, int ldda, int **ipiv, T **dB, int lddb,
                               int batch, cudaStream_t s)
{
    constexpr int NR = 4;
    dim3 grid(mlu_ceildiv(batch, SMALL_WARPS), mlu_ceildiv(nrhs, NR));
    MLU_LAUNCH(mlu::KC_GETRS, s, small_getrs_kernel<T, N, NR, TRANS><<<grid, SMALL_WARPS * 32, 0, s>>>(
        n, nrhs, dA, ldda, ipiv, dB, lddb, batch));
}

template <typename T>
magma_int_t small_getrs(bool trans, int n, int nrhs, T **dA, int ldda, int **ipiv, T **dB,
                        int lddb, int batch, magma_queue_t q)
{
    if (n > 32) return MAGMA_ERR;
    if (batch <= 0 || n == 0 || nrhs == 0) return MAGMA_SUCCESS;
    cudaStream_t s = q->stream;
    if (trans) {
        if (n <= 8)       launch_small_getrs<T, 8, true>(n, nrhs, dA, ldda, ipiv, dB, lddb, batch, s);
        else if (n <= 16) launch_small_getrs<T, 16, true>(n, nrhs, dA, ldda, ipiv, dB, lddb, batch, s);
        else              launch_small_getrs<T, 32, true>(n, nrhs, dA, ldda, ipiv, dB, lddb, batch, s);
    } else {
        if (n <= 8)       launch_small_getrs<T, 8, false>(n, nrhs, dA, ldda, ipiv, dB, lddb, batch, s);
        else if (n <= 16) launch_small_getrs<T, 16, false>(n, nrhs, dA, ldda, ipiv, dB, lddb, batch, s);
        else              launch_small_getrs<T, 32, false>(n, nrhs, dA, ldda, ipiv, dB, lddb, batch, s);
    }
    MLU_CHECK_LAUNCH();
    return MAGMA_SUCCESS;
}

template magma_int_t small_gesv<double>(int, int, double **, int, int **, double **, int, int *, int, magma_queue_t);
template magma_int_t small_gesv<float>(int, int, float **, int, int **, float **, int, int *, int, magma_queue_t);
template magma_int_t small_getrs<double>(bool, int, int, double **, int, int **, double **, int, int, magma_queue_t);
template magma_int_t small_getrs<float>(bool, int, int, float **, int, int **, float **, int, int, magma_queue_t);

}  // namespace mlu
