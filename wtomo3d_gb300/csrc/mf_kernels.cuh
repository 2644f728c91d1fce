// Multifrontal numeric kernels (templated on the real type T: float for the
// complex64 mixed-precision path, double for the complex128 oracle path).
//
// Front layout (row-major): the pivot rows P = F[0:p, 0:nf] (p x nf) are
// followed by the lower-left border block Lo = F[p:nf, 0:p] (b x p) in the
// factor pool; the Schur/update block F22 (b x b) lives in one of two
// level-parity update buffers.  Factorisation is right-looking blocked LU on
// the first p columns with KB-wide panels and partial pivoting restricted to
// the diagonal KB x KB tile; row interchanges are LINPACK style (applied to
// the columns right of the panel only), so the forward solve applies them
// block by block.
#pragma once
#include "common.cuh"

namespace wt3d {

constexpr int KB = 64;        // panel width
constexpr int MAXRHS = 32;    // right-hand sides per solve pass (a multiple of 32)

struct FrontDev {
    long long fac;     // P block offset in the factor pool (complex elements)
    long long upd;     // F22 offset in its parity buffer
    long long border;  // offset into the border index array
    int p, b, first, parity;
    long long inv;     // offset of the front's first block inverse in the inverse pool
};

struct PanelTask { int f, k; };
struct RowTask { int f, k, c0; };
struct ColTask { int f, k, r0, which; };
struct EATask { int child, parent; long long row0; };
template <class T>
struct GemmTask {
    const cx<T> *A;
    const cx<T> *B;
    cx<T> *C;
    const int *brow;   // optional row gather for B
    const int *crow;   // optional row scatter for C (atomic)
    int lda, ldb, ldc, M, N, K;
    int tiles_n;
    long long tile0;
    int conjA;         // use conj(A^T): A is read as its conjugate transpose
    int atom;          // C -= A B with atomics (a K-chunk of a split task)
};

template <class T>
__device__ __forceinline__ void atomic_sub(cx<T> *p, cx<T> v)
{
    atomicAdd(&p->re, -v.re);
    atomicAdd(&p->im, -v.im);
}

template <class Task>
__device__ __forceinline__ int find_task(const Task *tasks, int ntasks, long long key)
{
    int lo = 0, hi = ntasks - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].tile0 <= key) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// original entries -> fronts
// ---------------------------------------------------------------------------
// One thread per CSR row: a_ij * s_i * s_j into the front that owns the entry.
// s is the symmetric Jacobi scaling 1/sqrt|a_ii| (natural ordering): Dirichlet
// rows carry unit diagonals next to O(1e8) stiffness rows, and equilibrating
// both sides keeps the complex64 fronts well scaled.
template <class T>
__global__ void k_scatter(long long n, const int *__restrict__ irptr, const int *__restrict__ jcptr,
                          const long long *__restrict__ map, const double2 *__restrict__ a,
                          const double *__restrict__ s, cx<T> *__restrict__ fac)
{
    long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const double sr = s[r];
    for (int k = irptr[r]; k < irptr[r + 1]; k++) {
        double2 v = a[k];
        double w = sr * s[jcptr[k]];
        fac[map[k]] = cx<T>((T)(v.x * w), (T)(v.y * w));
    }
}

static __global__ void k_jacobi_scale(long long n, const int *__restrict__ irptr, const int *__restrict__ jcptr,
                               const double2 *__restrict__ a, double *__restrict__ s)
{
    long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    double d = 0;
    for (int k = irptr[r]; k < irptr[r + 1]; k++)
        if (jcptr[k] == r) d = sqrt(a[k].x * a[k].x + a[k].y * a[k].y);
    s[r] = (d > 0 && d < INFINITY) ? 1.0 / sqrt(d) : 1.0;
}

static __global__ void k_maxabs(long long n, const double2 *__restrict__ a, unsigned long long *out)
{
    double m = 0;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        double2 v = a[k];
        m = fmax(m, v.x * v.x + v.y * v.y);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// ---------------------------------------------------------------------------
// extend-add: child update matrix into the parent front (one warp per row)
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_extend_add(const EATask *__restrict__ tasks, int ntasks, long long nrows,
                             const FrontDev *__restrict__ fr, const int *__restrict__ rel, cx<T> *__restrict__ fac,
                             cx<T> *__restrict__ upd0, cx<T> *__restrict__ upd1)
{
    long long gr = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (gr >= nrows) return;
    int lo = 0, hi = ntasks - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].row0 <= gr) lo = mid;
        else hi = mid - 1;
    }
    const EATask t = tasks[lo];
    const FrontDev C = fr[t.child], P = fr[t.parent];
    const int i = (int)(gr - t.row0);
    const int *rl = rel + C.border;   // rel shares the border indexing
    const cx<T> *src = (C.parity ? upd1 : upd0) + C.upd + (long long)i * C.b;
    const int R = rl[i];
    const int nfP = P.p + P.b;
    cx<T> *pf = fac + P.fac;
    cx<T> *p22 = (P.parity ? upd1 : upd0) + P.upd;
    for (int j = lane; j < C.b; j += 32) {
        const int Cc = rl[j];
        cx<T> v = src[j];
        cx<T> *dst;
        if (R < P.p) dst = pf + (long long)R * nfP + Cc;
        else if (Cc < P.p) dst = pf + (long long)P.p * nfP + (long long)(R - P.p) * P.p + Cc;
        else dst = p22 + (long long)(R - P.p) * P.b + (Cc - P.p);
        *dst = *dst + v;
    }
}

// Row order of panel k after its LINPACK-style interchanges: idx[i] is the
// stored row that lands at position i, from gord, which holds for every pivot
// position of the new ordering the row that lands there (written by the panel
// kernel).  Threads tid < KB write idx; callers synchronise before reading it.
__device__ __forceinline__ void panel_rows(const int *__restrict__ gord, int first, int kb, int *idx)
{
    const int tid = threadIdx.x;
    if (tid < KB) idx[tid] = tid < kb ? gord[first + tid] - first : tid;
}

// ---------------------------------------------------------------------------
// panel: LU of the KB x KB diagonal tile with partial pivoting inside the tile
// ---------------------------------------------------------------------------
// The stored row at each position after the tile's interchanges goes to the
// positions of gord (the row band and the substitution passes read it).
template <class T>
__global__ void __launch_bounds__(256) k_panel(const PanelTask *__restrict__ tasks, const FrontDev *__restrict__ fr,
                                               cx<T> *__restrict__ fac, int *__restrict__ ipiv,
                                               const unsigned long long *__restrict__ amax2, double pivot_rel,
                                               int *__restrict__ npert, int *__restrict__ gord)
{
    // static-pivot threshold: pivot_rel * max |a_ij| of the assembled operator
    const T thresh = (T)(pivot_rel * sqrt(__longlong_as_double((long long)*amax2)));
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *S = reinterpret_cast<cx<T> *>(smraw);   // KB x (KB+1), then 2 KB scratch columns
    __shared__ int prow[KB];   // stored row at each position, as the interchanges go
    const PanelTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    const int LD = KB + 1;
    cx<T> *D = fac + F.fac + (long long)k * nf + k;
    const int tid = threadIdx.x;
    #pragma unroll 8   // several loads in flight per thread
    for (int idx = tid; idx < kb * kb; idx += blockDim.x) {
        int i = idx / kb, j = idx % kb;
        S[i * LD + j] = D[(long long)i * nf + j];
    }
    if (tid < KB) prow[tid] = tid;
    __syncthreads();
    // Column j: warp 0 finds the pivot, swaps the two rows, applies the
    // static-pivot threshold and scales the column below the diagonal (one
    // block barrier); then all threads update the trailing block, thread
    // (tid / 16, tid % 16) taking every 16th row and column (a second one).
    const int ty = tid >> 4, tx = tid & 15;
    for (int j = 0; j < kb; j++) {
        if (tid < 32) {
            T best = -1; int bi = j;
            for (int i = j + tid; i < kb; i += 32) {
                T v = cabs2(S[i * LD + j]);
                if (v > best) { best = v; bi = i; }
            }
            for (int o = 16; o > 0; o >>= 1) {   // every lane ends with the same (best, bi)
                T ov = __shfl_xor_sync(0xffffffffu, best, o);
                int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            const int pv = bi;
            if (pv != j)
                for (int c = tid; c < kb; c += 32) {
                    cx<T> a = S[j * LD + c];
                    S[j * LD + c] = S[pv * LD + c];
                    S[pv * LD + c] = a;
                }
            __syncwarp();
            if (tid == 0) {
                ipiv[F.first + k + j] = k + pv;
                const int a = prow[j];
                prow[j] = prow[pv];
                prow[pv] = a;
                cx<T> d = S[j * LD + j];
                T m2 = cabs2(d);
                if (!(m2 >= thresh * thresh)) {   // also catches NaN
                    T m = sqrt(m2);
                    S[j * LD + j] = (m > 0 && m == m) ? d * (thresh / m) : cx<T>(thresh);
                    atomicAdd(npert, 1);
                }
            }
            __syncwarp();
            const cx<T> inv = cdiv(cx<T>(1), S[j * LD + j]);
            for (int i = j + 1 + tid; i < kb; i += 32) S[i * LD + j] = S[i * LD + j] * inv;
        }
        __syncthreads();
        for (int i = j + 1 + ty; i < kb; i += 16) {
            const cx<T> l = S[i * LD + j];
            for (int c = j + 1 + tx; c < kb; c += 16) S[i * LD + c] = S[i * LD + c] - l * S[j * LD + c];
        }
        __syncthreads();
    }
    for (int idx = tid; idx < kb * kb; idx += blockDim.x) {
        int i = idx / kb, j = idx % kb;
        D[(long long)i * nf + j] = S[i * LD + j];
    }
    if (tid < kb) gord[F.first + k + tid] = F.first + k + prow[tid];
}

// ---------------------------------------------------------------------------
// row band right of the panel: swap rows, then L_D^{-1} (unit lower)
// ---------------------------------------------------------------------------
constexpr int TRW = 128;   // columns per CTA
template <class T>
__global__ void __launch_bounds__(TRW) k_trsm_row(const RowTask *__restrict__ tasks, const FrontDev *__restrict__ fr,
                                                  cx<T> *__restrict__ fac, const int *__restrict__ gord)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *L = reinterpret_cast<cx<T> *>(smraw);          // KB x (KB+1)
    cx<T> *Bt = L + KB * (KB + 1);                       // KB x (TRW+1)
    __shared__ int idx[KB];
    const RowTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    const int c0 = t.c0, nc = min(TRW, nf - c0);
    const int tid = threadIdx.x;
    cx<T> *base = fac + F.fac + (long long)k * nf;
    #pragma unroll 8   // several loads in flight per thread
    for (int q = tid; q < kb * kb; q += blockDim.x) {
        int i = q / kb, j = q % kb;
        L[i * (KB + 1) + j] = base[(long long)i * nf + k + j];
    }
    panel_rows(gord, F.first + k, kb, idx);
    __syncthreads();
    #pragma unroll 8   // several loads in flight per thread
    for (int q = tid; q < kb * nc; q += blockDim.x) {
        int i = q / nc, c = q % nc;
        Bt[i * (TRW + 1) + c] = base[(long long)idx[i] * nf + c0 + c];
    }
    __syncthreads();
    if (tid < nc) {
        for (int i = 1; i < kb; i++) {
            cx<T> s = Bt[i * (TRW + 1) + tid];
            for (int l = 0; l < i; l++) s = s - L[i * (KB + 1) + l] * Bt[l * (TRW + 1) + tid];
            Bt[i * (TRW + 1) + tid] = s;
        }
    }
    __syncthreads();
    for (int q = tid; q < kb * nc; q += blockDim.x) {
        int i = q / nc, c = q % nc;
        base[(long long)i * nf + c0 + c] = Bt[i * (TRW + 1) + c];
    }
}

// ---------------------------------------------------------------------------
// column band below the panel: X <- X U_D^{-1}
// ---------------------------------------------------------------------------
constexpr int TCR = 128;   // rows per CTA
template <class T>
__global__ void __launch_bounds__(TCR) k_trsm_col(const ColTask *__restrict__ tasks, const FrontDev *__restrict__ fr,
                                                  cx<T> *__restrict__ fac)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *U = reinterpret_cast<cx<T> *>(smraw);          // KB x (KB+1)
    cx<T> *Xs = U + KB * (KB + 1);                        // TCR x (KB+1)
    __shared__ cx<T> invd[KB];
    const ColTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    const int tid = threadIdx.x;
    const cx<T> *D = fac + F.fac + (long long)k * nf + k;
    #pragma unroll 8   // several loads in flight per thread
    for (int q = tid; q < kb * kb; q += blockDim.x) {
        int i = q / kb, j = q % kb;
        U[i * (KB + 1) + j] = D[(long long)i * nf + j];
    }
    cx<T> *xb;
    long long ld;
    int nr;
    if (t.which == 0) {
        xb = fac + F.fac + (long long)t.r0 * nf + k;
        ld = nf;
        nr = min(TCR, F.p - t.r0);
    } else {
        xb = fac + F.fac + (long long)F.p * nf + (long long)t.r0 * F.p + k;
        ld = F.p;
        nr = min(TCR, F.b - t.r0);
    }
    #pragma unroll 8   // several loads in flight per thread
    for (int q = tid; q < nr * kb; q += blockDim.x) {
        int r = q / kb, j = q % kb;
        Xs[r * (KB + 1) + j] = xb[(long long)r * ld + j];
    }
    __syncthreads();
    for (int j = tid; j < kb; j += blockDim.x) invd[j] = cdiv(cx<T>(1), U[j * (KB + 1) + j]);
    __syncthreads();
    if (tid < nr) {
        cx<T> *x = Xs + tid * (KB + 1);
        for (int j = 0; j < kb; j++) {
            cx<T> s = x[j];
            for (int l = 0; l < j; l++) s = s - x[l] * U[l * (KB + 1) + j];
            x[j] = s * invd[j];
        }
    }
    __syncthreads();
    for (int q = tid; q < nr * kb; q += blockDim.x) {
        int r = q / kb, j = q % kb;
        xb[(long long)r * ld + j] = Xs[r * (KB + 1) + j];
    }
}

// Asynchronous global -> shared copy of one complex element (8 or 16 bytes,
// naturally aligned), and the wait for all of a thread's copies.
template <class T>
__device__ __forceinline__ void cp_async_cx(cx<T> *dst, const cx<T> *src)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(cx<T>) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------------------
// complex64 band solves by substitution, one column (row band) or one row
// (column band) per thread, in eight groups of eight unknowns.  For group G
// the thread solves its eight unknowns in registers with the diagonal 8 x 8
// block of the tile, writes them back to its own column (row) in shared
// memory, and then subtracts their multiples from every later group H, one
// 8 x 8 block of the tile at a time (the tile's rows are read as 16-byte
// broadcasts).  The loops over G and H are not unrolled, so the kernel's code
// stays small: fully unrolled, the 2,016 multiply-adds of a 64-vector are
// some 12k instructions per thread, and the warps then wait on instruction
// fetch (ncu: 1.7 cycles per issue stalled on no_instruction, 24 % issue
// activity).  The tile is padded with the identity beyond kb (a last,
// narrower panel).
// ---------------------------------------------------------------------------
constexpr int TG = 8;                       // unknowns per group
constexpr int LDT = KB + 2;                 // tile row stride: 16-byte-aligned rows
__host__ __device__ constexpr size_t band_row_smem() { return sizeof(cx<float>) * (KB * LDT + KB * (TRW + 1)); }
__host__ __device__ constexpr size_t band_col_smem() { return sizeof(cx<float>) * (KB * LDT + TCR * (KB + 1)); }

__device__ __forceinline__ void cfms(cx<float> &d, const cx<float> a, const cx<float> b)   // d -= a b
{
    d.re = fmaf(-a.re, b.re, fmaf(a.im, b.im, d.re));
    d.im = fmaf(-a.re, b.im, fmaf(-a.im, b.re, d.im));
}

// eight consecutive complex values of a 16-byte-aligned shared-memory row
__device__ __forceinline__ void lds8(const cx<float> *p, cx<float> (&a)[TG])
{
#pragma unroll
    for (int j = 0; j < TG; j += 2) {
        const float4 u = reinterpret_cast<const float4 *>(p)[j / 2];
        a[j] = cx<float>(u.x, u.y);
        a[j + 1] = cx<float>(u.z, u.w);
    }
}

// the KB x KB diagonal tile into shared memory (row stride LDT), identity
// beyond kb
__device__ __forceinline__ void load_tile_padded(cx<float> *T, const cx<float> *D, long long nf, int kb)
{
    for (int q = threadIdx.x; q < KB * KB; q += blockDim.x) {
        const int i = q / KB, j = q % KB;
        if (i < kb && j < kb) cp_async_cx(T + i * LDT + j, D + (long long)i * nf + j);
        else T[i * LDT + j] = cx<float>(i == j ? 1.f : 0.f, 0.f);
    }
}

template <int UNUSED = 0>
__global__ void __launch_bounds__(TRW) k_trsm_row_h(const RowTask *__restrict__ tasks, const FrontDev *__restrict__ fr,
                                                    cx<float> *__restrict__ fac, const int *__restrict__ gord)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<float> *L = reinterpret_cast<cx<float> *>(smraw);   // KB x LDT
    cx<float> *Bt = L + KB * LDT;                         // KB x (TRW+1): band rows as stored
    __shared__ int idx[KB];
    const RowTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    const int c0 = t.c0, nc = min(TRW, nf - c0);
    const int tid = threadIdx.x;
    cx<float> *base = fac + F.fac + (long long)k * nf;
    load_tile_padded(L, base + k, nf, kb);
    for (int q = tid; q < kb * nc; q += blockDim.x) {
        const int i = q / nc, c = q % nc;
        cp_async_cx(Bt + i * (TRW + 1) + c, base + (long long)i * nf + c0 + c);
    }
    panel_rows(gord, F.first + k, kb, idx);
    cp_async_wait_all();
    __syncthreads();
    // Row i of the result is kept in the stored slot idx[i] of the row it
    // came from: the slots of rows not yet read stay untouched.  Unknowns at
    // or beyond kb are zero and stay zero (identity padding).
    if (tid < nc) {
        cx<float> *col = Bt + tid;
        const int ng = (kb + TG - 1) / TG;
#pragma unroll 1
        for (int G = 0; G < ng; G++) {
            cx<float> b[TG];
#pragma unroll
            for (int i = 0; i < TG; i++) b[i] = TG * G + i < kb ? col[idx[TG * G + i] * (TRW + 1)] : cx<float>(0.f, 0.f);
#pragma unroll
            for (int i = 1; i < TG; i++) {
                cx<float> lr[TG];
                lds8(L + (TG * G + i) * LDT + TG * G, lr);
#pragma unroll
                for (int l = 0; l < i; l++) cfms(b[i], lr[l], b[l]);
            }
#pragma unroll
            for (int i = 0; i < TG; i++)
                if (TG * G + i < kb) col[idx[TG * G + i] * (TRW + 1)] = b[i];
#pragma unroll 1
            for (int H = G + 1; H < ng; H++) {
#pragma unroll
                for (int i = 0; i < TG; i++) {
                    const int row = TG * H + i;
                    if (row < kb) {
                        cx<float> lr[TG];
                        lds8(L + row * LDT + TG * G, lr);
                        cx<float> c = col[idx[row] * (TRW + 1)];
#pragma unroll
                        for (int l = 0; l < TG; l++) cfms(c, lr[l], b[l]);
                        col[idx[row] * (TRW + 1)] = c;
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int q = tid; q < kb * nc; q += blockDim.x) {
        const int i = q / nc, c = q % nc;
        base[(long long)i * nf + c0 + c] = Bt[idx[i] * (TRW + 1) + c];
    }
}

template <int UNUSED = 0>
__global__ void __launch_bounds__(TCR) k_trsm_col_h(const ColTask *__restrict__ tasks, const FrontDev *__restrict__ fr,
                                                    cx<float> *__restrict__ fac)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<float> *U = reinterpret_cast<cx<float> *>(smraw);   // KB x LDT
    cx<float> *Xs = U + KB * LDT;                         // TCR x (KB+1)
    __shared__ cx<float> invd[KB];
    const ColTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    const int tid = threadIdx.x;
    load_tile_padded(U, fac + F.fac + (long long)k * nf + k, nf, kb);
    cx<float> *xb;
    long long ld;
    int nr;
    if (t.which == 0) {
        xb = fac + F.fac + (long long)t.r0 * nf + k;
        ld = nf;
        nr = min(TCR, F.p - t.r0);
    } else {
        xb = fac + F.fac + (long long)F.p * nf + (long long)t.r0 * F.p + k;
        ld = F.p;
        nr = min(TCR, F.b - t.r0);
    }
    for (int q = tid; q < nr * kb; q += blockDim.x) {
        const int r = q / kb, j = q % kb;
        cp_async_cx(Xs + r * (KB + 1) + j, xb + (long long)r * ld + j);
    }
    cp_async_wait_all();
    __syncthreads();
    for (int j = tid; j < KB; j += blockDim.x) invd[j] = cdiv(cx<float>(1.f, 0.f), U[j * LDT + j]);
    __syncthreads();
    if (tid < nr) {
        cx<float> *row = Xs + tid * (KB + 1);
        const int ng = (kb + TG - 1) / TG;
#pragma unroll 1
        for (int G = 0; G < ng; G++) {
            cx<float> x[TG];
#pragma unroll
            for (int j = 0; j < TG; j++) x[j] = TG * G + j < kb ? row[TG * G + j] : cx<float>(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < TG; j++) {
                x[j] = x[j] * invd[TG * G + j];
                cx<float> ur[TG];
                lds8(U + (TG * G + j) * LDT + TG * G, ur);
#pragma unroll
                for (int j2 = j + 1; j2 < TG; j2++) cfms(x[j2], x[j], ur[j2]);
            }
#pragma unroll
            for (int j = 0; j < TG; j++)
                if (TG * G + j < kb) row[TG * G + j] = x[j];
#pragma unroll 1
            for (int H = G + 1; H < ng; H++) {
                cx<float> y[TG];
#pragma unroll
                for (int j = 0; j < TG; j++) y[j] = TG * H + j < kb ? row[TG * H + j] : cx<float>(0.f, 0.f);
#pragma unroll
                for (int l = 0; l < TG; l++) {
                    cx<float> ur[TG];
                    lds8(U + (TG * G + l) * LDT + TG * H, ur);
#pragma unroll
                    for (int j = 0; j < TG; j++) cfms(y[j], x[l], ur[j]);
                }
#pragma unroll
                for (int j = 0; j < TG; j++)
                    if (TG * H + j < kb) row[TG * H + j] = y[j];
            }
        }
    }
    __syncthreads();
    for (int q = tid; q < nr * kb; q += blockDim.x) {
        const int r = q / kb, j = q % kb;
        xb[(long long)r * ld + j] = Xs[r * (KB + 1) + j];
    }
}

// ---------------------------------------------------------------------------
// SIMT complex GEMM  C -= op(A) * B  (64x64 tiles, 4x4 per thread)
// ---------------------------------------------------------------------------
constexpr int GBM = 64, GBN = 64, GBK = 16;
template <class T>
__global__ void __launch_bounds__(256) k_gemm(const GemmTask<T> *__restrict__ tasks, int ntasks)
{
    __shared__ cx<T> As[GBK][GBM + 1];
    __shared__ cx<T> Bs[GBK][GBN];
    const int ti = find_task(tasks, ntasks, (long long)blockIdx.x);
    const GemmTask<T> t = tasks[ti];
    const long long lt = (long long)blockIdx.x - t.tile0;
    const int m0 = (int)(lt / t.tiles_n) * GBM, n0 = (int)(lt % t.tiles_n) * GBN;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    cx<T> acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = cx<T>(0);
    for (int k0 = 0; k0 < t.K; k0 += GBK) {
        if (!t.conjA) {
#pragma unroll
            for (int q = 0; q < (GBM * GBK) / 256; q++) {
                int idx = tid + q * 256;
                int i = idx / GBK, kk = idx % GBK;
                int r = m0 + i, c = k0 + kk;
                As[kk][i] = (r < t.M && c < t.K) ? t.A[(long long)r * t.lda + c] : cx<T>(0);
            }
        } else {
            // op(A)[r][c] = conj(A[c][r])
#pragma unroll
            for (int q = 0; q < (GBM * GBK) / 256; q++) {
                int idx = tid + q * 256;
                int kk = idx / GBM, i = idx % GBM;
                int r = m0 + i, c = k0 + kk;
                As[kk][i] = (r < t.M && c < t.K) ? conj(t.A[(long long)c * t.lda + r]) : cx<T>(0);
            }
        }
#pragma unroll
        for (int q = 0; q < (GBK * GBN) / 256; q++) {
            int idx = tid + q * 256;
            int kk = idx / GBN, j = idx % GBN;
            int r = k0 + kk, c = n0 + j;
            cx<T> v(0);
            if (r < t.K && c < t.N) {
                long long row = t.brow ? (long long)t.brow[r] : (long long)r;
                v = t.B[row * t.ldb + c];
            }
            Bs[kk][j] = v;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GBK; kk++) {
            cx<T> a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = As[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc[i][j].re = fma(a[i].re, b[j].re, fma(-a[i].im, b[j].im, acc[i][j].re));
                    acc[i][j].im = fma(a[i].re, b[j].im, fma(a[i].im, b[j].re, acc[i][j].im));
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int r = m0 + ty + 16 * i;
        if (r >= t.M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int c = n0 + tx + 16 * j;
            if (c >= t.N) continue;
            if (t.crow) {
                atomic_sub(t.C + (long long)t.crow[r] * t.ldc + c, acc[i][j]);
            } else {
                cx<T> *p = t.C + (long long)r * t.ldc + c;
                *p = *p - acc[i][j];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Tall-skinny SIMT complex GEMM  C -= op(A) * B  for N <= 32 (the right-hand
// side blocks of the substitution passes): 128 x 32 tiles, 4 x 4 complex
// outputs per thread, every A element read once per tile.
// ---------------------------------------------------------------------------
constexpr int TSBM = 128, TSBN = 32, TSBK = 16;   // TSBK: K granularity of split-K chunks
template <class T> struct TsCfg { static constexpr int BK = sizeof(T) == 4 ? 32 : 16; };

// 128 x 32 tile per CTA of 256 threads; thread (tx, ty) owns rows 4ty..4ty+3
// and columns 4tx..4tx+3 (16 complex accumulators).  The K loop stages
// BK-deep slices of A (transposed in shared memory) and B, prefetching the
// next slice into registers while the current one is consumed.
template <class T>
__global__ void __launch_bounds__(256, 2) k_gemm_ts(const GemmTask<T> *__restrict__ tasks, int ntasks)
{
    constexpr int BK = TsCfg<T>::BK;
    constexpr int AP = TSBM + 1;                       // padded row of the A^T slice
    constexpr int NA = TSBM * BK / 256, NB = BK * TSBN / 256;
    __shared__ cx<T> As[BK][AP];
    __shared__ cx<T> Bs[BK][TSBN];
    const int ti = find_task(tasks, ntasks, (long long)blockIdx.x);
    const GemmTask<T> t = tasks[ti];
    const int m0 = (int)((long long)blockIdx.x - t.tile0) * TSBM;
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    cx<T> acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = cx<T>(0);
    cx<T> pa[NA], pb[NB];
    // A slice element q of this thread: non-conjugate A is read along K
    // (row-contiguous), the conjugate transpose along M.
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < NA; q++) {
            const int idx = tid + q * 256;
            int i, kk;
            if (!t.conjA) { i = idx / BK; kk = idx % BK; }
            else { kk = idx / TSBM; i = idx % TSBM; }
            const int r = m0 + i, c = k0 + kk;
            cx<T> v(0);
            if (r < t.M && c < t.K) v = t.conjA ? conj(t.A[(long long)c * t.lda + r]) : t.A[(long long)r * t.lda + c];
            pa[q] = v;
        }
#pragma unroll
        for (int q = 0; q < NB; q++) {
            const int idx = tid + q * 256;
            const int kk = idx / TSBN, j = idx % TSBN;
            const int r = k0 + kk;
            cx<T> v(0);
            if (r < t.K && j < t.N) v = t.B[(t.brow ? (long long)t.brow[r] : (long long)r) * t.ldb + j];
            pb[q] = v;
        }
    };
    auto store = [&]() {
#pragma unroll
        for (int q = 0; q < NA; q++) {
            const int idx = tid + q * 256;
            int i, kk;
            if (!t.conjA) { i = idx / BK; kk = idx % BK; }
            else { kk = idx / TSBM; i = idx % TSBM; }
            As[kk][i] = pa[q];
        }
#pragma unroll
        for (int q = 0; q < NB; q++) {
            const int idx = tid + q * 256;
            Bs[idx / TSBN][idx % TSBN] = pb[q];
        }
    };
    load(0);
    for (int k0 = 0; k0 < t.K; k0 += BK) {
        store();
        __syncthreads();
        if (k0 + BK < t.K) load(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            cx<T> a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = As[kk][4 * ty + i];
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = Bs[kk][4 * tx + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc[i][j].re = fma(a[i].re, b[j].re, fma(-a[i].im, b[j].im, acc[i][j].re));
                    acc[i][j].im = fma(a[i].re, b[j].im, fma(a[i].im, b[j].re, acc[i][j].im));
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = m0 + 4 * ty + i;
        if (r >= t.M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = 4 * tx + j;
            if (c >= t.N) continue;
            if (t.crow) atomic_sub(t.C + (long long)t.crow[r] * t.ldc + c, acc[i][j]);
            else if (t.atom) atomic_sub(t.C + (long long)r * t.ldc + c, acc[i][j]);
            else {
                cx<T> *p = t.C + (long long)r * t.ldc + c;
                *p = *p - acc[i][j];
            }
        }
    }
}

}  // namespace wt3d
