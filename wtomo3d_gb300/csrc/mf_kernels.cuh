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
#include <algorithm>
#include <vector>

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
struct EATask { int child, parent; long long row0; };
template <class T>
struct GemmTask {
    const cx<T> *A;
    const cx<T> *B;
    cx<T> *C;
    const int *brow;   // optional row gather for B
    const int *crow;   // optional row scatter for C (atomic)
    int lda, ldb, ldc, M, N, K;
    int conjA;         // use conj(A^T): A is read as its conjugate transpose
};

template <class T>
__device__ __forceinline__ void atomic_sub(cx<T> *p, cx<T> v)
{
    atomicAdd(&p->re, -v.re);
    atomicAdd(&p->im, -v.im);
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

// ---------------------------------------------------------------------------
// panel: LU of the KB x KB diagonal tile with partial pivoting inside the tile
// ---------------------------------------------------------------------------
// order-preserving unsigned keys of non-negative values, 0 for NaN
__device__ __forceinline__ unsigned pivot_key(float v) { return v == v ? __float_as_uint(v) : 0u; }
__device__ __forceinline__ unsigned long long pivot_key(double v)
{
    return v == v ? (unsigned long long)__double_as_longlong(v) : 0ull;
}
__device__ __forceinline__ unsigned warp_max(unsigned k) { return __reduce_max_sync(0xffffffffu, k); }
__device__ __forceinline__ unsigned long long warp_max(unsigned long long k)
{
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
    return ((unsigned long long)hi << 32) | lo;
}

// element i (a run-time index) of four registers
template <class T>
__device__ __forceinline__ cx<T> pick(const cx<T> &a0, const cx<T> &a1, const cx<T> &a2, const cx<T> &a3, int i)
{
    const cx<T> lo = (i & 1) ? a1 : a0, hi = (i & 1) ? a3 : a2;
    return (i & 2) ? hi : lo;
}

// One CTA per tile; a chain of 64 dependent columns, so the latency of a column
// is what counts.  The tile is held in registers: thread (tx, ty) =
// (tid / 16, tid % 16) owns rows ty + 16 i and columns tx + 16 c, so that a
// column's 64 entries sit in one half-warp and its pivot is found by two warp
// reductions, without a barrier.  Rows stay where they are: a chosen row is
// marked, the others go on, and rows are stored in the order they were chosen
// in (gord).  Two barriers per column: the multipliers and the pivot's row
// number, then the pivot row.  Equal magnitudes: the smallest stored row.
// With the tile and its row swaps in shared memory a launch of few tiles took
// 55 - 80 us.  Panels and bands together, 24x22x20: 59 steps 7.3 -> 3.9 ms;
// 64x64x48: 358 steps 72 -> 54 ms.
template <class T>
__global__ void __launch_bounds__(256, 1) k_panel(const PanelTask *__restrict__ tasks,
                                                  const FrontDev *__restrict__ fr, cx<T> *__restrict__ fac,
                                                  const unsigned long long *__restrict__ amax2, double pivot_rel,
                                                  int *__restrict__ npert, int *__restrict__ gord)
{
    // static-pivot threshold: pivot_rel * max |a_ij| of the assembled operator
    const T thresh = (T)(pivot_rel * sqrt(__longlong_as_double((long long)*amax2)));
    __shared__ cx<T> lcol[2][KB], urow[KB];
    __shared__ int s_p[2], pos[KB];
    const PanelTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    cx<T> *D = fac + F.fac + (long long)k * nf + k;
    const int tid = threadIdx.x, tx = tid >> 4, ty = tid & 15, warp = tid >> 5, lane = tid & 31;
    cx<T> a[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int r = ty + 16 * i, q = tx + 16 * c;
            a[i][c] = (r < kb && q < kb) ? D[(long long)r * nf + q] : cx<T>(0);
        }
    unsigned used = 0;   // bit i: row ty + 16 i has been chosen, or is none of the tile's
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (ty + 16 * i >= kb) used |= 1u << i;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        for (int jj = 0; jj < 16; jj++) {
            const int j = 16 * c + jj, buf = j & 1;
            if (j >= kb) break;
            if (warp == jj >> 1) {
                const bool mine = (lane >> 4) == (jj & 1);   // the half-warp that holds column j
                decltype(pivot_key(T(0))) key = 0, ki[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    ki[i] = pivot_key(cabs2(a[i][c]));
                    if (!((used >> i) & 1u) && ki[i] > key) key = ki[i];
                }
                if (!mine) key = 0;
                const auto best = warp_max(key);
                int row = KB;
#pragma unroll
                for (int i = 3; i >= 0; i--)
                    if (mine && !((used >> i) & 1u) && ki[i] == best) row = ty + 16 * i;
                const int p = (int)__reduce_min_sync(0xffffffffu, (unsigned)row);
                const int src = (p & 15) + 16 * (jj & 1);
                cx<T> d = pick(a[0][c], a[1][c], a[2][c], a[3][c], p >> 4);
                d.re = __shfl_sync(0xffffffffu, d.re, src);
                d.im = __shfl_sync(0xffffffffu, d.im, src);
                const T m2 = cabs2(d);
                if (!(m2 >= thresh * thresh)) {   // also catches NaN
                    const T m = sqrt(m2);
                    d = (m > 0 && m == m) ? d * (thresh / m) : cx<T>(thresh);
                    if (lane == src) atomicAdd(npert, 1);
                }
                const cx<T> inv = cdiv(cx<T>(1), d);
                if (mine) {
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int r = ty + 16 * i;
                        if (r == p) a[i][c] = d;
                        else if (!((used >> i) & 1u)) {
                            a[i][c] = a[i][c] * inv;
                            lcol[buf][r] = a[i][c];
                        }
                    }
                    if (lane == src) {
                        s_p[buf] = p;
                        pos[p] = j;
                    }
                }
            }
            __syncthreads();
            const int p = s_p[buf];
            if ((p & 15) == ty) {
                const int i = p >> 4;
#pragma unroll
                for (int q = c; q < 4; q++) urow[tx + 16 * q] = pick(a[0][q], a[1][q], a[2][q], a[3][q], i);
                used |= 1u << i;
            }
            __syncthreads();
            cx<T> l[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (!((used >> i) & 1u)) l[i] = lcol[buf][ty + 16 * i];
#pragma unroll
            for (int q = c; q < 4; q++) {
                if (q == c && tx <= jj) continue;
                const cx<T> u = urow[tx + 16 * q];
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (!((used >> i) & 1u)) {
                        a[i][q].re = fma(-l[i].re, u.re, fma(l[i].im, u.im, a[i][q].re));
                        a[i][q].im = fma(-l[i].re, u.im, fma(-l[i].im, u.re, a[i][q].im));
                    }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = ty + 16 * i;
        if (r >= kb) continue;
        const int o = pos[r];
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (tx + 16 * c < kb) D[(long long)o * nf + tx + 16 * c] = a[i][c];
        if (tx == 0) gord[F.first + k + o] = F.first + k + r;
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

template <class T>
__device__ __forceinline__ void cfms(cx<T> &d, const cx<T> a, const cx<T> b)   // d -= a b
{
    d.re = fma(-a.re, b.re, fma(a.im, b.im, d.re));
    d.im = fma(-a.re, b.im, fma(-a.im, b.re, d.im));
}

// 16-byte-aligned shared loads of N consecutive complex values
template <int N>
__device__ __forceinline__ void lds_cx(const cx<float> *p, cx<float> (&a)[N])
{
    if constexpr (N == 1) {
        a[0] = *p;
    } else {
#pragma unroll
        for (int j = 0; j < N; j += 2) {
            const float4 u = reinterpret_cast<const float4 *>(p)[j / 2];
            a[j] = cx<float>(u.x, u.y);
            a[j + 1] = cx<float>(u.z, u.w);
        }
    }
}
template <int N>
__device__ __forceinline__ void lds_cx(const cx<double> *p, cx<double> (&a)[N])
{
#pragma unroll
    for (int j = 0; j < N; j++) {
        const double2 u = reinterpret_cast<const double2 *>(p)[j];
        a[j] = cx<double>(u.x, u.y);
    }
}

// ---------------------------------------------------------------------------
// bands of a panel: the rows right of it, B <- L_D^{-1} P B, and the columns
// below it, X <- X U_D^{-1}, by substitution, in one launch (they do not depend
// on one another).  Both are solves with a lower triangle T, vector by vector:
// T = L_D (unit) for a column of the row band, T = U_D^T for a row of the column
// band.  Four threads share a vector, in groups of TG unknowns: each of them
// solves the group's diagonal block (redundantly, in registers) and subtracts
// its multiples from every fourth row below, so that the dependent chain of a
// vector is a third of one thread's.  A launch of the small and middle levels
// has few vectors and is bound by that chain: 27 us each for the two launches
// with one thread per vector.  The loops over groups are not unrolled: the
// kernel's code stays in the instruction cache.  The tile is padded with the
// identity beyond kb (a last, narrower panel).
// ---------------------------------------------------------------------------
struct BandTask { int f, k, c0, which; };   // which: 0 columns right, 1 pivot rows below, 2 border rows; c0: the first
constexpr int BD_V = 32, BD_TH = 4 * BD_V;  // vectors and threads per CTA
template <class T>
struct BandCfg {
    static constexpr int TG = sizeof(T) == 4 ? 8 : 4;       // unknowns per group
    static constexpr int LDT = KB + 16 / (int)sizeof(cx<T>);   // tile rows on 16 bytes, four rows on different banks
    static constexpr int LDX = sizeof(T) == 4 ? BD_V + 4 : BD_V + 2;
    static constexpr size_t smem = sizeof(cx<T>) * (KB * LDT + KB * LDX);
};

// T x = b for the BD_V vectors of X (b on entry, zero before group first / TG);
// unit: T's diagonal is one, otherwise invd holds its inverse.
template <class T>
__device__ __forceinline__ void band_solve(const cx<T> *Tm, cx<T> *X, const cx<T> *invd, bool unit, int first, int kb)
{
    constexpr int TG = BandCfg<T>::TG, LDT = BandCfg<T>::LDT, LDX = BandCfg<T>::LDX;
    const int v = threadIdx.x >> 2, q4 = threadIdx.x & 3;
    const int ng = (kb + TG - 1) / TG;
    cx<T> *x = X + v;
#pragma unroll 1
    for (int G = first / TG; G < ng; G++) {
        cx<T> b[TG];
#pragma unroll
        for (int i = 0; i < TG; i++) b[i] = x[(TG * G + i) * LDX];
#pragma unroll
        for (int i = 0; i < TG; i++) {
            if (i > 0) {
                cx<T> lr[TG];
                lds_cx<TG>(Tm + (TG * G + i) * LDT + TG * G, lr);
#pragma unroll
                for (int l = 0; l < i; l++) cfms(b[i], lr[l], b[l]);
            }
            if (!unit) b[i] = b[i] * invd[TG * G + i];
        }
        __syncwarp();   // the four threads have read the group
#pragma unroll
        for (int i = 0; i < TG; i++)
            if ((i & 3) == q4) x[(TG * G + i) * LDX] = b[i];
#pragma unroll 1
        for (int H = TG * (G + 1) + q4; H < TG * ng; H += TG) {
#pragma unroll
            for (int i = 0; i < TG; i += 4) {
                cx<T> lr[TG], c = x[(H + i) * LDX];
                lds_cx<TG>(Tm + (H + i) * LDT + TG * G, lr);
#pragma unroll
                for (int l = 0; l < TG; l++) cfms(c, lr[l], b[l]);
                x[(H + i) * LDX] = c;
            }
        }
        __syncwarp();
    }
}

template <class T>
__global__ void __launch_bounds__(BD_TH) k_bands(const BandTask *__restrict__ tasks, const FrontDev *__restrict__ fr,
                                                 cx<T> *__restrict__ fac, const int *__restrict__ gord)
{
    using C = BandCfg<T>;
    constexpr int LDT = C::LDT, LDX = C::LDX;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *Tm = reinterpret_cast<cx<T> *>(smraw);   // KB x LDT
    cx<T> *X = Tm + KB * LDT;                       // KB x LDX: unknown i of vector v
    __shared__ int idx[KB];
    __shared__ cx<T> invd[KB];
    const BandTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    const int tid = threadIdx.x;
    const bool row = t.which == 0;
    const cx<T> *D = fac + F.fac + (long long)k * nf + k;
    for (int q = tid; q < KB * KB; q += BD_TH) {
        const int i = q / KB, j = q % KB;   // tile entry (i, j) as stored
        cx<T> *dst = row ? Tm + i * LDT + j : Tm + j * LDT + i;
        if (i < kb && j < kb) cp_async_cx(dst, D + (long long)i * nf + j);
        else *dst = cx<T>(i == j ? T(1) : T(0));
    }
    cx<T> *xb;     // unknown i of vector v at xb + i * si + v * sv
    long long si, sv;
    int nv;
    if (row) {
        xb = fac + F.fac + (long long)k * nf + t.c0;
        si = nf;
        sv = 1;
        nv = min(BD_V, nf - t.c0);
        if (tid < KB) idx[tid] = tid < kb ? gord[F.first + k + tid] - F.first - k : 0;
        __syncthreads();
        for (int q = tid; q < KB * BD_V; q += BD_TH) {
            const int i = q / BD_V, v = q % BD_V;
            if (i < kb && v < nv) cp_async_cx(X + i * LDX + v, xb + idx[i] * si + v);
            else X[i * LDX + v] = cx<T>(0);
        }
    } else {
        if (t.which == 1) {
            xb = fac + F.fac + (long long)t.c0 * nf + k;
            sv = nf;
            nv = min(BD_V, F.p - t.c0);
        } else {
            xb = fac + F.fac + (long long)F.p * nf + (long long)t.c0 * F.p + k;
            sv = F.p;
            nv = min(BD_V, F.b - t.c0);
        }
        si = 1;
        for (int q = tid; q < KB * BD_V; q += BD_TH) {
            const int i = q % KB, v = q / KB;
            if (i < kb && v < nv) cp_async_cx(X + i * LDX + v, xb + v * sv + i);
            else X[i * LDX + v] = cx<T>(0);
        }
    }
    cp_async_wait_all();
    __syncthreads();
    if (tid < KB) invd[tid] = row ? cx<T>(1) : cdiv(cx<T>(1), Tm[tid * LDT + tid]);
    __syncthreads();
    band_solve<T>(Tm, X, invd, row, 0, kb);
    __syncthreads();
    for (int q = tid; q < KB * BD_V; q += BD_TH) {
        const int i = row ? q / BD_V : q % KB, w = row ? q % BD_V : q / KB;
        if (i < kb && w < nv) xb[i * si + w * sv] = X[i * LDX + w];
    }
}

// ---------------------------------------------------------------------------
// SIMT complex GEMM  C -= A B: the products that are too small for the
// tensor-core kernel and its operand split, and all complex128 ones
// ---------------------------------------------------------------------------
// One CTA per unit: a BM x 32 tile of C (4 x 4 per thread) and a range of K.
// Operands go through a ring of three asynchronous-copy stages; the tile of C,
// which does not depend on the product, is loaded first.  Complex64 tiles are 64
// rows high (73 TF/s FP32 peak; the unpipelined 64 x 64 kernel reached 4 - 11).
// Complex128 tiles are 32 rows high: the FP64 pipe (2 FMA per cycle and SM) is
// the bound, and smaller tiles fill the last wave (a 630 x 630 x 600 update is
// 100 tiles of 64 x 64 on 152 SMs, but 400 of 32 x 32).
struct GemmUnit { int task, m0, n0, k0, k1, atom; };
template <class T>
struct GemmCfg {
    static constexpr int BM = sizeof(T) == 4 ? 64 : 32, BN = 32;
    static constexpr int BK = sizeof(T) == 4 ? 16 : 8, NS = 3;
    static constexpr int TH = (BM / 4) * (BN / 4), VK = 16 / (int)sizeof(cx<T>), LDA = BK + VK;
};

template <class T>
__device__ __forceinline__ void cp_async_cx_z(cx<T> *dst, const cx<T> *src, bool ok)   // zeros when !ok
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(cx<T>) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

template <class T>
__global__ void __launch_bounds__(GemmCfg<T>::TH) k_gemm(const GemmTask<T> *__restrict__ tasks,
                                                         const GemmUnit *__restrict__ units)
{
    using C = GemmCfg<T>;
    constexpr int BM = C::BM, BN = C::BN, BK = C::BK, NS = C::NS, TH = C::TH, VK = C::VK, LDA = C::LDA;
    __shared__ __align__(16) cx<T> As[NS][BM * LDA];
    __shared__ __align__(16) cx<T> Bs[NS][BK * BN];
    const GemmUnit u = units[blockIdx.x];
    const GemmTask<T> t = tasks[u.task];
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;   // rows ty + (BM / 4) i, columns 4 tx + j
    const int M = t.M - u.m0, N = t.N - u.n0, K = u.k1 - u.k0, nst = (K + BK - 1) / BK;
    const cx<T> *A = t.A + (long long)u.m0 * t.lda + u.k0, *B = t.B + (long long)u.k0 * t.ldb + u.n0;
    auto load = [&](int s) {
        cx<T> *da = As[s % NS], *db = Bs[s % NS];
#pragma unroll
        for (int q = 0; q < BM * BK / TH; q++) {
            const int idx = tid + q * TH, i = idx / BK, kk = idx % BK, k = s * BK + kk;
            const bool ok = i < M && k < K;
            cp_async_cx_z(da + i * LDA + kk, A + (ok ? (long long)i * t.lda + k : 0), ok);
        }
#pragma unroll
        for (int q = 0; q < BK * BN / TH; q++) {
            const int idx = tid + q * TH, kk = idx / BN, j = idx % BN, k = s * BK + kk;
            const bool ok = j < N && k < K;
            cp_async_cx_z(db + idx, B + (ok ? (long long)k * t.ldb + j : 0), ok);
        }
    };
    for (int s = 0; s < NS - 1; s++) {
        if (s < nst) load(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    cx<T> *Cp = t.C + (long long)u.m0 * t.ldc + u.n0;
    cx<T> acc[4][4];   // C minus the products so far
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int r = ty + BM / 4 * i, c = 4 * tx + j;
            acc[i][j] = (!u.atom && r < M && c < N) ? Cp[(long long)r * t.ldc + c] : cx<T>(0);
        }
    for (int s = 0; s < nst; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
        __syncthreads();   // stage s is there for all; stage s - 1 is no longer read
        if (s + NS - 1 < nst) load(s + NS - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const cx<T> *Aw = As[s % NS], *Bw = Bs[s % NS];
#pragma unroll
        for (int kq = 0; kq < BK; kq += VK) {
            cx<T> a[4][VK];
#pragma unroll
            for (int i = 0; i < 4; i++) lds_cx<VK>(Aw + (ty + BM / 4 * i) * LDA + kq, a[i]);
#pragma unroll
            for (int v = 0; v < VK; v++) {
                cx<T> b[4];
                lds_cx<4>(Bw + (kq + v) * BN + 4 * tx, b);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) cfms(acc[i][j], a[i][v], b[j]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int r = ty + BM / 4 * i, c = 4 * tx + j;
            if (r >= M || c >= N) continue;
            cx<T> *p = Cp + (long long)r * t.ldc + c;
            if (u.atom) atomic_sub(p, -acc[i][j]);
            else *p = acc[i][j];
        }
}

// The units of tasks v, numbered from `first` in the launch's task array.  A
// launch with fewer tiles than half the SMs is also cut along K.
template <class T>
void gemm_units(const std::vector<GemmTask<T>> &v, int first, std::vector<GemmUnit> &out)
{
    using C = GemmCfg<T>;
    long long tiles = 0;
    for (const auto &g : v) tiles += (long long)((g.M + C::BM - 1) / C::BM) * ((g.N + C::BN - 1) / C::BN);
    const int cut = tiles > 0 && tiles < 76 ? (int)(152 / tiles) : 1;
    for (size_t i = 0; i < v.size(); i++) {
        const auto &g = v[i];
        const int n = std::max(1, std::min(cut, g.K / 64));
        const int len = ((g.K + n - 1) / n + C::BK - 1) / C::BK * C::BK;
        for (int m0 = 0; m0 < g.M; m0 += C::BM)
            for (int n0 = 0; n0 < g.N; n0 += C::BN)
                for (int k0 = 0; k0 < g.K; k0 += len)
                    out.push_back(GemmUnit{first + (int)i, m0, n0, k0, std::min(g.K, k0 + len), len < g.K ? 1 : 0});
    }
}

}  // namespace wt3d
