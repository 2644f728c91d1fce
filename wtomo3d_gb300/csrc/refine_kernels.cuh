// FP64 kernels of the refinement: layout changes, the residual, and the batched
// Krylov operations.  A block of right-hand sides is row-major, [row][nc], with
// nc = sk_columns(m) columns (1, 4, 8, 16 or 32) in the natural ordering;
// columns m .. nc - 1 are zero.  With a fixed row of 32 columns one source
// moved 32 times its own bytes, and its residual took the FP64 time of 32: a
// warp instruction occupies the FP64 pipe for the same 16 cycles whether one
// lane or all of them take part.
#pragma once
#include "sub_kernels.cuh"

namespace wt3d {

// One instantiation per width.
#define WT_SWITCH_NC(nc, ...)                                  \
    switch (nc) {                                              \
    case 1: { constexpr int NC = 1; __VA_ARGS__; break; }      \
    case 4: { constexpr int NC = 4; __VA_ARGS__; break; }      \
    case 8: { constexpr int NC = 8; __VA_ARGS__; break; }      \
    case 16: { constexpr int NC = 16; __VA_ARGS__; break; }    \
    default: { constexpr int NC = 32; __VA_ARGS__; break; }    \
    }

// Column-major n x m to and from [row][NC], 32 rows per block through shared
// memory, so that both sides are read and written in whole segments.
template <int NC>
__global__ void __launch_bounds__(256) k_cm_to_rm(long long n, int m, const double2 *__restrict__ cm,
                                                  double2 *__restrict__ rm)
{
    __shared__ double2 tile[NC][33];
    const long long i0 = 32LL * blockIdx.x;
    const int nr = (int)min(32LL, n - i0);
    for (int e = threadIdx.x; e < 32 * NC; e += 256) {
        const int c = e / 32, r = e % 32;
        tile[c][r] = (c < m && r < nr) ? cm[(long long)c * n + i0 + r] : make_double2(0, 0);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nr * NC; e += 256) rm[i0 * NC + e] = tile[e % NC][e / NC];
}

template <int NC>
__global__ void __launch_bounds__(256) k_rm_to_cm(long long n, int m, const double2 *__restrict__ rm,
                                                  double2 *__restrict__ cm)
{
    __shared__ double2 tile[NC][33];
    const long long i0 = 32LL * blockIdx.x;
    const int nr = (int)min(32LL, n - i0);
    for (int e = threadIdx.x; e < nr * NC; e += 256) tile[e % NC][e / NC] = rm[i0 * NC + e];
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * NC; e += 256) {
        const int c = e / 32, r = e % 32;
        if (c < m && r < nr) cm[(long long)c * n + i0 + r] = tile[c][r];
    }
}

__device__ __forceinline__ bool finite_bits(double v)
{
    return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000;
}

// integer test: a comparison in FP64 takes the FP64 pipe as long as a product
__device__ __forceinline__ bool zero_bits(double v)
{
    return (((unsigned)__double2hiint(v) << 1) | (unsigned)__double2loint(v)) == 0;
}

// R = B - op(A) X (op = A or A^H; R = op(A) X when B is null), per-column
// squared norms of R added to nr and of B to nb.  A warp per group of NQ rows
// with one column list (the three rows u, v, w of a grid node; NQ = 1 for a
// general pattern): lane = (entry group, column), the 32 / NC entry groups
// taking every (32 / NC)-th entry.  Bound by the FP64 pipe (2 FMA per cycle
// and SM): a complex product is 4 FMAs, 2 where the matrix entry is real and
// none where it is zero - outside the absorbing layers of an elastic model the
// operator is real, 37 % of the entries at 40^3 with 10-node layers, and 8 %
// are zero.  Entries are only dropped next to finite X, so that infinities and
// NaNs spread as in the full product; the test is a warp's (with NC < 32 its
// lanes hold different entries).
template <int NC, int NQ>
__global__ void __launch_bounds__(256) k_residual(long long ngroups, const int *__restrict__ irptr,
                                                  const int *__restrict__ jcptr, const double2 *__restrict__ a,
                                                  const int *__restrict__ tpos, const double2 *__restrict__ X,
                                                  const double2 *__restrict__ B, double2 *__restrict__ R,
                                                  double *__restrict__ nr, double *__restrict__ nb, int adjoint)
{
    constexpr int G = 32 / NC;
    __shared__ double red[2][8][NC];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col = lane % NC, grp = lane / NC;
    const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    double sr = 0, sb = 0;
    for (long long g = w0; g < ngroups; g += nw) {
        const long long r0 = NQ * g;
        const int k0 = irptr[r0];
        const int len = irptr[r0 + 1] - k0;
        double2 acc[NQ];
#pragma unroll
        for (int q = 0; q < NQ; q++) acc[q] = make_double2(0, 0);
#pragma unroll 3
        for (int t0 = 0; t0 < len; t0 += G) {
            const int t = t0 + grp, k = k0 + t;
            const bool on = G == 1 || t < len;
            const double2 x = on ? X[(long long)jcptr[k] * NC + col] : make_double2(0, 0);
            const bool fin = __all_sync(0xffffffffu, finite_bits(x.x) && finite_bits(x.y));
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                double2 av = make_double2(0, 0);
                if (on) {
                    if (adjoint) { av = a[tpos[k + q * len]]; av.y = -av.y; }
                    else av = a[k + q * len];
                }
                const bool re = !fin || !__all_sync(0xffffffffu, zero_bits(av.x));
                const bool im = !fin || !__all_sync(0xffffffffu, zero_bits(av.y));
                if (im) {
                    acc[q].x = fma(-av.y, x.y, acc[q].x);
                    acc[q].y = fma(av.y, x.x, acc[q].y);
                }
                if (re) {
                    acc[q].x = fma(av.x, x.x, acc[q].x);
                    acc[q].y = fma(av.x, x.y, acc[q].y);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < NQ; q++) {
#pragma unroll
            for (int o = NC; o < 32; o <<= 1) {
                acc[q].x += __shfl_xor_sync(0xffffffffu, acc[q].x, o);
                acc[q].y += __shfl_xor_sync(0xffffffffu, acc[q].y, o);
            }
            if (grp == 0) {
                const double2 b = B ? B[(r0 + q) * NC + col] : make_double2(0, 0);
                const double2 r = B ? make_double2(b.x - acc[q].x, b.y - acc[q].y) : acc[q];
                R[(r0 + q) * NC + col] = r;
                sr += r.x * r.x + r.y * r.y;
                sb += b.x * b.x + b.y * b.y;
            }
        }
    }
    // one addition per block and column
    if (grp == 0) { red[0][warp][col] = sr; red[1][warp][col] = sb; }
    __syncthreads();
    if (threadIdx.x < 2 * NC) {
        const int h = threadIdx.x / NC, c = threadIdx.x % NC;
        double s = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) s += red[h][w][c];
        atomicAdd((h ? nb : nr) + c, s);
    }
}

// ---- batched Krylov kernels ------------------------------------------------
// Column c of every block is an independent system; reductions go through
// per-block partial sums and a second pass, so they do not depend on
// scheduling.  Grid strides are multiples of nc: a thread stays in its column.
constexpr int GM_KMAX = 16;      // longest restart of the flexible GMRES (per-call length: gmres_restart())
constexpr int GM_BLOCKS = 304;   // 2 blocks per SM for the reductions
constexpr int GM_CHUNK = 4;      // basis vectors per sweep over W

// Sum over the block's 256 threads of the values of equal column (tid % nc),
// returned to threads tid < nc.  red: 8 x 32 values.
__device__ __forceinline__ double block_column_sum(double v, int nc, double (*red)[32])
{
    for (int o = 16; o >= nc; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    red[warp][lane] = v;
    __syncthreads();
    double s = 0;
    if (threadIdx.x < nc)
        for (int w = 0; w < 8; w++) s += red[w][threadIdx.x];
    return s;
}

// part[i][b][c] = sum over the rows of block b of conj(V_i[row, c]) W[row, c], i < nv.
__global__ void __launch_bounds__(256) k_mdot(long long tot, int nc, int nv, const double2 *__restrict__ V,
                                              const double2 *__restrict__ W, double2 *__restrict__ part)
{
    __shared__ double red[8][32];
    const long long q0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    for (int i0 = 0; i0 < nv; i0 += GM_CHUNK) {
        double2 acc[GM_CHUNK];
#pragma unroll
        for (int j = 0; j < GM_CHUNK; j++) acc[j] = make_double2(0, 0);
        for (long long q = q0; q < tot; q += stride) {
            const double2 w = W[q];
#pragma unroll
            for (int j = 0; j < GM_CHUNK; j++) {
                if (i0 + j >= nv) break;
                const double2 v = V[(long long)(i0 + j) * tot + q];
                acc[j].x = fma(v.x, w.x, fma(v.y, w.y, acc[j].x));
                acc[j].y = fma(v.x, w.y, fma(-v.y, w.x, acc[j].y));
            }
        }
#pragma unroll
        for (int j = 0; j < GM_CHUNK; j++) {
            if (i0 + j >= nv) break;
            const double sx = block_column_sum(acc[j].x, nc, red), sy = block_column_sum(acc[j].y, nc, red);
            if (threadIdx.x < nc)
                part[((long long)(i0 + j) * gridDim.x + blockIdx.x) * nc + threadIdx.x] = make_double2(sx, sy);
        }
    }
}

// h[i][c] = sum_b part[i][b][c], one block per i (h's rows are MAXRHS apart)
__global__ void __launch_bounds__(256) k_mdot_reduce(int nblocks, int nc, const double2 *__restrict__ part,
                                                     double2 *__restrict__ h)
{
    __shared__ double red[8][32];
    double2 t = make_double2(0, 0);
    for (int q = threadIdx.x; q < nblocks * nc; q += 256) {
        const double2 v = part[(long long)blockIdx.x * nblocks * nc + q];
        t.x += v.x;
        t.y += v.y;
    }
    const double sx = block_column_sum(t.x, nc, red), sy = block_column_sum(t.y, nc, red);
    if (threadIdx.x < nc) h[blockIdx.x * MAXRHS + threadIdx.x] = make_double2(sx, sy);
}

// W[row, c] -= sum_{i < nv} coef[i][c] V_i[row, c]; with part != nullptr also
// part[b][c] = per-block sum of |W_new[row, c]|^2.  Bound by the FP64 pipe (two
// multiply-adds per cycle and SM): four explicit multiply-adds per entry, where a
// difference of products compiled to six operations (532 -> 394 us a call on average
// in a 48^3 solve with 32 columns).
__global__ void __launch_bounds__(256) k_maxpy(long long tot, int nc, int nv, const double2 *__restrict__ V,
                                               const double2 *__restrict__ coef, double2 *__restrict__ W,
                                               double *__restrict__ part)
{
    __shared__ double red[8][32];
    const long long q0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    const int c = (int)(q0 % nc);
    double2 cf[GM_KMAX + 1];
#pragma unroll
    for (int i = 0; i <= GM_KMAX; i++) cf[i] = i < nv ? coef[i * MAXRHS + c] : make_double2(0, 0);
    double s2 = 0;
    for (long long q = q0; q < tot; q += stride) {
        double2 w = W[q];
#pragma unroll
        for (int i = 0; i <= GM_KMAX; i++) {
            if (i >= nv) break;
            const double2 v = V[(long long)i * tot + q];
            w.x = fma(-cf[i].x, v.x, fma(cf[i].y, v.y, w.x));
            w.y = fma(-cf[i].x, v.y, fma(-cf[i].y, v.x, w.y));
        }
        W[q] = w;
        s2 = fma(w.x, w.x, fma(w.y, w.y, s2));
    }
    if (!part) return;
    const double s = block_column_sum(s2, nc, red);
    if (threadIdx.x < nc) part[(long long)blockIdx.x * nc + threadIdx.x] = s;
}

__global__ void __launch_bounds__(256) k_norm_reduce(int nblocks, int nc, const double *__restrict__ part,
                                                     double *__restrict__ out)
{
    __shared__ double red[8][32];
    double t = 0;
    for (int q = threadIdx.x; q < nblocks * nc; q += 256) t += part[q];
    const double s = block_column_sum(t, nc, red);
    if (threadIdx.x < nc) out[threadIdx.x] = s;
}

// W[row, c] = s[c] S[row, c] (S may be W)
__global__ void k_colscale(long long tot, int nc, const double *__restrict__ sc, const double2 *S, double2 *W)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= tot) return;
    const double f = sc[q % nc];
    const double2 v = S[q];
    W[q] = make_double2(v.x * f, v.y * f);
}

// ---- between the natural ordering and the engine's -------------------------
// Xs = S R (new ordering, engine precision); S the Jacobi scaling of the
// factor.  The pass's other two blocks are zeroed.
template <class T>
__global__ void k_gather_new(long long tot, int nc, const int *__restrict__ perm, const double *__restrict__ s,
                             const double2 *__restrict__ R, cx<T> *__restrict__ Xs, cx<T> *__restrict__ Zs,
                             cx<T> *__restrict__ Ys)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= tot) return;
    const long long o = perm[q / nc];
    const double2 v = R[o * nc + q % nc];
    const double w = s[o];
    Xs[q] = cx<T>((T)(v.x * w), (T)(v.y * w));
    Zs[q] = cx<T>(0);
    Ys[q] = cx<T>(0);
}

// Xn = S Ys or, with add, Xn += S Ys (natural ordering, FP64).
template <class T>
__global__ void k_scatter_nat(long long tot, int nc, const int *__restrict__ perm, const double *__restrict__ s,
                              const cx<T> *__restrict__ Ys, double2 *__restrict__ Xn, int add)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= tot) return;
    const cx<T> v = Ys[q];
    const long long o = perm[q / nc];
    const double w = s[o];
    double2 *d = Xn + o * nc + q % nc;
    const double2 x = add ? *d : make_double2(0, 0);
    *d = make_double2(x.x + (double)v.re * w, x.y + (double)v.im * w);
}

// Xn[row, c] -= sum_{i < nv} coef[i][c] S Z_i[row, c], Z_i the passes' results as
// the engine left them (new ordering, its precision: nothing is lost by keeping
// those instead of their FP64 copies, half the bytes for complex64).  The row's
// scale is applied to the sum, not to every Z_i: bound by the FP64 pipe, 1362 ->
// 829 us on 48^3 with 32 columns and 8 - 10 bases.
template <class T>
__global__ void __launch_bounds__(256) k_zaxpy(long long tot, int nc, int nv, const int *__restrict__ perm,
                                               const double *__restrict__ s, const cx<T> *__restrict__ Z,
                                               const double2 *__restrict__ coef, double2 *__restrict__ Xn)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= tot) return;
    const long long o = perm[q / nc];
    const int c = (int)(q % nc);
    const double w = s[o];
    double2 *d = Xn + o * nc + c, x = *d, y = make_double2(0, 0);
    for (int i = 0; i < nv; i++) {
        const double2 cf = coef[i * MAXRHS + c];
        const cx<T> z = Z[(long long)i * tot + q];
        const double zx = z.re, zy = z.im;
        y.x = fma(cf.x, zx, fma(-cf.y, zy, y.x));
        y.y = fma(cf.x, zy, fma(cf.y, zx, y.y));
    }
    *d = make_double2(fma(-w, y.x, x.x), fma(-w, y.y, x.y));
}

}  // namespace wt3d
