// Multifrontal numeric kernels (templated on the real type T: float for the
// complex64 mixed-precision path, double for the complex128 oracle path).
//
// Front layout (row-major): the pivot rows P = F[0:p, 0:nf] (p x nf) are
// followed by the lower-left border block Lo = F[p:nf, 0:p] (b x p) in the
// factor pool; the Schur/update block F22 (b x b) lives in one of two
// level-parity update buffers.  Factorisation is right-looking blocked LU on
// the first p columns with KB-wide panels and partial pivoting restricted to
// the diagonal KB x KB tile; a panel's row order (gord) applies to the columns
// right of the panel only, and the substitutions' block inverses take it in.
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
struct EATask { int front, child0, child1; long long pos0, pos1; };   // children -1: none
struct EAUnit { int task, row0; };
template <class T>
struct GemmTask {
    const cx<T> *A;
    const cx<T> *B;
    cx<T> *C;
    int lda, ldb, ldc, M, N, K;
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
// extend-add: the children's update matrices into a front, gathered by the front's
// rows (one warp per row)
// ---------------------------------------------------------------------------
// Bound by memory traffic.  Each entry of the front's own update block F22 is
// written once, as the sum of what its children have there (pos: the front's row or
// column of each child's border, inverted; -1 where the child has none); adding one
// child after the other into a zeroed block read and wrote it twice more and took
// two launches and a memset per level (64x64x48: 30 ms of a factorisation).
constexpr int EA_ROWS = 8;   // rows per CTA
template <class T>
__global__ void __launch_bounds__(32 * EA_ROWS) k_extend_add(const EATask *__restrict__ tasks,
                                                             const EAUnit *__restrict__ units,
                                                             const FrontDev *__restrict__ fr,
                                                             const int *__restrict__ pos, cx<T> *__restrict__ fac,
                                                             cx<T> *__restrict__ upd0, cx<T> *__restrict__ upd1)
{
    const EAUnit u = units[blockIdx.x];
    const EATask t = tasks[u.task];
    const FrontDev P = fr[t.front];
    const int nf = P.p + P.b, R = u.row0 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (R >= nf) return;
    const int *m0 = pos + t.pos0, *m1 = pos + t.pos1;
    const int i0 = t.child0 >= 0 ? m0[R] : -1, i1 = t.child1 >= 0 ? m1[R] : -1;
    if (i0 < 0 && i1 < 0 && R < P.p) return;
    const cx<T> *s0 = nullptr, *s1 = nullptr;   // the children's rows
    if (i0 >= 0) {
        const FrontDev C = fr[t.child0];
        s0 = (C.parity ? upd1 : upd0) + C.upd + (long long)i0 * C.b;
    }
    if (i1 >= 0) {
        const FrontDev C = fr[t.child1];
        s1 = (C.parity ? upd1 : upd0) + C.upd + (long long)i1 * C.b;
    }
    auto sum = [&](int c, bool &any) {
        const int j0 = s0 ? m0[c] : -1, j1 = s1 ? m1[c] : -1;
        any = j0 >= 0 || j1 >= 0;
        cx<T> v = j0 >= 0 ? s0[j0] : cx<T>(0);
        if (j1 >= 0) v = v + s1[j1];
        return v;
    };
    // the factor part: columns of the pivot rows, pivot columns of the border rows
    cx<T> *row = fac + P.fac + (R < P.p ? (long long)R * nf : (long long)P.p * nf + (long long)(R - P.p) * P.p);
    const int w = R < P.p ? nf : P.p;
    if (s0 || s1) {
#pragma unroll 4
        for (int c = lane; c < w; c += 32) {
            bool any;
            const cx<T> v = sum(c, any);
            if (any) row[c] = row[c] + v;
        }
    }
    if (R < P.p) return;
    cx<T> *p22 = (P.parity ? upd1 : upd0) + P.upd + (long long)(R - P.p) * P.b;
#pragma unroll 4
    for (int c = lane; c < P.b; c += 32) {
        bool any;
        p22[c] = sum(P.p + c, any);
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

// 1 / d for |d|^2 = m2 far from overflow and underflow (panel_group's bounds): conj(d)
// times a hardware approximation of 1 / m2 (with one Newton step for its 20 bits in
// FP64), then one step of Newton's iteration z (2 - d z), which leaves it more
// accurate than the scaled division, without its branches and divisions (a panel
// takes 26 us with it, 34 us with cdiv).
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double rcp_approx(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return fma(r, fma(-x, r, 1.0), r);
}
template <class T>
__device__ __forceinline__ cx<T> cinv_fast(const cx<T> d, T m2)
{
    const T r = rcp_approx(m2);
    const cx<T> z(d.re * r, -d.im * r);
    const cx<T> e(fma(-d.re, z.re, fma(d.im, z.im, T(1))), -fma(d.re, z.im, d.im * z.re));
    return cx<T>(fma(z.re, e.re, fma(-z.im, e.im, z.re)), fma(z.re, e.im, fma(z.im, e.re, z.im)));
}

// PG columns of a panel in one warp, which holds two rows per lane (rows lane and
// lane + 32; used: chosen before).  piv[jj] is the row that column jj chose.
// FAST: straight-line code, so that the next column's pivot search overlaps the
// update of the columns behind it; it returns false, with nothing to keep, when a
// pivot is below the threshold or its square near overflow or underflow, and the
// other form (branches for those cases, and for a narrower last group) has to do
// the group.
template <class T, int PG, bool FAST>
__device__ __forceinline__ bool panel_group(cx<T> (&x0)[PG], cx<T> (&x1)[PG], bool &used0, bool &used1, int nc,
                                            T thresh, int lane, int (&piv)[PG], int &npert)
{
    constexpr T big = sizeof(T) == 4 ? T(1e30) : T(1e250);
    bool good = true;
#pragma unroll
    for (int jj = 0; jj < PG; jj++) {
        if (!FAST && jj >= nc) break;
        const auto k0 = pivot_key(cabs2(x0[jj])), k1 = pivot_key(cabs2(x1[jj]));
        auto key = used0 ? decltype(k0)(0) : k0;
        if (!used1 && k1 > key) key = k1;
        const auto best = warp_max(key);
        const unsigned b0 = __ballot_sync(0xffffffffu, !used0 && k0 == best);
        const unsigned b1 = __ballot_sync(0xffffffffu, !used1 && k1 == best);
        const bool up = b0 == 0;   // the pivot is in rows 32 - 63
        const int src = __ffs(up ? b1 : b0) - 1;
        cx<T> u[PG];               // the pivot row
#pragma unroll
        for (int c = jj; c < PG; c++) {
            const cx<T> v(up ? x1[c].re : x0[c].re, up ? x1[c].im : x0[c].im);
            u[c] = cx<T>(__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src));
        }
        piv[jj] = src + (up ? 32 : 0);
        used0 |= lane == src && !up;
        used1 |= lane == src && up;
        cx<T> d = u[jj], inv;
        T m2 = cabs2(d);
        if constexpr (FAST) {
            good = good && m2 >= thresh * thresh && m2 < big && m2 > T(1) / big;
            inv = cinv_fast(d, m2);
        } else {
            if (!(m2 >= thresh * thresh)) {   // also catches NaN
                const T m = sqrt(m2);
                d = (m > 0 && m == m) ? d * (thresh / m) : cx<T>(thresh);
                npert++;
                if (lane == src) {
                    if (up) x1[jj] = d;
                    else x0[jj] = d;
                }
            }
            inv = cdiv(cx<T>(1), d);
        }
        // multipliers; zero for chosen rows, which stay as they are
        const cx<T> l0 = used0 ? cx<T>(0) : x0[jj] * inv, l1 = used1 ? cx<T>(0) : x1[jj] * inv;
        if (!used0) x0[jj] = l0;
        if (!used1) x1[jj] = l1;
#pragma unroll
        for (int c = jj + 1; c < PG; c++) {
            cfms(x0[c], l0, u[c]);
            cfms(x1[c], l1, u[c]);
        }
    }
    return good;
}

// One CTA per tile: a chain of 64 dependent columns, so the latency of a column
// is what counts.  The columns are taken in groups of PG: warp 0 holds the
// group's 64 rows in registers, finds every pivot with a warp reduction and
// broadcasts the pivot row with shuffles - no barrier inside a group; then all
// threads update the columns to the right with the group's PG rank-one products
// at once.  Rows stay where they are: a chosen row is marked, and rows are stored
// in the order they were chosen in (gord).  Equal magnitudes: the smallest stored
// row.  A launch of few tiles took 55 - 80 us with the tile and its row swaps in
// shared memory, 42 us with the tile in the registers of 256 threads and two
// barriers per column, and takes 26 us.
// Columns per group.  complex128: warp 0 has a quarter of the SM's FP64 rate and is
// what bounds the panel, so narrower groups leave more of the work to all warps (348 us
// with groups of 8 and scaled divisions, 237 us with groups of 4, 217 us with 2).
template <class T> constexpr int panel_group_cols = sizeof(T) == 4 ? 8 : 2;
constexpr int PLD = KB + 2;   // row stride: 16-byte-aligned rows
template <class T> constexpr size_t panel_smem() { return sizeof(cx<T>) * KB * PLD; }

template <class T>
__global__ void __launch_bounds__(256, 1) k_panel(const PanelTask *__restrict__ tasks,
                                                  const FrontDev *__restrict__ fr, cx<T> *__restrict__ fac,
                                                  const unsigned long long *__restrict__ amax2, double pivot_rel,
                                                  int *__restrict__ npert, int *__restrict__ gord)
{
    // static-pivot threshold: pivot_rel * max |a_ij| of the assembled operator
    const T thresh = (T)(pivot_rel * sqrt(__longlong_as_double((long long)*amax2)));
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *S = reinterpret_cast<cx<T> *>(smraw);   // KB x PLD
    constexpr int PG = panel_group_cols<T>;
    __shared__ int spiv[2][PG], pos[KB];           // two sets: a group's is read while the next is found
    __shared__ unsigned s_used[2];                 // rows chosen so far: bits of rows 0-31, 32-63
    const PanelTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    cx<T> *D = fac + F.fac + (long long)k * nf + k;
    const int tid = threadIdx.x, lane = tid & 31;
    for (int q = tid; q < KB * KB; q += 256) {
        const int i = q / KB, j = q % KB;
        if (i < kb && j < kb) cp_async_cx(S + i * PLD + j, D + (long long)i * nf + j);
        else S[i * PLD + j] = cx<T>(0);
    }
    bool used0 = lane >= kb, used1 = lane + 32 >= kb;   // warp 0: this lane's rows lane and lane + 32
    cp_async_wait_all();
    __syncthreads();
    const int ng = (kb + PG - 1) / PG;
    for (int G = 0; G < ng; G++) {
        const int j0 = PG * G;
        int *piv = spiv[G & 1];
        if (tid < 32) {
            const bool w0 = !used0, w1 = !used1;   // rows this group may change
            cx<T> x0[PG], x1[PG];
            int pv[PG], np = 0;
            auto fetch = [&]() {
#pragma unroll
                for (int c = 0; c < PG; c++) x0[c] = x1[c] = cx<T>(0);
                if (w0) lds_cx<PG>(S + lane * PLD + j0, x0);
                if (w1) lds_cx<PG>(S + (lane + 32) * PLD + j0, x1);
            };
            fetch();
            const int nc = min(PG, kb - j0);
            if (nc < PG || !panel_group<T, PG, true>(x0, x1, used0, used1, nc, thresh, lane, pv, np)) {
                used0 = !w0;
                used1 = !w1;
                fetch();
                panel_group<T, PG, false>(x0, x1, used0, used1, nc, thresh, lane, pv, np);
                if (lane == 0 && np) atomicAdd(npert, np);
            }
            if (lane == 0) {
#pragma unroll
                for (int jj = 0; jj < PG; jj++)
                    if (jj < nc) {
                        piv[jj] = pv[jj];
                        pos[pv[jj]] = j0 + jj;
                    }
            }
#pragma unroll
            for (int c = 0; c < PG; c++) {
                if (w0) S[lane * PLD + j0 + c] = x0[c];
                if (w1) S[(lane + 32) * PLD + j0 + c] = x1[c];
            }
            const unsigned m0 = __ballot_sync(0xffffffffu, used0), m1 = __ballot_sync(0xffffffffu, used1);
            if (lane == 0) { s_used[0] = m0; s_used[1] = m1; }
        }
        __syncthreads();
        if (G + 1 == ng) break;
        // columns right of the group (all PG pivots exist: kb > j0 + PG): thread
        // (column, quarter of the rows)
        const int c = tid & (KB - 1), r0 = (tid >> 6) * (KB / 4);
        const bool on = c >= j0 + PG && c < kb;
        cx<T> u[PG];
        if (on) {
#pragma unroll
            for (int q = 0; q < PG; q++) {
                const cx<T> *row = S + piv[q] * PLD;
                u[q] = row[c];
#pragma unroll
                for (int l = 0; l < q; l++) cfms(u[q], row[j0 + l], u[l]);
            }
            const unsigned used = s_used[r0 >> 5] >> (r0 & 31);
#pragma unroll 2
            for (int i = 0; i < KB / 4; i++) {
                if ((used >> i) & 1u) continue;
                cx<T> *row = S + (r0 + i) * PLD, a = row[c], l[PG];
                lds_cx<PG>(row + j0, l);
#pragma unroll
                for (int q = 0; q < PG; q++) cfms(a, l[q], u[q]);
                row[c] = a;
            }
        }
        __syncthreads();
        // the pivot rows' part of U: nobody reads it before the tile is stored
        if (on && r0 == 0) {
#pragma unroll
            for (int q = 0; q < PG; q++) S[piv[q] * PLD + c] = u[q];
        }
    }
    __syncthreads();
    for (int q = tid; q < kb * KB; q += 256) {
        const int i = q / KB, j = q % KB;
        if (j < kb) D[(long long)pos[i] * nf + j] = S[i * PLD + j];
    }
    if (tid < kb) gord[F.first + k + pos[tid]] = F.first + k + tid;
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
// NV vectors per four threads: with two, a row of the tile is read from shared
// memory once for both; a launch of many vectors is bound by those reads, one of
// few by the chain, which is shorter with one.
constexpr int BD_TH = 128;
template <class T, int NV>
struct BandCfg {
    static constexpr int V = BD_TH / 4 * NV;                // vectors per CTA
    static constexpr int TG = sizeof(T) == 4 ? 8 : 4;       // unknowns per group
    static constexpr int LDT = KB + 16 / (int)sizeof(cx<T>);   // tile rows on 16 bytes, four rows on different banks
    static constexpr int LDX = V + (sizeof(T) == 4 ? 4 : 2);
    static constexpr size_t smem = sizeof(cx<T>) * (KB * LDT + KB * LDX);
};

// T x = b for the vectors of X (b on entry, zero before group first / TG); unit:
// T's diagonal is one, otherwise invd holds its inverse.  Vector e of a quad is
// vector quad + 32 e.
template <class T, int NV>
__device__ __forceinline__ void band_solve(const cx<T> *Tm, cx<T> *X, const cx<T> *invd, bool unit, int first, int kb)
{
    using C = BandCfg<T, NV>;
    constexpr int TG = C::TG, LDT = C::LDT, LDX = C::LDX;
    const int q4 = threadIdx.x & 3, ng = (kb + TG - 1) / TG;
    cx<T> *x = X + (threadIdx.x >> 2);
#pragma unroll 1
    for (int G = first / TG; G < ng; G++) {
        cx<T> b[NV][TG];
#pragma unroll
        for (int e = 0; e < NV; e++)
#pragma unroll
            for (int i = 0; i < TG; i++) b[e][i] = x[(TG * G + i) * LDX + 32 * e];
#pragma unroll
        for (int i = 0; i < TG; i++) {
            if (i > 0) {
                cx<T> lr[TG];
                lds_cx<TG>(Tm + (TG * G + i) * LDT + TG * G, lr);
#pragma unroll
                for (int e = 0; e < NV; e++)
#pragma unroll
                    for (int l = 0; l < i; l++) cfms(b[e][i], lr[l], b[e][l]);
            }
            if (!unit) {
                const cx<T> d = invd[TG * G + i];
#pragma unroll
                for (int e = 0; e < NV; e++) b[e][i] = b[e][i] * d;
            }
        }
        __syncwarp();   // the four threads have read the group
#pragma unroll
        for (int e = 0; e < NV; e++)
#pragma unroll
            for (int i = 0; i < TG; i++)
                if ((i & 3) == q4) x[(TG * G + i) * LDX + 32 * e] = b[e][i];
#pragma unroll 1
        for (int H = TG * (G + 1) + q4; H < TG * ng; H += TG) {
#pragma unroll
            for (int i = 0; i < TG; i += 4) {
                cx<T> lr[TG], c[NV];
#pragma unroll
                for (int e = 0; e < NV; e++) c[e] = x[(H + i) * LDX + 32 * e];
                lds_cx<TG>(Tm + (H + i) * LDT + TG * G, lr);
#pragma unroll
                for (int l = 0; l < TG; l++)
#pragma unroll
                    for (int e = 0; e < NV; e++) cfms(c[e], lr[l], b[e][l]);
#pragma unroll
                for (int e = 0; e < NV; e++) x[(H + i) * LDX + 32 * e] = c[e];
            }
        }
        __syncwarp();
    }
}

template <class T, int NV>
__global__ void __launch_bounds__(BD_TH) k_bands(const BandTask *__restrict__ tasks, const FrontDev *__restrict__ fr,
                                                 cx<T> *__restrict__ fac, const int *__restrict__ gord)
{
    using C = BandCfg<T, NV>;
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
        nv = min(C::V, nf - t.c0);
        if (tid < KB) idx[tid] = tid < kb ? gord[F.first + k + tid] - F.first - k : 0;
        __syncthreads();
        for (int q = tid; q < KB * C::V; q += BD_TH) {
            const int i = q / C::V, v = q % C::V;
            if (i < kb && v < nv) cp_async_cx(X + i * LDX + v, xb + idx[i] * si + v);
            else X[i * LDX + v] = cx<T>(0);
        }
    } else {
        if (t.which == 1) {
            xb = fac + F.fac + (long long)t.c0 * nf + k;
            sv = nf;
            nv = min(C::V, F.p - t.c0);
        } else {
            xb = fac + F.fac + (long long)F.p * nf + (long long)t.c0 * F.p + k;
            sv = F.p;
            nv = min(C::V, F.b - t.c0);
        }
        si = 1;
        for (int q = tid; q < KB * C::V; q += BD_TH) {
            const int i = q % KB, v = q / KB;
            if (i < kb && v < nv) cp_async_cx(X + i * LDX + v, xb + v * sv + i);
            else X[i * LDX + v] = cx<T>(0);
        }
    }
    cp_async_wait_all();
    __syncthreads();
    if (tid < KB) invd[tid] = row ? cx<T>(1) : cdiv(cx<T>(1), Tm[tid * LDT + tid]);
    __syncthreads();
    band_solve<T, NV>(Tm, X, invd, row, 0, kb);
    __syncthreads();
    for (int q = tid; q < KB * C::V; q += BD_TH) {
        const int i = row ? q / C::V : q % KB, w = row ? q % C::V : q / KB;
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
