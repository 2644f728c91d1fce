// Kernels of the substitution passes: explicit inverses of the diagonal blocks
// of every front, computed once per factorisation, and the skinny products the
// passes consist of (block inverse times right-hand sides, and the updates of
// the rows outside a block).
//
// A front's pivot block is cut into diagonal blocks of up to SB columns.  With
// the inverses of the block's triangular factors at hand, a substitution step
// over SB unknowns is one product instead of SB / KB dependent ones.  The
// length of the dependent chain is what bounds a pass on all but the largest
// grids, not its bytes: a 40^3 pass was 364 dependent 64-wide steps of 18 us,
// against 0.5 ms to read the factors at the memory rate.
#pragma once
#include "mf_kernels.cuh"

namespace wt3d {

// Start of a kernel that is launched as a programmatic dependent of the one before
// it: the next kernel may be set up from here on; after the wait everything before
// this kernel is complete and visible.
__device__ __forceinline__ void chain_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// d += a b and d += conj(a) b as four fused multiply-adds
template <class T>
__device__ __forceinline__ void cmac(cx<T> &d, const cx<T> a, const cx<T> b)
{
    d.re = fma(a.re, b.re, fma(-a.im, b.im, d.re));
    d.im = fma(a.re, b.im, fma(a.im, b.re, d.im));
}
template <class T>
__device__ __forceinline__ void cmac_conj(cx<T> &d, const cx<T> a, const cx<T> b)
{
    d.re = fma(a.re, b.re, fma(a.im, b.im, d.re));
    d.im = fma(a.re, b.im, fma(-a.im, b.re, d.im));
}

// ---------------------------------------------------------------------------
// block inverses
// ---------------------------------------------------------------------------
// Columns per diagonal block of the substitutions (a multiple of KB).  Longer blocks
// make shorter chains; their inverses cost more.  complex64: 128, 256 and 512 give
// passes of 14.5, 11.9 and 11.0 ms on 48^3 with 32 columns.  complex128: the inverses
// are bound by the FP64 pipe, and those of 512 took 10 ms of the 41 ms of kernel
// time of a 16x15x14 factorisation.
template <class T> constexpr int SB = sizeof(T) == 4 ? 512 : 256;

// Row stride of a block inverse of w columns (even: rows start on 16 bytes).
__host__ __device__ __forceinline__ int inv_ld(int w) { return (w + 1) & ~1; }

// Entries of all block inverses of a front with p pivots.
template <class T>
inline long long inv_entries(int p)
{
    const int full = p / SB<T>, rest = p % SB<T>;
    return (long long)full * SB<T> * inv_ld(SB<T>) + (long long)rest * inv_ld(rest);
}

// The inverse of block c0 of a front is stored packed, row-major: the upper
// triangle with the diagonal holds U^-1, the strict lower triangle L^-1 (unit
// diagonal).  L is the block's lower factor with the rows of every KB-wide
// panel in the order its interchanges leave them in, so that the forward
// substitution of the block is z = L^-1 y[gord].
//
// Diagonal KB x KB tiles first, with the bands' solver on unit vectors: four CTAs
// per tile, 32 columns of L_D^-1 (parts 0, 1) or 32 rows of U_D^-1 (parts 2, 3)
// each.  A tile is final once its panel step is done (later steps change only
// rows and columns to its right and below).  One thread per column, with a
// complex division per entry of U_D^-1, took 4.7 ms for the 16x15x14 tiles in
// complex128.
template <class T>
__global__ void __launch_bounds__(BD_TH) k_tile_inverse(const PanelTask *__restrict__ tasks,
                                                        const FrontDev *__restrict__ fr,
                                                        const cx<T> *__restrict__ fac, const int *__restrict__ gord,
                                                        int *__restrict__ ipiv, cx<T> *__restrict__ inv)
{
    using C = BandCfg<T, 1>;
    constexpr int LDT = C::LDT, LDX = C::LDX;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *Tm = reinterpret_cast<cx<T> *>(smraw);
    cx<T> *X = Tm + KB * LDT;
    __shared__ cx<T> invd[KB];
    const PanelTask t = tasks[blockIdx.x >> 2];
    const int part = blockIdx.x & 3, v0 = C::V * (part & 1);
    const bool row = part < 2;
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, k = t.k, kb = min(KB, F.p - k);
    const cx<T> *D = fac + F.fac + (long long)k * nf + k;
    const int tid = threadIdx.x;
    if (part == 0) {
        // the tile's row order as a sequence of interchanges (checks read it): at
        // step j the row that ends at position j is at position where[row]
        __shared__ int at[KB], where[KB];
        if (tid < KB) at[tid] = where[tid] = tid;
        __syncthreads();
        if (tid == 0)
            for (int j = 0; j < kb; j++) {
                const int r = gord[F.first + k + j] - F.first - k, q = where[r], o = at[j];
                ipiv[F.first + k + j] = k + q;
                at[q] = o;
                where[o] = q;
            }
    }
    if (v0 >= kb) return;
    for (int q = tid; q < KB * KB; q += BD_TH) {
        const int i = q / KB, j = q % KB;
        cx<T> *dst = row ? Tm + i * LDT + j : Tm + j * LDT + i;
        if (i < kb && j < kb) cp_async_cx(dst, D + (long long)i * nf + j);
        else *dst = cx<T>(i == j ? T(1) : T(0));
    }
    for (int q = tid; q < KB * C::V; q += BD_TH) {
        const int i = q / C::V, v = q % C::V;
        X[i * LDX + v] = cx<T>(i == v0 + v ? T(1) : T(0));
    }
    cp_async_wait_all();
    __syncthreads();
    if (tid < KB) invd[tid] = row ? cx<T>(1) : cdiv(cx<T>(1), Tm[tid * LDT + tid]);
    __syncthreads();
    band_solve<T, 1>(Tm, X, invd, row, v0, kb);
    __syncthreads();
    const int c0 = k / SB<T> * SB<T>, w = min(SB<T>, F.p - c0), ldw = inv_ld(w), o = k - c0;
    cx<T> *W = inv + F.inv + (long long)(c0 / SB<T>) * (SB<T> * SB<T>) + (long long)o * ldw + o;
    for (int q = tid; q < KB * C::V; q += BD_TH) {
        const int i = row ? q / C::V : q % KB, v = row ? q % C::V : q / KB, e = v0 + v;
        if (i >= kb || e >= kb) continue;
        if (row) { if (i > e) W[(long long)i * ldw + e] = X[i * LDX + v]; }
        else if (i >= e) W[(long long)e * ldw + i] = X[i * LDX + v];
    }
}

// The off-diagonal tiles, by columns: one CTA per 32 columns (h: the first or
// second half of tile column t) of one triangle of one block.  For L, from the
// tile below the diagonal down: X_s = -L_ss^-1 sum_{u=t}^{s-1} L_su X_u; for
// U, from the tile above the diagonal up: X_s = -U_ss^-1 sum_{u>s} U_su X_u.
// A CTA reads only tiles that it wrote itself, and the diagonal ones.  FP32
// (FP64) sums as in the substitutions themselves.
struct InvTask { int f, c0, t, h, upper; };
constexpr int IV_TH = 128, IV_BK = 16, IV_N = 32;

template <class T>
__global__ void __launch_bounds__(IV_TH) k_block_inverse(const InvTask *__restrict__ tasks,
                                                         const FrontDev *__restrict__ fr,
                                                         const cx<T> *__restrict__ fac, const int *__restrict__ gord,
                                                         cx<T> *__restrict__ inv)
{
    __shared__ cx<T> As[KB][IV_BK + 1];
    __shared__ cx<T> Bs[IV_BK][IV_N];
    __shared__ cx<T> Ss[KB][IV_N];
    __shared__ int rows[KB];
    const InvTask t = tasks[blockIdx.x];
    const FrontDev F = fr[t.f];
    const int nf = F.p + F.b, w = min(SB<T>, F.p - t.c0), ldw = inv_ld(w), nt = (w + KB - 1) / KB;
    const cx<T> *D = fac + F.fac + (long long)t.c0 * nf + t.c0;   // the block's factors
    cx<T> *W = inv + F.inv + (long long)(t.c0 / SB<T>) * (SB<T> * SB<T>);
    const bool up = t.upper != 0;
    const int col0 = KB * t.t + IV_N * t.h;
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;   // rows ty + 16 i, columns 4 tx + j
    constexpr int NA = KB * IV_BK / IV_TH, NB = IV_BK * IV_N / IV_TH;
    cx<T> pa[NA], pb[NB], acc[4][4];
    for (int s = up ? t.t - 1 : t.t + 1; up ? s >= 0 : s < nt; s += up ? -1 : 1) {
        const int r0 = KB * s, mr = min(KB, w - r0);
        const int k0 = up ? KB * (s + 1) : KB * t.t, k1 = up ? min(w, KB * (t.t + 1)) : r0;
        if (tid < KB) rows[tid] = !up && tid < mr ? gord[F.first + t.c0 + r0 + tid] - F.first - t.c0 : r0 + tid;
        __syncthreads();   // also: the tile stored last is visible to the whole CTA
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = cx<T>(0);
        // phase 0: S = (factor tiles) X; phase 1: X_s = -(tile inverse) S
        for (int phase = 0; phase < 2; phase++) {
            const int ka = phase ? r0 : k0, kz = phase ? r0 + mr : k1;
            auto load = [&](int kk0) {
#pragma unroll
                for (int q = 0; q < NA; q++) {
                    const int idx = tid + q * IV_TH, i = idx / IV_BK, k = kk0 + idx % IV_BK;
                    cx<T> v(0);
                    if (i < mr && k < kz) {
                        if (!phase) v = D[(long long)rows[i] * nf + k];
                        else if (up ? k >= r0 + i : k < r0 + i) v = W[(long long)(r0 + i) * ldw + k];
                        else if (!up && k == r0 + i) v = cx<T>(1);
                    }
                    pa[q] = v;
                }
                if (!phase) {
#pragma unroll
                    for (int q = 0; q < NB; q++) {
                        const int idx = tid + q * IV_TH, k = kk0 + idx / IV_N, c = col0 + idx % IV_N;
                        cx<T> v(0);
                        if (k < kz && c < w) {
                            if (up ? k <= c : k > c) v = W[(long long)k * ldw + c];
                            else if (!up && k == c) v = cx<T>(1);
                        }
                        pb[q] = v;
                    }
                }
            };
            load(ka);
            for (int kk0 = ka; kk0 < kz; kk0 += IV_BK) {
#pragma unroll
                for (int q = 0; q < NA; q++) {
                    const int idx = tid + q * IV_TH;
                    As[idx / IV_BK][idx % IV_BK] = pa[q];
                }
                if (!phase) {
#pragma unroll
                    for (int q = 0; q < NB; q++) {
                        const int idx = tid + q * IV_TH;
                        Bs[idx / IV_N][idx % IV_N] = pb[q];
                    }
                }
                __syncthreads();
                if (kk0 + IV_BK < kz) load(kk0 + IV_BK);
                const cx<T>(*B)[IV_N] = phase ? Ss + (kk0 - r0) : Bs;
#pragma unroll
                for (int kk = 0; kk < IV_BK; kk++) {
                    cx<T> a[4], b[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) a[i] = As[ty + 16 * i][kk];
#pragma unroll
                    for (int j = 0; j < 4; j++) b[j] = B[kk][4 * tx + j];
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++) cmac(acc[i][j], a[i], b[j]);
                }
                __syncthreads();
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int r = ty + 16 * i, c = col0 + 4 * tx + j;
                    if (!phase) Ss[r][4 * tx + j] = acc[i][j];
                    else if (r < mr && c < w) W[(long long)(r0 + r) * ldw + c] = -acc[i][j];
                    acc[i][j] = cx<T>(0);
                }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// skinny products  out (=, +=, -=) op(A) in  over NC right-hand sides
// ---------------------------------------------------------------------------
// One unit per CTA: up to SK_M output rows and up to SK_KMAX input rows of a
// factor block or a block inverse.  Blocks are cut along K so that every
// launch has a few units per SM: a single 64 x 512 unit of 32 columns would
// keep one SM busy for 17 us while the others idle.  Units of one task then
// add up atomically.
struct SkUnit {
    const void *A;     // op = A: tile element (0, 0), rows lda apart; op = A^H: stored row 0, column 0
    const int *bmap;   // input row of k: bmap[k], or b0 + k
    const int *cmap;   // output row of i: cmap[i], or c0 + i
    int b0, c0, lda, M, K;
    int flags;
    int d;             // triangles: first k of the unit minus its first row
};
enum { SK_LOWER = 1, SK_UPPER = 2, SK_SUB = 4, SK_ATOM = 8 };
constexpr int SK_M = 64, SK_TH = 128, SK_KMAX = 1024;

// Right-hand-side blocks are stored [row][NC]: NC is the smallest of these that
// holds the pass's columns, so that one source does not pay for 32.
inline int sk_columns(int m) { return m <= 1 ? 1 : m <= 4 ? 4 : m <= 8 ? 8 : m <= 16 ? 16 : 32; }

// Products that go to the tensor cores (skinny_tc.cu), by width and K per unit.  At 8
// columns a launch of units shorter than 128 k is faster on the FP32 pipe: a pass of
// 24x22x20 took 0.55 ms with it, 0.65 ms on the tensor cores; one of 64x64x48 takes 7.1
// and 6.6 ms.  At 16 and 32 columns the tensor cores win at every size measured, FP32 and
// they in ms per pass: 24x22x20 0.68 and 0.58, 0.86 and 0.75; 40^3 3.2 and 2.5, 4.4 and
// 3.7; 64x64x48 10.5 and 8.0, 15.4 and 12.4.
inline bool sk_tensor(int nc, int chunk) { return nc > 8 || (nc == 8 && chunk >= 128); }
void sk_tensor_launch(int nc, bool herm, const SkUnit *u, int n, const cx<float> *in, cx<float> *out, cudaStream_t st);

// Stage depth along K, and stages: 40 KB per CTA at 32 columns.
template <class T, int NC>
struct SkCfg {
    static constexpr int BK = (NC >= 32 ? 16 : 32) / (sizeof(T) / 4);
    static constexpr int NS = 3;
    static constexpr int VK = 16 / (int)sizeof(cx<T>);              // complex per 16 bytes
    static constexpr int lda(bool h) { return h ? SK_M + VK : BK + VK; }
    static constexpr int a_elems(bool h) { return (h ? BK : SK_M) * lda(h); }
    static constexpr int b_elems() { return (BK * NC + 1) / 2 * 2; }
    static constexpr size_t stage(bool h) { return sizeof(cx<T>) * (a_elems(h) + b_elems()); }
    static constexpr size_t smem(bool h) { return NS * stage(h) + sizeof(int) * (SK_KMAX + SK_M); }
};

__device__ __forceinline__ void cp_async_16_z(void *dst, const void *src, bool ok)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

__device__ __forceinline__ void red_add(cx<float> *p, const cx<float> v)
{
    atomicAdd(reinterpret_cast<float2 *>(p), make_float2(v.re, v.im));
}
__device__ __forceinline__ void red_add(cx<double> *p, const cx<double> v)
{
    atomicAdd(&p->re, v.re);
    atomicAdd(&p->im, v.im);
}

// 128 threads in KG groups of 16 x TX: a group sums every KG-th k of a stage
// for the whole 64 x NC tile, 4 rows x CT columns per thread (32 FP32
// accumulators; narrower blocks have more groups, so that every thread works
// at any NC).  A and the right-hand sides go through a ring of three
// asynchronous-copy stages.  Launched as a programmatic dependent of the
// previous product: the factor entries, which no product writes, are on their
// way before the wait for it.  One pass, against KB-wide steps and 128 x 32
// products that computed 32 columns whatever the pass held: 40^3 with 1 column
// 11.4 -> 2.0 ms, with 32 columns 12.4 -> 4.4 ms (3.7 ms on the tensor cores),
// complex128 16x15x14 with 4 columns 23 -> 1.1 ms.
template <class T, int NC, bool H>
__global__ void __launch_bounds__(SK_TH) k_skinny(const SkUnit *__restrict__ units, const cx<T> *__restrict__ in,
                                                  cx<T> *__restrict__ out)
{
    chain_start();
    using C = SkCfg<T, NC>;
    constexpr int BK = C::BK, NS = C::NS, VK = C::VK, LDA = C::lda(H), AE = C::a_elems(H), BE = C::b_elems();
    constexpr int CT = NC < 4 ? NC : 4, TX = NC / CT, TPG = 16 * TX, KG = SK_TH / TPG;
    static_assert(KG <= BK / VK && KG * SK_M * NC <= NS * (AE + BE), "groups per stage; the sums fit the ring");
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *As = reinterpret_cast<cx<T> *>(smraw), *Bs = As + NS * AE;
    int *brow = reinterpret_cast<int *>(Bs + NS * BE), *crow = brow + SK_KMAX;
    const SkUnit u = units[blockIdx.x];
    const int tid = threadIdx.x, K = u.K, M = u.M;
    const int g = tid / TPG, tx = tid % TX, ty = (tid % TPG) / TX;
    const int nst = (K + BK - 1) / BK;
    const cx<T> *A = reinterpret_cast<const cx<T> *>(u.A);
    auto load_a = [&](int s) {
        cx<T> *dst = As + (s % NS) * AE;
#pragma unroll
        for (int q = 0; q < SK_M * BK / SK_TH; q++) {
            const int idx = tid + q * SK_TH;
            const int i = H ? idx % SK_M : idx / BK, kk = H ? idx / SK_M : idx % BK, k = s * BK + kk;
            const bool ok = i < M && k < K;
            const long long o = !ok ? 0 : H ? (long long)k * u.lda + i : (long long)i * u.lda + k;
            cp_async_cx_z(dst + (H ? kk * LDA + i : i * LDA + kk), A + o, ok);
        }
    };
    auto load_b = [&](int s) {
        cx<T> *dst = Bs + (s % NS) * BE;
        if constexpr (sizeof(cx<T>) * NC < 16) {
            for (int kk = tid; kk < BK; kk += SK_TH) {
                const int k = s * BK + kk;
                cp_async_cx_z(dst + kk, in + (k < K ? brow[k] : 0), k < K);
            }
        } else {
            constexpr int CPR = NC / VK;   // 16-byte pieces per row
#pragma unroll
            for (int idx = tid; idx < BK * CPR; idx += SK_TH) {
                const int kk = idx / CPR, c = idx % CPR, k = s * BK + kk;
                cp_async_16_z(dst + kk * NC + c * VK, in + (k < K ? (long long)brow[k] * NC + c * VK : 0), k < K);
            }
        }
    };
    for (int s = 0; s < NS - 1; s++)
        if (s < nst) load_a(s);
    for (int k = tid; k < K; k += SK_TH) brow[k] = u.bmap ? u.bmap[k] : u.b0 + k;
    if (tid < M) crow[tid] = u.cmap ? u.cmap[tid] : u.c0 + tid;
    __syncthreads();
    chain_wait();
    for (int s = 0; s < NS - 1; s++) {
        if (s < nst) load_b(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    cx<T> acc[4][CT];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < CT; j++) acc[i][j] = cx<T>(0);
    for (int s = 0; s < nst; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
        __syncthreads();   // stage s is there for all; stage s - 1 is no longer read
        if (s + NS - 1 < nst) {
            load_a(s + NS - 1);
            load_b(s + NS - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        cx<T> *Aw = As + (s % NS) * AE;
        const cx<T> *Bw = Bs + (s % NS) * BE;
        if (u.flags & (SK_LOWER | SK_UPPER)) {
            // the other triangle's entries of a stage that the diagonal crosses
            // become zeros (and ones on the unit diagonal); e: stored column minus
            // stored row of (row i, k)
            const int e0 = s * BK + u.d;
            if (e0 + BK > 0 && e0 - (SK_M - 1) <= 0) {
                for (int idx = tid; idx < SK_M * BK; idx += SK_TH) {
                    const int i = H ? idx % SK_M : idx / BK, kk = H ? idx / SK_M : idx % BK;
                    const int e = H ? i - (e0 + kk) : e0 + kk - i;
                    cx<T> *p = Aw + (H ? kk * LDA + i : i * LDA + kk);
                    if (u.flags & SK_UPPER) {
                        if (e < 0) *p = cx<T>(0);
                    } else if (e >= 0) {
                        *p = cx<T>(e == 0 ? T(1) : T(0));
                    }
                }
                __syncthreads();
            }
        }
        if constexpr (!H) {
#pragma unroll
            for (int kp = 0; kp < BK / VK; kp += KG) {
                const int kq = (kp + g) * VK;
                cx<T> a[4][VK];
#pragma unroll
                for (int i = 0; i < 4; i++) lds_cx<VK>(Aw + (ty + 16 * i) * LDA + kq, a[i]);
#pragma unroll
                for (int v = 0; v < VK; v++) {
                    cx<T> b[CT];
                    lds_cx<CT>(Bw + (kq + v) * NC + tx * CT, b);
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < CT; j++) cmac(acc[i][j], a[i][v], b[j]);
                }
            }
        } else {
#pragma unroll
            for (int kp = 0; kp < BK; kp += KG) {
                const int kq = kp + g;
                cx<T> a[4], b[CT];
                lds_cx<4>(Aw + kq * LDA + 4 * ty, a);
                lds_cx<CT>(Bw + kq * NC + tx * CT, b);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < CT; j++) cmac_conj(acc[i][j], a[i], b[j]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the groups' sums through shared memory, then whole rows of the output
    cx<T> *red = As;   // KG x SK_M x NC
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = H ? 4 * ty + i : ty + 16 * i;
#pragma unroll
        for (int j = 0; j < CT; j++) red[(g * SK_M + r) * NC + tx * CT + j] = acc[i][j];
    }
    __syncthreads();
    for (int idx = tid; idx < M * NC; idx += SK_TH) {
        cx<T> v = red[idx];
#pragma unroll
        for (int q = 1; q < KG; q++) v = v + red[q * SK_M * NC + idx];
        cx<T> *p = out + (long long)crow[idx / NC] * NC + idx % NC;
        if (u.flags & SK_SUB) v = -v;
        if (u.flags & SK_ATOM) red_add(p, v);
        else if (u.flags & SK_SUB) *p = *p + v;
        else *p = v;
    }
}

// The products with one column, except forward passes of small grids and of
// complex128.  Bound by
// reading A, once, so entries go from memory to registers without a stop in shared
// memory: as stored, a warp reads eight rows at a time, 32 neighbouring k each; of
// A^H, a warp reads whole stored rows, a lane per output row.  The loads are a tile
// ahead, the first two before the wait.  The large launches read 5.4 - 6 TB/s,
// 3.3 - 3.7 with the ring of k_skinny.
template <class T> __device__ __forceinline__ cx<T> ldg_cx(const cx<T> *p)
{
    if constexpr (sizeof(T) == 4) {
        const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
        return cx<T>(v.x, v.y);
    } else {
        const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
        return cx<T>(v.x, v.y);
    }
}
template <class T> __device__ __forceinline__ cx<T> ldcg_cx(const cx<T> *p)   // through L2
{
    if constexpr (sizeof(T) == 4) {
        const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
        return cx<T>(v.x, v.y);
    } else {
        const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
        return cx<T>(v.x, v.y);
    }
}

template <class T, bool H>
__global__ void __launch_bounds__(SK_TH) k_gemv(const SkUnit *__restrict__ units, const cx<T> *__restrict__ in,
                                                cx<T> *__restrict__ out)
{
    chain_start();
    // a warp's tile of entries: R rows x U times 32 k; of A^H U k x 64 rows
    constexpr int W = SK_TH / 32, R = H ? 2 : 8, U = (H ? 8 : 2) / ((int)sizeof(T) / 4);
    __shared__ cx<T> x[SK_KMAX], red[H ? W : 1][H ? SK_M : 1];
    const SkUnit u = units[blockIdx.x];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, K = u.K, M = u.M;
    const cx<T> *A = reinterpret_cast<const cx<T> *>(u.A);
    // a tile of the warp: its rows' group and its step along k
    struct Tile { int group, step; };
    const int nk = H ? (K + U * W - 1) / (U * W) : (K + 32 * U - 1) / (32 * U);
    const int ng = H ? 1 : max(0, (M - R * w + R * W - 1) / (R * W));
    auto next = [&](Tile n) { return n.step + 1 < nk ? Tile{n.group, n.step + 1} : Tile{n.group + 1, 0}; };
    auto row_of = [&](Tile n, int r) { return H ? lane + 32 * r : R * (w + W * n.group) + r; };
    auto k_of = [&](Tile n, int j) { return H ? (n.step * U + j) * W + w : (n.step * U + j) * 32 + lane; };
    auto load = [&](Tile n, cx<T>(&a)[U][R]) {
        if (n.group >= ng) return;
#pragma unroll
        for (int j = 0; j < U; j++)
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int k = k_of(n, j), i = row_of(n, r);
                a[j][r] = k < K && i < M ? ldg_cx(A + (H ? (long long)k * u.lda + i : (long long)i * u.lda + k))
                                         : cx<T>(0);
            }
    };
    cx<T> a[U][R], b[U][R], s[R];
    Tile at{0, 0}, ahead = next(at);   // K >= 1
    load(at, a);
    load(ahead, b);
    int row[SK_KMAX / SK_TH];   // of the input
#pragma unroll
    for (int j = 0; j < SK_KMAX / SK_TH; j++) {
        const int k = tid + j * SK_TH;
        row[j] = k >= K ? 0 : u.bmap ? u.bmap[k] : u.b0 + k;
    }
    chain_wait();
#pragma unroll
    for (int j = 0; j < SK_KMAX / SK_TH; j++)
        if (tid + j * SK_TH < K) x[tid + j * SK_TH] = ldcg_cx(in + row[j]);
    __syncthreads();
    const bool cut = (u.flags & (SK_LOWER | SK_UPPER)) != 0;
    auto store = [&](int i, cx<T> v) {
        cx<T> *p = out + (u.cmap ? u.cmap[i] : u.c0 + i);
        if (u.flags & SK_SUB) v = -v;
        if (u.flags & SK_ATOM) red_add(p, v);
        else if (u.flags & SK_SUB) *p = *p + v;
        else *p = v;
    };
#pragma unroll
    for (int r = 0; r < R; r++) s[r] = cx<T>(0);
    auto sum = [&](Tile n, cx<T>(&a)[U][R]) {
#pragma unroll
        for (int j = 0; j < U; j++) {
            const int k = k_of(n, j);
            const cx<T> xk = k < K ? x[k] : cx<T>(0);
#pragma unroll
            for (int r = 0; r < R; r++) {
                cx<T> v = a[j][r];
                if (cut) {   // the other triangle, as in k_skinny
                    const int e = H ? row_of(n, r) - (k + u.d) : k + u.d - row_of(n, r);
                    if ((u.flags & SK_UPPER) && e < 0) v = cx<T>(0);
                    if ((u.flags & SK_LOWER) && e >= 0) v = cx<T>(e == 0 ? T(1) : T(0));
                }
                if constexpr (H) cmac_conj(s[r], v, xk);
                else cmac(s[r], v, xk);
            }
        }
        if constexpr (!H) {
            if (n.step != nk - 1) return;
            // the lanes' sums: halves of the 2 R values are exchanged, so that after
            // four steps a pair of lanes holds one value
            T v[2 * R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                v[2 * r] = s[r].re;
                v[2 * r + 1] = s[r].im;
                s[r] = cx<T>(0);
            }
#pragma unroll
            for (int h = R, o = 16; h >= 1; h /= 2, o /= 2)
#pragma unroll
                for (int i = 0; i < h; i++) {
                    const T send = lane & o ? v[i] : v[i + h], keep = lane & o ? v[i + h] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            const T re = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
            const T im = __shfl_down_sync(0xffffffffu, re, 2);
            const int i = row_of(n, lane >> 2);
            if (lane % 4 == 0 && i < M) store(i, cx<T>(re, im));
        }
    };
    while (at.group < ng) {
        sum(at, a);
        at = next(ahead);
        load(at, a);
        if (ahead.group >= ng) break;
        sum(ahead, b);
        ahead = next(at);
        load(ahead, b);
    }
    if constexpr (H) {
        red[w][lane] = s[0];
        red[w][lane + 32] = s[1];
        __syncthreads();
        if (tid < M) {
            cx<T> v = red[0][tid];
#pragma unroll
            for (int q = 1; q < W; q++) v = v + red[q][tid];
            store(tid, v);
        }
    }
}

}  // namespace wt3d
