// The substitution passes' products over 8, 16 or 32 complex64 right-hand sides, on
// the tensor cores with the accuracy of FP32 multiply-adds.
//
// On the FP32 pipe these products are bound by its 73 TF/s (36 - 39 TF/s
// reached: at 32 columns a factor entry costs 128 multiply-adds for its 8 bytes).
// 16-bit mma.sync does 604 TF/s here (FP16), eight times that, for six products of split
// operands.  Every operand is h + m + l of 8 bits each, all 24 bits of FP32 and (BF16
// has FP32's exponents) whatever the magnitudes of the entries beside it; an entry of
// A below 2^-110 is held to 2^-134, and one of X likewise against its column's largest
// of 16 k, as the columns are scaled by powers of two; from 3.39e38 on an entry rounds
// to infinity.  Two halves in FP16 with three products take 2/3 to 3/4 of the time of
// a pass, but hold 22 bits, and fewer of an entry below 2^-16 of the largest of its
// row or column in 16 k.
// l h + h l + m m + m h + h m + h h of a k16 step is summed by the tensor cores, whose
// additions truncate, and only then added to FP32 sums with rounded operations: the
// error is 1.6e-7 at K = 1024 and 6e-8 at K = 32 (Gaussian entries), with FP32
// multiply-adds 4.0e-7 (8 columns) to 8.2e-7 (32) and 8e-8.  The operands come
// from tables through plain copies: a tcgen05 kernel that expanded B to real form in
// memory and kept its sums in tensor memory reached 63 TF/s on the largest blocks.
//
// A pass of 64x64x48 with 32, 16, 8 columns: 15.4, 10.5, 7.1 ms with FP32 products,
// 12.4, 8.0, 6.6 ms with these; 48^3 with 32: 8.2 and 6.7 ms.  Bound by the tensor
// pipe: half busy on 24576 x 1024 entries and 32 columns, 1.26 waves of CTAs, and the
// order of the products (one, two or four chains of them at a time) changes nothing.
#include <cuda_bf16.h>
#include "sub_kernels.cuh"

namespace wt3d {

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_bf16_0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%10, %10, %10, %10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// Two FP32 operations in one instruction: the instructions around the matrix
// products, not the products, fill the issue slots.
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 d;
    asm("{.reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; add.rn.f32x2 z, x, y; mov.b64 {%0, %1}, z;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    float2 d;
    asm("{.reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mul.rn.f32x2 z, x, y; mov.b64 {%0, %1}, z;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 d;
    asm("{.reg .b64 x, y, w, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mov.b64 w, {%6, %7}; "
        "fma.rn.f32x2 z, x, y, w; mov.b64 {%0, %1}, z;}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// (re, im) = h + m + l, each a pair of BF16 (re in the low half): 8 + 8 + 8 bits
__device__ __forceinline__ uint32_t bf16_pair(float2 v)
{
    const __nv_bfloat162 b = __floats2bfloat162_rn(v.x, v.y);
    return *reinterpret_cast<const uint32_t *>(&b);
}
__device__ __forceinline__ float2 minus_bf16(float2 v, uint32_t b)
{
    return fma2(make_float2(__uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u)), make_float2(-1.f, -1.f), v);
}
__device__ __forceinline__ void split_pair(float2 v, uint32_t &h, uint32_t &m, uint32_t &l)
{
    h = bf16_pair(v);
    v = minus_bf16(v, h);
    m = bf16_pair(v);
    l = bf16_pair(minus_bf16(v, m));
}

// Powers of two that take a largest magnitude m to [1, 2) ([2, 4) at the upper end of
// the range), and back
__device__ __forceinline__ void split_scale(float m, float &s, float &inv)
{
    const int e = min(max((int)(__float_as_uint(m) >> 23), 1), 253);
    s = __uint_as_float((unsigned)(254 - e) << 23);
    inv = __uint_as_float((unsigned)e << 23);
}

__device__ __forceinline__ float max_abs(float m, float2 v) { return fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))); }

// The units and their semantics are k_skinny's.  Four warps of 16 rows x NC
// columns.  A complex entry is one 32-bit register of an A fragment - the pair
// (re, im) along K, which a warp splits once; the pairs of B whose products with it are
// the real and the imaginary part are formed in registers.  B is split once per CTA, into shared memory in fragment order (two buffers, one barrier per
// chunk; loads one chunk ahead).  A comes through a ring per warp: fragments loaded
// straight from the matrix touch eight rows with every load, and those loads, not the
// tensor cores, were the bound.
// Units of fewer than st_kmin k are summed with FP32 multiply-adds: a chunk's
// truncated additions have an error of 6e-8 whatever its length.
constexpr int ST_KC = 16;   // complex k of a chunk: two k16 steps of the tensor cores
__host__ __device__ constexpr int st_kmin(int nc) { return nc == 8 ? 64 : 32; }
constexpr int ST_NS = 3;    // stages of a warp's ring
constexpr int ST_LD = 20;   // stride of its rows (of 16): a warp's reads of fragments meet no bank twice

template <int NC, bool H>
__global__ void __launch_bounds__(SK_TH, 4) k_skinny_tc(const SkUnit *__restrict__ units,
                                                        const cx<float> *__restrict__ in, cx<float> *__restrict__ out)
{
    chain_start();
    constexpr int NT = NC / 8;              // tiles of 8 columns
    constexpr int XV = NC == 32 ? 2 : 1;    // k16 steps of B per lane
    constexpr int CW = NC / 4;              // columns a warp splits
    constexpr int KMIN = st_kmin(NC);
    __shared__ __align__(16) float2 Aw[SK_TH / 32][ST_NS][16 * ST_LD];   // a ring per warp
    __shared__ uint4 Bf[2][KMIN * NC / 4 > 2 * NT * 32 ? KMIN * NC / 4 : 2 * NT * 32];   // h, m
    __shared__ uint2 Bl[2][2 * NT * 32];                                                 // l
    __shared__ float2 sb[2][NC / 2];
    __shared__ int brow[SK_KMAX], crow[SK_M];
    const SkUnit u = units[blockIdx.x];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, q = lane & 3, g = lane >> 2;
    const int K = u.K, M = u.M, nst = (K + ST_KC - 1) / ST_KC;
    const cx<float> *A = reinterpret_cast<const cx<float> *>(u.A);
    const float2 *in2 = reinterpret_cast<const float2 *>(in);
    const bool work = 16 * w < M;
    // rows g and g + 8 of a fragment are two neighbours of A^H: one 16-byte read
    const int r0 = 16 * w + (H ? 2 * g : g), r1 = H ? r0 + 1 : r0 + 8;
    const bool ok0 = r0 < M, ok1 = r1 < M;
    // c: along a stored row; stored rows l0, l0 + 2, ..
    const int c = lane & 15, l0 = lane >> 4;
    const cx<float> *Al = A + (H ? (long long)l0 * u.lda + 16 * w + c : (long long)(16 * w + l0) * u.lda + c);
    const long long step = H ? (long long)ST_KC * u.lda : ST_KC;
    auto load_a = [&](int s) {
        cx<float> *dst = reinterpret_cast<cx<float> *>(Aw[w][s % ST_NS]) + l0 * ST_LD + c;
        const cx<float> *src = Al + s * step;
        const int ki = K - s * ST_KC, mi = M - 16 * w;   // k and rows left
        if (ki >= ST_KC && mi >= 16) {
#pragma unroll
            for (int h = 0; h < 8; h++) cp_async_cx(dst + 2 * h * ST_LD, src + 2 * h * (long long)u.lda);
        } else {
#pragma unroll
            for (int h = 0; h < 8; h++) {
                const bool ok = c < (H ? mi : ki) && l0 + 2 * h < (H ? ki : mi);
                cp_async_cx_z(dst + 2 * h * ST_LD, ok ? src + 2 * h * (long long)u.lda : A, ok);
            }
        }
    };
    // lane (k within a step, column [, step]) of B
    const int xc = CW * w + g % CW, xs = XV == 2 ? 0 : (g / CW) & 1;
    const bool xw = lane < 8 * CW;          // 8 columns: half of the lanes
    float2 x[2 * XV];
    auto load_x = [&](int s) {
#pragma unroll
        for (int j = 0; j < 2 * XV; j++) {
            const int k = s * ST_KC + 8 * xs + 4 * j + q;
            // through L2: another kernel of the chain has written it
            x[j] = k < K ? __ldcg(in2 + (long long)brow[k] * NC + xc) : make_float2(0.f, 0.f);
        }
    };
    const bool fp32 = K < KMIN;
    if (!fp32)
        for (int s = 0; s < ST_NS - 1; s++) {   // the factor's entries: no product writes them
            if (work && s < nst) load_a(s);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    for (int k = tid; k < K; k += SK_TH) brow[k] = u.bmap ? u.bmap[k] : u.b0 + k;
    if (tid < M) crow[tid] = u.cmap ? u.cmap[tid] : u.c0 + tid;
    __syncthreads();
    chain_wait();
    // [tile][re, im][r0, r1]: columns 2 q and 2 q + 1 of the tile
    float2 acc[NT][2][2];
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[t][j >> 1][j & 1] = make_float2(0.f, 0.f);
    if (fp32) {
        float2 *X = reinterpret_cast<float2 *>(&Bf[0][0]);   // K x NC
        static_assert(sizeof(Bf) >= sizeof(float2) * KMIN * NC, "B of a short unit");
        for (int i = tid; i < K * NC; i += SK_TH) X[i] = __ldcg(in2 + (long long)brow[i / NC] * NC + i % NC);
        __syncthreads();
        constexpr int KG = 32 / NC;   // sums of every KG-th k
        for (int k0 = 0; k0 < KG; k0++) {
            float2 sum[NT][2][2];
#pragma unroll
            for (int t = 0; t < NT; t++)
#pragma unroll
                for (int j = 0; j < 4; j++) sum[t][j >> 1][j & 1] = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int k = k0; k < K; k += KG) {
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int i = r ? r1 : r0, e = H ? i - (k + u.d) : k + u.d - i;
                    cx<float> v(0);
                    if (r ? ok1 : ok0) v = A[H ? (long long)k * u.lda + i : (long long)i * u.lda + k];
                    if ((u.flags & SK_UPPER) && e < 0) v = cx<float>(0);
                    if ((u.flags & SK_LOWER) && e >= 0) v = cx<float>(e == 0 ? 1.f : 0.f);
                    if (H) v.im = -v.im;
#pragma unroll
                    for (int t = 0; t < NT; t++) {
                        // columns 2 q and 2 q + 1
                        const float4 b = *reinterpret_cast<const float4 *>(X + k * NC + 8 * t + 2 * q);
                        float2 &re = sum[t][0][r], &im = sum[t][1][r];
                        re.x = fmaf(v.re, b.x, fmaf(-v.im, b.y, re.x));
                        re.y = fmaf(v.re, b.z, fmaf(-v.im, b.w, re.y));
                        im.x = fmaf(v.re, b.y, fmaf(v.im, b.x, im.x));
                        im.y = fmaf(v.re, b.w, fmaf(v.im, b.z, im.y));
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < NT; t++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[t][j >> 1][j & 1] = add2(acc[t][j >> 1][j & 1], sum[t][j >> 1][j & 1]);
        }
    } else {
        load_x(0);
    }
    for (int s = 0; s < (fp32 ? 0 : nst); s++) {
        const int buf = s & 1;
        {
            float m = 0.f, sc, inv;
#pragma unroll
            for (int j = 0; j < 2 * XV; j++) m = max_abs(m, x[j]);
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            if (XV == 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4 * CW));
            split_scale(m, sc, inv);
            if (q == 0 && xs == 0 && xw) reinterpret_cast<float *>(sb[buf])[xc] = inv;
#pragma unroll
            for (int j = 0; j < XV; j++) {
                uint4 v;
                uint2 l;
                split_pair(mul2(x[2 * j], make_float2(sc, sc)), v.x, v.z, l.x);
                split_pair(mul2(x[2 * j + 1], make_float2(sc, sc)), v.y, v.w, l.y);
                const int at = ((xs + j) * NT + (xc >> 3)) * 32 + 4 * (xc & 7) + q;
                if (xw) {
                    Bf[buf][at] = v;
                    Bl[buf][at] = l;
                }
            }
        }
        if (s + 1 < nst) load_x(s + 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(ST_NS - 2) : "memory");
        __syncthreads();   // the chunk's A and B are there; the ones before are no longer read
        if (!work) continue;
        if (s + ST_NS - 1 < nst) load_a(s + ST_NS - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        float2 a[8];       // [k16 step][k or k + 4][row]
        const float2 *Ar = Aw[w][s % ST_NS];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            if constexpr (H) {
                const float4 v = *reinterpret_cast<const float4 *>(Ar + (4 * h + q) * ST_LD + 2 * g);
                a[2 * h] = make_float2(v.x, v.y);
                a[2 * h + 1] = make_float2(v.z, v.w);
            } else {
                a[2 * h] = Ar[g * ST_LD + 4 * h + q];
                a[2 * h + 1] = Ar[(g + 8) * ST_LD + 4 * h + q];
            }
        }
        if (u.flags & (SK_LOWER | SK_UPPER)) {
            // as in k_skinny: zeros (ones on the unit diagonal) for the other triangle
            const int e0 = s * ST_KC + u.d;
            if (e0 + ST_KC > 0 && e0 - (SK_M - 1) <= 0) {
#pragma unroll
                for (int h = 0; h < 8; h++) {
                    const int i = h & 1 ? r1 : r0, kk = 4 * (h >> 1) + q;
                    const int e = H ? i - (e0 + kk) : e0 + kk - i;
                    if (u.flags & SK_UPPER) {
                        if (e < 0) a[h] = make_float2(0.f, 0.f);
                    } else if (e >= 0) {
                        a[h] = make_float2(e == 0 ? 1.f : 0.f, 0.f);
                    }
                }
            }
        }
        uint32_t ah[2][4], am[2][4], al[2][4];   // [k16 step]
#pragma unroll
        for (int h = 0; h < 8; h++) split_pair(a[h], ah[h >> 2][h & 3], am[h >> 2][h & 3], al[h >> 2][h & 3]);
#pragma unroll
        for (int t = 0; t < NT; t++) {
            float d[2][2][4];   // [re, im][k16 step]: four independent chains
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const uint4 f = Bf[buf][(e * NT + t) * 32 + lane];
                const uint2 f2 = Bl[buf][(e * NT + t) * 32 + lane];
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    // (xr, -xi) and (xi, xr); for A^H (xr, xi) and (xi, -xr)
                    auto form = [&](uint32_t v) {
                        if (c == 0) return H ? v : v ^ 0x80000000u;
                        const uint32_t r = __byte_perm(v, 0, 0x1032);
                        return H ? r ^ 0x80000000u : r;
                    };
                    const uint32_t h0 = form(f.x), h1 = form(f.y), m0 = form(f.z), m1 = form(f.w), l0 = form(f2.x),
                                   l1 = form(f2.y);
                    // the small products first
                    mma_bf16_0(d[c][e], al[e], h0, h1);
                    mma_bf16(d[c][e], ah[e], l0, l1);
                    mma_bf16(d[c][e], am[e], m0, m1);
                    mma_bf16(d[c][e], am[e], h0, h1);
                    mma_bf16(d[c][e], ah[e], m0, m1);
                    mma_bf16(d[c][e], ah[e], h0, h1);
                }
            }
            const float2 sx = sb[buf][4 * t + q];
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const float(&d0)[4] = d[c][0], (&d1)[4] = d[c][1];
                    const float2 v = add2(make_float2(d0[2 * r], d0[2 * r + 1]), make_float2(d1[2 * r], d1[2 * r + 1]));
                    acc[t][c][r] = fma2(v, sx, acc[t][c][r]);
                }
        }
    }
    const float sgn = u.flags & SK_SUB ? -1.f : 1.f;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (!(r ? ok1 : ok0)) continue;
        float4 *row = reinterpret_cast<float4 *>(out + (long long)crow[r ? r1 : r0] * NC) + q;   // two columns
#pragma unroll
        for (int t = 0; t < NT; t++) {
            const float2 re = acc[t][0][r], im = acc[t][1][r];
            float4 v = make_float4(sgn * re.x, sgn * im.x, sgn * re.y, sgn * im.y);
            float4 *p = row + 4 * t;
            if (u.flags & SK_ATOM) {
                atomicAdd(p, v);
                continue;
            }
            if (u.flags & SK_SUB) {
                const float4 o = *p;
                v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
            }
            *p = v;
        }
    }
}

template <int NC, bool H>
static void launch(const SkUnit *u, int n, const cx<float> *in, cx<float> *out, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n);
    cfg.blockDim = dim3(SK_TH);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_skinny_tc<NC, H>, u, in, out);
}

void sk_tensor_launch(int nc, bool herm, const SkUnit *u, int n, const cx<float> *in, cx<float> *out, cudaStream_t st)
{
    if (nc == 8) (herm ? launch<8, true> : launch<8, false>)(u, n, in, out, st);
    else if (nc == 16) (herm ? launch<16, true> : launch<16, false>)(u, n, in, out, st);
    else (herm ? launch<32, true> : launch<32, false>)(u, n, in, out, st);
}

}  // namespace wt3d
