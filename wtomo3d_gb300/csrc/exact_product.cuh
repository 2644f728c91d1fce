// Products of the grid's operator with blocks of 8, 16 or 32 complex128 right-hand
// sides (5 columns and more), on the tensor cores, every row to the accuracy of an FP64
// sum or better.
//
// The FP64 pipe (2 FMA per cycle and SM) bounds the residual r = b - A x: 8.8 ms
// for 32 columns of 64x64x48, a third of a refinement step, where reading the
// operator takes 0.1 ms.  Here every operand is an integer of 62 bits and sign
// times a power of two (per row of A; per column and 6 x 6 x 6 block of nodes of
// X, so that a quiet region is not held to the scale of a source elsewhere), cut
// into eight signed digits of 8 bits.  Before that the columns of A are brought to
// a largest entry in [1, 2) by powers of two, and the rows of X multiplied by
// them: Dirichlet rows carry a unit diagonal next to stiffness entries of 1e8, and
// in a conjugate-transpose solve their unknowns are 1e8 times the others.  A product of two digits is an integer of
// at most 2^14; the sums of 162 products over up to seven digit pairs of equal
// weight stay below 2^24, so FP16 tensor-core products with FP32 accumulation are
// exact (the error-free splitting of Ozaki, Ogita, Oishi and Rump, 2012).  The 43
// digit pairs down to weight 2^-64 of the leading one are summed; what is left
// out is of the order of 2^-65 of the row's largest |a| times the block's largest
// |x|, against 2^-53 per operation of an FP64 sum.  The integers are added in 64 bits
// and rounded once.
//
// A result all of whose products are far smaller than that product of maxima would
// lose bits: next to a source, at the outer corners of the absorbing layers, in a
// component that is small beside the others.  So each result's largest |a| |x|, by its
// exponents, is held against the unit of the integers, and what would lose more than
// EP_LOSS bits takes the plain FP64 sum, as do rows and columns with an infinity or a
// NaN: every row has the error of its own FP64 sum, whatever surrounds it.  Rows with
// one entry (Dirichlet rows) are one FP64 product.
//
// Errors against extended precision, 2-norm over the product, 13x12x11: random
// fields 4.7e-17 (FP64 kernel 1.6e-16), wave fields 4.3e-17 (1.4e-15).  32 columns
// of 64x64x48 in 3.2 ms instead of 8.8; the digits of the operator, 0.3 ms, are
// made once per call.
#pragma once
#include "refine_kernels.cuh"
#include <cuda_fp16.h>

namespace wt3d {

constexpr int EP_SLOTS = 88;      // complex entries per row: 27 neighbours x 3, padded to 11 steps of 8
constexpr int EP_T = 4, EP_H = EP_T + 2;   // nodes of a block and of its halo per axis
constexpr int EP_COLS = 16;       // columns per CTA (the M of the tensor-core shape)
constexpr int EP_ES = EP_COLS + 2;   // row of one entry in shared memory (16-byte units; four entries on different banks)
constexpr int EP_THREADS = 512;
constexpr int EP_ENTRIES = EP_H * EP_H * EP_H * 3;
constexpr size_t EP_SMEM = (size_t)EP_ENTRIES * (EP_ES * 16 + EP_COLS * 2);
constexpr unsigned long long EP_BIAS = 0x8080808080808080ull;   // digit + 128 in every byte
constexpr int EP_BAD = 1 << 20;   // exponent of rows and columns with infinities or NaNs
constexpr int EP_NONE = -(1 << 20);   // ... of all zeros
constexpr int EP_SINGLE = 1 << 21;   // ... of rows with one entry: plus its position in the row
constexpr int EP_LOSS = 8;        // bits a row may lose: the error stays at that of an FP64 sum
constexpr int EP_NOWHERE = -8192;   // scaled exponent of a zero entry of X
constexpr unsigned EP_ZERO = 6144;   // bits from which a product is one of zeros (others: at most 4346)

// The operator of a product: A, A^H, or B - A (the sources of an incident field).
struct ProductOp {
    const int *irptr, *jcptr, *tpos;
    const double2 *a, *b;         // b: with b != nullptr the operator is b - a
    int adjoint;
    __device__ __forceinline__ double2 at(long long k) const
    {
        if (b) {
            const double2 u = b[k], v = a[k];
            return make_double2(u.x - v.x, u.y - v.y);
        }
        if (adjoint) {
            const double2 v = a[tpos[k]];
            return make_double2(v.x, -v.y);
        }
        return a[k];
    }
};

// larger exponent field of the two parts, EP_NONE for zero
__device__ __forceinline__ int ep_exponent(double2 v)
{
    const int m = max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff), e = m >> 20;
    return e == 0x7ff ? EP_BAD : (m | __double2loint(v.x) | __double2loint(v.y)) == 0 ? EP_NONE : max(e, 1);
}

// v 2^(s + 62 - (E - 1022)) rounded to an integer, plus the digits' bias; E the
// largest of the exponents + s of v's row or column, so that the integer is below
// 2^62
__device__ __forceinline__ unsigned long long ep_quantise(double v, int s, int E)
{
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
    const int e = (int)(bits >> 52) & 0x7ff;
    unsigned long long m = bits & 0xfffffffffffffull;
    if (e) m |= 0x10000000000000ull;
    const int sh = 9 - (E - (max(e, 1) + s));
    unsigned long long q = sh >= 0 ? m << min(sh, 9) : sh > -60 ? (m + (1ull << (-sh - 1))) >> -sh : 0ull;
    if ((long long)bits < 0) q = 0ull - q;
    return q + EP_BIAS;
}

// pe[j]: exponent of column j of the operator (1023, that is no scaling, for a
// column of zeros or with infinities or NaNs): a warp per row of its transpose
__global__ void __launch_bounds__(256) k_column_exponents(long long n, ProductOp op, int *__restrict__ pe)
{
    const long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    int E = EP_NONE;
    for (int k = op.irptr[r] + lane; k < op.irptr[r + 1]; k += 32) {
        const int j = op.adjoint ? k : op.tpos[k];   // entry (column r) of A, of A^H: row r of A
        double2 v = op.a[j];
        if (op.b) { const double2 u = op.b[j]; v = make_double2(u.x - v.x, u.y - v.y); }
        E = max(E, ep_exponent(v));
    }
    E = __reduce_max_sync(0xffffffffu, E);
    if (lane == 0) pe[r] = E == EP_NONE || E == EP_BAD ? 1023 : E;
}

// A biased pair (re, im) as the kernels keep it: word p holds digits 2 p and 2 p + 1
// (0: the most significant) as bytes re, im, re, im, so that one byte permutation
// makes a pair of FP16 numbers (three instructions per pair of digits with the halves
// of re and im in words of their own: 1986 us, now 1761, for 32 columns of 48^3)
__device__ __forceinline__ uint4 ep_pack(unsigned long long re, unsigned long long im)
{
    const uint32_t rh = (uint32_t)(re >> 32), rl = (uint32_t)re, ih = (uint32_t)(im >> 32), il = (uint32_t)im;
    return make_uint4(__byte_perm(rh, ih, 0x6273), __byte_perm(rh, ih, 0x4051), __byte_perm(rl, il, 0x6273),
                      __byte_perm(rl, il, 0x4051));
}

// digit i of a pair as two FP16 values: bytes 0x64xx are 1024 + xx; mul and add turn
// them into the digits or their negatives.  s0, s1: permutations of the even and the
// odd digit of a word, EP_S0 and EP_S1 for (re, im), their ^ 0x0101 for (im, re)
constexpr uint32_t EP_S0 = 0x4140, EP_S1 = 0x4342;
__device__ __forceinline__ uint32_t ep_digit(const uint4 &q, int i, uint32_t s0, uint32_t s1, __half2 mul, __half2 add)
{
    const uint32_t w = i < 2 ? q.x : i < 4 ? q.y : i < 6 ? q.z : q.w;
    const uint32_t t = __byte_perm(w, 0x64646464u, i & 1 ? s1 : s0);
    const __half2 h = __hfma2(*reinterpret_cast<const __half2 *>(&t), mul, add);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// Rows of the operator as digits: a warp per node; row q of node g holds its 27
// neighbours (dy, dx, dz) x 3 components at aq[(3 g + q) EP_SLOTS ..], zeros where
// there is no neighbour, at the same places of below how many bits the entry is below
// the row's largest (255: at least as many, or a zero), and in aexp the row's exponent
// times 256 plus that number of its diagonal.
__global__ void __launch_bounds__(256) k_operator_digits(int nx, int ny, int nz, ProductOp op,
                                                         const int *__restrict__ pe, uint4 *__restrict__ aq,
                                                         unsigned char *__restrict__ below,
                                                         int *__restrict__ aexp)
{
    const long long nn = (long long)nx * ny * nz;
    const long long g = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (g >= nn) return;
    const int iz = (int)(g % nz), ix = (int)((g / nz) % nx), iy = (int)(g / ((long long)nz * nx));
    const int z0 = max(iz - 1, 0), z1 = min(iz + 1, nz - 1), x0 = max(ix - 1, 0), x1 = min(ix + 1, nx - 1),
              y0 = max(iy - 1, 0);
    const int y1 = min(iy + 1, ny - 1);
    const long long k0 = op.irptr[3 * g];
    const int len = op.irptr[3 * g + 1] - (int)k0;
    int pos[3], sc[3];   // the lane's slots lane + 32 j: position in the row, -1 for none; column scaling
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int s = lane + 32 * j, nb = s / 3, c = s % 3;
        const int y = iy + nb / 9 - 1, x = ix + (nb / 3) % 3 - 1, z = iz + nb % 3 - 1;
        pos[j] = (s < 81 && y >= y0 && y <= y1 && x >= x0 && x <= x1 && z >= z0 && z <= z1)
                     ? (((y - y0) * (x1 - x0 + 1) + (x - x0)) * (z1 - z0 + 1) + (z - z0)) * 3 + c
                     : -1;
        sc[j] = pos[j] >= 0 ? 1023 - pe[op.jcptr[k0 + pos[j]]] : 0;
    }
#pragma unroll
    for (int q = 0; q < 3; q++) {
        double2 v[3];
        int ex[3], E = EP_NONE, cnt = 0, at = -1;   // exponents, the largest scaled one; nonzero entries
#pragma unroll
        for (int j = 0; j < 3; j++) {
            v[j] = pos[j] >= 0 ? op.at(k0 + (long long)q * len + pos[j]) : make_double2(0, 0);
            ex[j] = ep_exponent(v[j]);
            E = max(E, ex[j] == EP_BAD ? EP_BAD : ex[j] + sc[j]);
            if (ex[j] != EP_NONE) {
                cnt++;
                at = pos[j];
            }
        }
        E = __reduce_max_sync(0xffffffffu, E);
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        at = __reduce_max_sync(0xffffffffu, at);
        int low[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int s = lane + 32 * j;
            low[j] = ex[j] == EP_NONE ? 255 : min(255, E - (ex[j] + sc[j]));
            if (s < EP_SLOTS) {
                aq[(3 * g + q) * EP_SLOTS + s] = ep_pack(ep_quantise(v[j].x, sc[j], E), ep_quantise(v[j].y, sc[j], E));
                below[(3 * g + q) * EP_SLOTS + s] = (unsigned char)low[j];
            }
        }
        const int diag = __shfl_sync(0xffffffffu, low[1], 39 + q - 32);   // slot 39 + q
        if (lane == 0) aexp[3 * g + q] = (E >= EP_BAD || E < EP_NONE / 2 || cnt != 1 ? E : EP_SINGLE + at) * 256 + diag;
    }
}

__device__ __forceinline__ void ep_mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// an integer of magnitude below 2^51 as a double
__device__ __forceinline__ double ep_double(long long v)
{
    return __longlong_as_double(v + 0x4338000000000000ll) - 6755399441055744.0;
}

// R = B - A X, with the column norms of R and B added to nr and nb as k_residual
// does it; with B null R = A X, no norms.  One CTA per 4 x 4 x 4 nodes and
// 16 columns: the block's X with its halo goes into shared memory as biased integers; then a
// warp per node (four in turn) runs the node's three rows as the N = 8 side (re and
// im of each row, two unused) and the columns as the M = 16 side of
// m16n8k16 products, 8 entries per step, making the digits of both sides in
// registers.  The results that take the FP64 sum are left to k_product_rest (24 us for
// 1 % of the nodes of 32x32x24 with 16 columns): a lane's sum of 81 products in here
// held up its tile, 376 us instead of 240.  rest[0] counts its tasks, from rest[2] on: twice the row plus
// the column group, and the columns (bit 4 g: column g, bit 4 g + 1: column g + 8).
template <int NC>
__global__ void __launch_bounds__(EP_THREADS, 1)
    k_product_tc(int nx, int ny, int nz, ProductOp op, const uint4 *__restrict__ aq,
                 const unsigned char *__restrict__ below, const int *__restrict__ aexp,
                 const int *__restrict__ pe, const double2 *__restrict__ X, const double2 *__restrict__ B,
                 double2 *__restrict__ R, double *__restrict__ nr, double *__restrict__ nb, unsigned *__restrict__ rest)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    uint4 *Xq = reinterpret_cast<uint4 *>(smraw);   // EP_ENTRIES x EP_ES
    // scaled exponents: columns c and c + 8 in a word
    uint32_t *xe = reinterpret_cast<uint32_t *>(Xq + EP_ENTRIES * EP_ES);   // EP_ENTRIES x EP_COLS / 2
    __shared__ int cexp[EP_COLS], off[EP_SLOTS];
    __shared__ double red[2][EP_THREADS / 32][EP_COLS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tz = (nz + EP_T - 1) / EP_T, tx = (nx + EP_T - 1) / EP_T;
    // the column groups of a tile follow one another: the second finds A in L2
    constexpr int NG = (NC + EP_COLS - 1) / EP_COLS;
    const long long tile = blockIdx.x / NG;
    const int bz = (int)(tile % tz) * EP_T, bx = (int)((tile / tz) % tx) * EP_T,
              by = (int)(tile / ((long long)tz * tx)) * EP_T;
    const int c0 = EP_COLS * (int)(blockIdx.x % NG);
    // the tile's operator rows are read one step ahead of their use, which does not
    // cover DRAM: on their way to L2 while X is loaded (runs of 4 nodes along z)
    for (int q = tid; q < EP_T * EP_T * (EP_T * 3 * EP_SLOTS * 16 / 128); q += EP_THREADS) {
        constexpr int LINES = EP_T * 3 * EP_SLOTS * 16 / 128;
        const int ix = bx + (q / LINES) % EP_T, iy = by + q / (LINES * EP_T);
        const long long node = bz + (long long)nz * (ix + (long long)nx * iy);
        const long long off = (3 * node * EP_SLOTS) * 16 + (long long)(q % LINES) * 128;
        if (ix < nx && iy < ny && off < 3LL * nx * ny * nz * EP_SLOTS * 16)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(aq) + off));
    }
    if (tid < EP_COLS) cexp[tid] = EP_NONE;
    if (tid < EP_SLOTS) {
        const int s = min(tid, 80), k = s / 3;
        off[tid] = (k % 3 + EP_H * ((k / 3) % 3 + EP_H * (k / 9))) * 3 + s % 3;
    }
    __syncthreads();
    // X with halo, as stored; the columns' exponents
    {
        const int c = tid % EP_COLS;
        const bool col = c0 + c < NC;
        int E = EP_NONE;
        auto row_of = [&](int e) -> long long {   // entry's row of X, -1 outside the grid
            const int h = e / 3;
            const int z = bz + h % EP_H - 1, x = bx + (h / EP_H) % EP_H - 1, y = by + h / (EP_H * EP_H) - 1;
            if (z < 0 || z >= nz || x < 0 || x >= nx || y < 0 || y >= ny) return -1;
            return 3 * (z + (long long)nz * (x + (long long)nx * y)) + e % 3;
        };
#pragma unroll 4
        for (int e = tid / EP_COLS; e < EP_ENTRIES; e += EP_THREADS / EP_COLS) {
            const long long r = row_of(e);
            double2 v = make_double2(0, 0);
            int low = EP_NOWHERE;
            if (col && r >= 0) {
                v = X[r * NC + c0 + c];
                const int x = ep_exponent(v);
                low = x == EP_NONE ? EP_NOWHERE : x + pe[r] - 1023;
                E = max(E, x == EP_BAD ? x : x == EP_NONE ? E : low);
            }
            reinterpret_cast<short *>(xe)[e * EP_COLS + 2 * (c & 7) + (c >> 3)] = (short)low;
            reinterpret_cast<double2 *>(Xq)[e * EP_ES + c] = v;
        }
        atomicMax(&cexp[c], E);
        __syncthreads();
        E = cexp[c];
        for (int e = tid / EP_COLS; e < EP_ENTRIES; e += EP_THREADS / EP_COLS) {
            const long long r = row_of(e);
            const int s = r >= 0 ? pe[r] - 1023 : 0;
            const double2 v = reinterpret_cast<const double2 *>(Xq)[e * EP_ES + c];
            Xq[e * EP_ES + c] = ep_pack(ep_quantise(v.x, s, E), ep_quantise(v.y, s, E));
        }
    }
    __syncthreads();
    const int g = lane >> 2, t = lane & 3;   // fragment coordinates
    // this lane's operand of A: row q = g / 2, (ar, -ai) for its real part, (ai, ar)
    // for its imaginary part; g = 6, 7 are the unused ones
    const int qa = g >> 1;
    const bool part = g & 1, live = g < 6;
    const __half2 one = __floats2half2_rn(1.f, 1.f), one_off = __floats2half2_rn(-1152.f, -1152.f);
    const uint32_t sa = part ? 0x0101u : 0u;
    const __half2 zero = __floats2half2_rn(0.f, 0.f);
    const __half2 amul = !live ? zero : part ? one : __floats2half2_rn(1.f, -1.f);
    const __half2 aadd = !live ? zero : part ? one_off : __floats2half2_rn(-1152.f, 1152.f);
    double sr[2] = {0, 0}, sb[2] = {0, 0};
    auto node_of = [&](int ln) -> long long {   // node ln of the tile, -1 outside the grid
        const int iz = bz + ln % EP_T, ix = bx + (ln / EP_T) % EP_T, iy = by + ln / (EP_T * EP_T);
        return ln >= EP_T * EP_T * EP_T || iz >= nz || ix >= nx || iy >= ny ? -1 : iz + (long long)nz * (ix + (long long)nx * iy);
    };
    auto fetch_exponent = [&](long long node) { return node < 0 ? 0 : aexp[3 * node + min(t, 2)]; };
    int next = fetch_exponent(node_of(warp));   // of the lane's row, a node ahead of its use
    for (int ln = warp; ln < EP_T * EP_T * EP_T; ln += EP_THREADS / 32) {
        const long long node = node_of(ln);
        const int ea = next;
        next = fetch_exponent(node_of(ln + EP_THREADS / 32));
        if (node < 0) continue;
        const int lz = ln % EP_T, lx = (ln / EP_T) % EP_T, ly = ln / (EP_T * EP_T);
        const uint4 *ar = aq + (3 * node + (live ? qa : 0)) * EP_SLOTS + t;
        uint4 p0 = ar[0], p1 = ar[4];
        const int first = (lz + EP_H * (lx + EP_H * ly)) * 3;   // entry of the node's first neighbour
        const uint4 *xb = Xq + first * EP_ES + g;
        // The bits a result loses: its largest product against the unit of the integers.
        // First a bound, the product of the diagonal; where that is too far below, all
        // 81, every fourth by each of the four lanes of a column pair.  Bit h of plain:
        // column g + 8 h takes the FP64 sum.
        const int Ea = ea >> 8, diag = ea & 255, q = min(t, 2);
        const int Ex[2] = {cexp[g], cexp[g + 8]};
        unsigned plain = 0;
        {
            bool low = false;
            const uint32_t centre = xe[(first + off[39 + q]) * (EP_COLS / 2) + g];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (c0 + g + 8 * h >= NC) continue;
                if (Ex[h] == EP_BAD || Ea == EP_BAD) plain |= 1u << h;
                else if (abs(Ea) < EP_BAD / 2 && abs(Ex[h]) < EP_BAD / 2)
                    low |= diag + Ex[h] - (int)(short)(centre >> (16 * h)) > EP_LOSS;
            }
            if (__any_sync(0xffffffffu, low)) {
                const unsigned char *bl = below + 3 * node * EP_SLOTS;
                const uint32_t top = (uint32_t)(Ex[0] & 0xffff) | (uint32_t)Ex[1] << 16;
                uint32_t least[3] = {0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu};
                for (int s = t; s < 81; s += 4) {
                    const uint32_t x = __vsub2(top, xe[(first + off[s]) * (EP_COLS / 2) + g]);
#pragma unroll
                    for (int r = 0; r < 3; r++)
                        least[r] = __viaddmin_s16x2(bl[r * EP_SLOTS + s] * 0x10001u, x, least[r]);
                }
#pragma unroll
                for (int r = 0; r < 3; r++)
#pragma unroll
                    for (int o = 1; o < 4; o <<= 1)
                        least[r] = __vmins2(least[r], __shfl_xor_sync(0xffffffffu, least[r], o));
                const uint32_t l = q == 0 ? least[0] : q == 1 ? least[1] : least[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const unsigned b = l >> (16 * h) & 0xffffu;   // from EP_ZERO: a sum of zeros, exact
                    if (c0 + g + 8 * h < NC && abs(Ea) < EP_BAD / 2 && abs(Ex[h]) < EP_BAD / 2 && b > EP_LOSS &&
                        b < EP_ZERO)
                        plain |= 1u << h;
                }
            }
            const unsigned m0 = __ballot_sync(0xffffffffu, plain & 1u), m1 = __ballot_sync(0xffffffffu, plain & 2u);
            if (m0 | m1) {
                const unsigned m = (m0 >> t & 0x11111111u) | (m1 >> t & 0x11111111u) << 1;
                if (lane < 3 && m) {
                    const unsigned i = atomicAdd(rest, 1u);
                    rest[2 + 2 * (size_t)i] = (unsigned)(2 * (3 * node + t)) + (unsigned)(c0 / EP_COLS);
                    rest[3 + 2 * (size_t)i] = m;
                }
            }
        }
        float acc[11][4];   // digit pairs of weight 0 .. 6, 7 and 8 (two halves each: sums below 2^24)
#pragma unroll
        for (int s = 0; s < 11; s++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[s][j] = 0.f;
#pragma unroll 1
        for (int st = 0; st < EP_SLOTS / 8; st++) {
            const uint4 a0 = p0, a1 = p1;
            if (st + 1 < EP_SLOTS / 8) { p0 = ar[8 * st + 8]; p1 = ar[8 * st + 12]; }
            const uint4 *e0 = xb + off[8 * st + t] * EP_ES, *e1 = xb + off[8 * st + 4 + t] * EP_ES;
            const uint4 x0 = e0[0], x1 = e0[8], x2 = e1[0], x3 = e1[8];
            uint32_t ad[8][2];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                ad[j][0] = ep_digit(a0, j, EP_S0 ^ sa, EP_S1 ^ sa, amul, aadd);
                ad[j][1] = ep_digit(a1, j, EP_S0 ^ sa, EP_S1 ^ sa, amul, aadd);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                uint32_t dg[4];
                dg[0] = ep_digit(x0, i, EP_S0, EP_S1, one, one_off);
                dg[1] = ep_digit(x1, i, EP_S0, EP_S1, one, one_off);
                dg[2] = ep_digit(x2, i, EP_S0, EP_S1, one, one_off);
                dg[3] = ep_digit(x3, i, EP_S0, EP_S1, one, one_off);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (i + j < 9) ep_mma(acc[i + j < 7 ? i + j : 2 * (i + j) - 7 + (i < 4 ? 0 : 1)], dg, ad[j]);
            }
        }
        if (t < 3) {
            // entries (column g or g + 8, row q = t): re and im
            const long long row = 3 * node + t;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int c = c0 + g + 8 * h;
                if (c >= NC || (plain >> h & 1u)) continue;
                double2 v;
                if (Ea >= EP_SINGLE) {
                    const long long k = op.irptr[row] + (Ea - EP_SINGLE);
                    const double2 av = op.at(k), x = X[(long long)op.jcptr[k] * NC + c];
                    v = make_double2(fma(av.x, x.x, -av.y * x.y), fma(av.x, x.y, av.y * x.x));
                } else {
                    double w[2];
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        long long hi = 0, lo = 0;
#pragma unroll
                        for (int s = 0; s < 4; s++) hi = hi * 256 + __float2int_rn(acc[s][2 * h + p]);
#pragma unroll
                        for (int s = 4; s < 7; s++) lo = lo * 256 + __float2int_rn(acc[s][2 * h + p]);
                        lo = lo * 256 + __float2int_rn(acc[7][2 * h + p]) + __float2int_rn(acc[8][2 * h + p]);
                        // weight 8: rounded to the unit of lo, 2^-68 of the leading product
                        lo += (__float2int_rn(acc[9][2 * h + p]) + __float2int_rn(acc[10][2 * h + p]) + 128) >> 8;
                        w[p] = fma(ep_double(hi), 4294967296.0, ep_double(lo));
                    }
                    // unit of the integers: 2^56 from the digits, 2^(E - 1022 - 62) of each side
                    if (Ea < EP_NONE / 2 || Ex[h] < EP_NONE / 2) {
                        v = make_double2(0, 0);
                    } else {
                        const int e = Ea + Ex[h] - 2 * (1022 + 62) + 56;
                        if (e > -900 && e < 900) {
                            const double f = __hiloint2double((e + 1023) << 20, 0);
                            v = make_double2(w[0] * f, w[1] * f);
                        } else {
                            v = make_double2(scalbn(w[0], e), scalbn(w[1], e));
                        }
                    }
                }
                const double2 b = B ? B[row * NC + c] : make_double2(0, 0);
                const double2 r = B ? make_double2(b.x - v.x, b.y - v.y) : v;
                R[row * NC + c] = r;
                if (B) {
                    sr[h] = fma(r.x, r.x, fma(r.y, r.y, sr[h]));
                    sb[h] = fma(b.x, b.x, fma(b.y, b.y, sb[h]));
                }
            }
        }
    }
    if (!B) return;
#pragma unroll
    for (int h = 0; h < 2; h++) {
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            sr[h] += __shfl_xor_sync(0xffffffffu, sr[h], o);
            sb[h] += __shfl_xor_sync(0xffffffffu, sb[h], o);
        }
        if (t == 0) {
            red[0][warp][g + 8 * h] = sr[h];
            red[1][warp][g + 8 * h] = sb[h];
        }
    }
    __syncthreads();
    if (tid < 2 * EP_COLS) {
        const int h = tid / EP_COLS, c = tid % EP_COLS;
        double s = 0;
        for (int w = 0; w < EP_THREADS / 32; w++) s += red[h][w][c];
        if (c0 + c < NC) atomicAdd((h ? nb : nr) + c0 + c, s);
    }
}

// The results that k_product_tc left, by FP64 sums: a warp per row and 16 columns
// (8 of them: four lanes share a column, else two).
constexpr int EP_REST_BLOCKS = 152 * 4, EP_REST_TH = 128;
template <int NC>
__global__ void __launch_bounds__(EP_REST_TH)
    k_product_rest(ProductOp op, const double2 *__restrict__ X, const double2 *__restrict__ B, double2 *__restrict__ R,
                   double *__restrict__ nr, double *__restrict__ nb, const unsigned *__restrict__ rest)
{
    constexpr int CW = NC < EP_COLS ? NC : EP_COLS, NG = NC / CW;
    const int lane = threadIdx.x & 31, col = lane % CW;
    const unsigned n = rest[0], bit = 4 * (col & 7) + (col >> 3);
    double sr[NG], sb[NG];
#pragma unroll
    for (int i = 0; i < NG; i++) sr[i] = sb[i] = 0;
    for (unsigned i = (blockIdx.x * EP_REST_TH + threadIdx.x) / 32; i < n; i += EP_REST_BLOCKS * EP_REST_TH / 32) {
        const unsigned w = rest[2 + 2 * (size_t)i], m = rest[3 + 2 * (size_t)i];
        const long long row = w / 2;
        const int grp = w & 1, c = CW * grp + col, k1 = op.irptr[row + 1];
        double2 v = make_double2(0, 0);
#pragma unroll 8
        for (int k = op.irptr[row] + lane / CW; k < k1; k += 32 / CW) {
            const double2 av = op.at(k), x = X[(long long)op.jcptr[k] * NC + c];
            v.x = fma(av.x, x.x, fma(-av.y, x.y, v.x));
            v.y = fma(av.x, x.y, fma(av.y, x.x, v.y));
        }
#pragma unroll
        for (int o = CW; o < 32; o <<= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if (lane >= CW || !(m >> bit & 1u)) continue;
        const double2 b = B ? B[row * NC + c] : make_double2(0, 0);
        const double2 r = B ? make_double2(b.x - v.x, b.y - v.y) : v;
        R[row * NC + c] = r;
#pragma unroll
        for (int j = 0; j < NG; j++)
            if (j == grp) {
                sr[j] = fma(r.x, r.x, fma(r.y, r.y, sr[j]));
                sb[j] = fma(b.x, b.x, fma(b.y, b.y, sb[j]));
            }
    }
    if (!B || lane >= CW || (blockIdx.x * EP_REST_TH + threadIdx.x) / 32 >= n) return;
#pragma unroll
    for (int j = 0; j < NG; j++) {
        atomicAdd(nr + CW * j + col, sr[j]);
        atomicAdd(nb + CW * j + col, sb[j]);
    }
}

}  // namespace wt3d
