// Basis flush on the tensor cores: x_j += xi_j Pmat_j + sum_l Xc[j][l] V[l],
// p_j = rho_j Pmat_j + sum_l Pc[j][l] V[l], with FP64 accuracy from FP16
// tcgen05 MMAs.
//
// GB300 runs FP64 at ~1.2 TFLOP/s, so the FP64 form of this product is the
// solver's bottleneck.  Here each FP64 operand becomes a signed fixed point
// integer (62 bits for the basis, 63 for the coefficients) against a
// power-of-two scale — per output row for the coefficients, per vector element
// for the basis, after normalising every basis slot by a power of two — cut into
// eight balanced 8-bit digits in [-128, 128], each exact in FP16.  A digit
// product is at most 2^14, so the sum over K = 64 slots of all pairs of one
// diagonal (s + t = d, at most eight pairs) stays below 2^23: each diagonal
// d = 0..7 accumulates exactly in its own FP32 TMEM accumulator.  Diagonals past
// 7 are dropped (their total is below 2^-54 of the row/element scale, the
// accuracy of an FP64 dot product of the same length: the coefficients' 63rd bit
// pays for that; with nine 7-bit digits the bound is the same).
// The epilogue joins the eight exact diagonal sums in 64-bit integer arithmetic
// (keeping T / 2^13 of the 75-bit sum T, rounded: a unit is 2^-56 of the row x
// element scale) and rounds once to FP64; only the
// own-vector terms use the FP64 pipe.  (The digit splitting is the error-free
// splitting of Ozaki, Ogita, Oishi and Rump for matrix products, arranged here
// so that the exact sums fit TMEM.)
//
// One CTA per SM (166 KB of shared memory, all 512 TMEM columns), persistent
// over tiles of 48 vector elements (one panel of the panel-major x_j and p_j
// arrays, whose values for all shifts lie in one contiguous block); 128
// output rows per group of 64 shifts, ordered so that
// TMEM lanes 32q..32q+15 hold the x rows of shifts 16q..16q+15 and lanes
// 32q+16..32q+31 their p rows.  Warps 0-2 make the basis digits of a tile
// into one of two buffers (tile t+1's while the tensor core reads tile t's);
// one thread of warp 3 issues its MMAs (M=128, N up to 256, K=16; 44 per
// tile; coefficient digit slices 0-3 from TMEM, 4-7 from shared memory) into
// eight accumulators, so that the digit builders never wait behind the MMA
// issue; warps 4-15 empty the accumulators into registers first, so that the
// next tile's MMAs run while they round, add the own-vector terms and write x
// and p.  Every wait is bounded: a timeout sets an error flag, the CTA skips
// its remaining work and still frees its TMEM.
//
// What bounds it (clock stamps, n = 2 M, 64 shifts, 59 slots; 13 k clocks per
// tile, of which HBM needs 5.6 k and the tensor core 4 to 5 k): two chains of
// about the same length, both short of issue slots and registers rather than of
// bandwidth.  A builder warp makes 32 digit rows per thread from values that
// wait in registers; an epilogue warp drains, rounds and adds for 16 columns,
// 4.6 k clocks of it the quarter's FP64 pipe.  Each of these shortened a flush
// (n = 2 M, 64 shifts; 256^3 in brackets):
//   eight digits instead of nine (fewer digits, MMAs, accumulators to join) and
//     four coefficient slices in TMEM: 2.21 to 2.17 ms (alone; it frees the
//     registers for the next two);
//   the next tile's basis loads one item at a time, as its registers come
//     free: -5 %;
//   each x addition issued for two columns at once (below): -6 %;
//   together 2.21 to 1.99 ms (17.3 to 15.6).
// The error against quad precision is no larger (rms 5 to 9 % smaller without
// own terms, from rounding T / 2^13 instead of flooring it).
// Tried and not kept: basis values by bulk copies to shared memory (2.3 ms: the
// builders' reads queue behind the MMAs' operands), a sub-tile of 16 columns with
// barriers of its own per epilogue column group (+20 %: smaller MMAs), a fourth
// builder warp (+7 %), prefetching the basis to L2 (no change), rounding all 16
// columns before the first FP64 operation (+25 %).
//
// Only the live shifts are formed: a shift that had converged by the previous
// flush has zero coefficients and own terms (0, 1) since that flush's reset,
// so its rows would come out unchanged.  The rows of a group are the live
// shifts in index order; a group without live shifts does nothing, and the
// epilogue warps of a TMEM quadrant without live rows sit the tiles out.
#include <cuda_fp16.h>
#include <math.h>
#include <stdint.h>

#include "hbk_device.cuh"

using namespace hbk;

namespace {

constexpr int TC_M = 128;
constexpr int TC_N = 48;
constexpr int TC_K = 64;
static_assert(TC_N == HBK_PANEL, "a tile is one panel of x_j and p_j");
constexpr int NDIG = 8;
constexpr int NDIAG = 8;
constexpr int A_SLICE = TC_M * TC_K * 2;  // 16384 B
constexpr int B_SLICE = TC_N * TC_K * 2;  // 6144 B
constexpr int A_BYTES = NDIG * A_SLICE;   // 131072 B (a group's coefficient digits in global memory)
constexpr int B_BYTES = NDIG * B_SLICE;   // 49152 B (one buffer of a tile's basis digits)
// Coefficient digit slices 0 to 3 live in TMEM (columns after the eight
// accumulators: all 512 are used), the other four in shared memory: less for the
// MMAs to read there (2 slices in TMEM: +8 %).  Two basis-digit buffers, so the
// builders write tile t+1's digits while the tensor core works through tile t.
constexpr int A_TMEM_SLICES = 4;
constexpr int A_SMEM_BYTES = (NDIG - A_TMEM_SLICES) * A_SLICE;  // 65536 B
constexpr int A_TCOL = NDIAG * TC_N;                             // first TMEM column of slice 0 (32 per slice)
constexpr int NBUF = 2;                                          // basis-digit buffers
constexpr int BUILD_WARPS = 3;            // warps 0-2: basis digits
constexpr int MMA_WARP = 3;               // warp 3: coefficient copy + MMA issue (one thread)
constexpr int EPI_WARP0 = MMA_WARP + 1;   // first epilogue warp (a multiple of 4: warp w reads TMEM quadrant w % 4)
constexpr int EPI_WARPS = 12;             // warps 4-15: epilogue
constexpr int TC_THREADS = 32 * (BUILD_WARPS + 1 + EPI_WARPS);
constexpr int BUILD_THREADS = 32 * BUILD_WARPS;
constexpr int EPI_COLS = TC_N / (EPI_WARPS / 4);  // 16 columns per epilogue thread
constexpr int ITEMS = (TC_K / 8) * TC_N;          // (slot octet, element) pairs per tile
constexpr int ITEMS_PER = ITEMS / BUILD_THREADS;  // 4
constexpr int TMEM_COLS = 512;
constexpr int SMEM_MISC = 6144;
constexpr int SMEM_BYTES = A_SMEM_BYTES + NBUF * B_BYTES + SMEM_MISC;  // 169984 B
constexpr long long WAIT_LIMIT = 1ll << 26;  // polls of an mbarrier before giving up
constexpr int EXP_NONE = -100000;            // exponent of an all-zero row or column
// sum_s 128 * 2^(56 - 8 s): adding it to a 62-bit signed value makes every
// byte of the sum the balanced digit + 128
constexpr uint64_t DIGIT_BIAS = 0x8080808080808080ull;

static_assert(ITEMS % BUILD_THREADS == 0, "builder items");
static_assert(EPI_WARP0 % 4 == 0 && EPI_WARP0 + EPI_WARPS == TC_THREADS / 32, "epilogue warps: whole quadrant sets");
static_assert((TC_THREADS / 32 - 1 - EPI_WARP0) / 4 == EPI_WARPS / 4 - 1, "epilogue column groups");
static_assert(EPI_COLS % 4 == 0 && TC_N % 8 == 0, "epilogue columns");
static_assert(A_TCOL + 32 * A_TMEM_SLICES <= TMEM_COLS, "accumulators and the TMEM coefficient slices fit TMEM");
static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");
static_assert(A_SMEM_BYTES % 1024 == 0 && B_BYTES % 1024 == 0, "1024-byte aligned operand buffers");

// byte offset of element (row, k) in a K-major, no-swizzle UMMA operand:
// core matrices of 8 rows x 16 bytes; K-adjacent core matrices 128 B apart
// (leading byte offset), 8-row groups 1024 B apart (stride byte offset).
__device__ __forceinline__ uint32_t umma_off(int row, int k) {
    return (uint32_t)(((row >> 3) * 8 + (k >> 3)) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

// shared memory matrix descriptor: start >> 4 (bits 0-13), LBO >> 4 (16-29),
// SBO >> 4 (32-45), fixed 0b001 (46-48), base offset 0, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)(128 >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait; false on timeout or when another warp has already failed
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, const int *fail) {
    for (long long i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try(bar, parity)) return true;
        if (i > 64) {
            if ((i & 1023) == 0 && *(const volatile int *)fail) return false;
            __nanosleep(64);
        }
    }
    return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// exponent e with |v| < 2^e for a nonzero double, from its bits
__device__ __forceinline__ int exp_of_bits(uint64_t bits) {
    const int eb = (int)((bits >> 52) & 0x7ff);
    const uint64_t frac = bits & ((1ull << 52) - 1);
    if (eb) return eb - 1022;
    return (64 - __clzll((long long)frac)) - 1074;
}

// v * 2^(62 - scale) truncated toward zero, as a two's complement integer
// (|v| < 2^scale, so the result is below 2^62), plus DIGIT_BIAS.  The
// significand M < 2^53 is placed at M 2^10 and shifted right by
// r = 1023 + scale - max(eb, 1) >= 0 (|v| < 2^scale bounds the left shift
// M 2^(62 - scale + eb - 1075) by 2^10); M 2^10 < 2^63, so a shift by 63
// stands for every longer one.
__device__ __forceinline__ uint64_t biased62(uint64_t bits, int scale) {
    const uint32_t hi = (uint32_t)(bits >> 32);
    const int eb = (int)((hi >> 20) & 0x7ffu);
    const uint32_t mh = (hi & 0xfffffu) | (eb ? 1u << 20 : 0u);
    const uint64_t M = ((uint64_t)mh << 32) | (uint32_t)bits;
    const int r = 1023 + scale - max(eb, 1);
    const uint64_t q = (M << 10) >> min(r, 63);
    const uint64_t sg = (uint64_t)((int64_t)bits >> 63);  // 0 or all ones
    return (q ^ sg) + DIGIT_BIAS + (hi >> 31);            // -q = ~q + 1
}

// v * 2^(63 - scale) truncated toward zero (|v| < 2^scale, so r >= 1 and the
// magnitude is below 2^63): a bit more than biased62, for the coefficients,
// whose digit 0 then reaches 128
__device__ __forceinline__ int64_t fixed63(uint64_t bits, int scale) {
    const int eb = (int)((bits >> 52) & 0x7ffu);
    const uint64_t M = (bits & ((1ull << 52) - 1)) | (eb ? 1ull << 52 : 0ull);
    const int64_t q = (int64_t)((M << 11) >> min(1023 + scale - max(eb, 1), 63));
    return (int64_t)bits < 0 ? -q : q;
}

// balanced digits s (weight 2^(56 - 8 s)) of two biased values as an FP16 pair:
// FP16 0x6400 + e is 1024 + e for e = 0..255 (ten fraction bits), so one packed
// subtraction of 1152 leaves the digits e - 128, exact
template <int S>
__device__ __forceinline__ uint32_t digit_pair(uint64_t U0, uint64_t U1) {
    constexpr uint32_t b = 3 - (S & 3);  // byte of the upper (S < 4) or lower word
    const uint32_t x0 = (uint32_t)(U0 >> (S < 4 ? 32 : 0)), x1 = (uint32_t)(U1 >> (S < 4 ? 32 : 0));
    const uint32_t e = (__byte_perm(x0, x1, b | (b << 4) | ((4 + b) << 8) | ((4 + b) << 12)) & 0x00ff00ffu) | 0x64006400u;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&e), __half2half2(__ushort_as_half(0x6480)));
    return *reinterpret_cast<const uint32_t *>(&h);
}

// 8 consecutive slots of one element (Us[0..7]) -> one 16-byte row of a core
// matrix in every digit slice
template <int S>
__device__ __forceinline__ void store_digits(unsigned char *sB, uint32_t off, const uint64_t *Us) {
    uint4 w;
    w.x = digit_pair<S>(Us[0], Us[1]);
    w.y = digit_pair<S>(Us[2], Us[3]);
    w.z = digit_pair<S>(Us[4], Us[5]);
    w.w = digit_pair<S>(Us[6], Us[7]);
    *reinterpret_cast<uint4 *>(sB + S * B_SLICE + off) = w;
    if constexpr (S + 1 < NDIG) store_digits<S + 1>(sB, off, Us);
}

// 32 x 32 + 64 -> 64-bit multiply-add
__device__ __forceinline__ long long madw(int a, int b, long long c) {
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}

// T / 2^13 of the exact diagonal sum T = sum_d D_d 2^(8 (7 - d)), to within 0.54
// units (rounded: 2048 more halves before the shift).  |D_d| <= (d + 1/2) 2^20 (|digit| <= 128 on both sides, 64 for the
// basis' digit 0).  Up to D_3 (below 2^22) an FP32 add of 1.5 2^23 leaves the
// integer in the sum's low bits; the larger ones take 1.5 2^24, which rounds to
// an even integer: D_4's and D_5's odd unit goes to the next diagonal (256 units
// there; exact), D_6's and D_7's is dropped (2^-5 of the result's unit, which is
// 2^-56 of the row x element scale).  Conversion instructions instead: +9 %.
// Pairs D_2i 2^8 + D_2i+1 fit 32 bits, |T| < 2^75.1 and the result 64.
constexpr float MAGIC = 12582912.0f, MAGIC2 = 25165824.0f;  // 1.5 2^23, 1.5 2^24
constexpr uint32_t MAGIC_BITS = 0x4B400000u, MAGIC2_BITS = 0x4BC00000u;
__device__ __forceinline__ int pair_sum(float a, float b, uint32_t bias, uint32_t more = 0) {
    return (int)(__float_as_uint(a) * 256u + (__float_as_uint(b) - (bias * 257u - more)));
}
__device__ __forceinline__ long long diag_sum(const float (&D)[NDIAG]) {
    const int h0 = pair_sum(D[0] + MAGIC, D[1] + MAGIC, MAGIC_BITS), h1 = pair_sum(D[2] + MAGIC, D[3] + MAGIC, MAGIC_BITS);
    const float f4 = D[4] + MAGIC2;
    const float d5 = fmaf(D[4] - (f4 - MAGIC2), 256.0f, D[5]), f5 = d5 + MAGIC2;
    const float f6 = fmaf(d5 - (f5 - MAGIC2), 256.0f, D[6]) + MAGIC2, f7 = D[7] + MAGIC2;
    const int h2 = pair_sum(f4, f5, MAGIC2_BITS), h3 = pair_sum(f6, f7, MAGIC2_BITS, 2048u);  // halves
    const long long t = madw(h1, 1 << 19, madw(h2, 1 << 4, (long long)(h3 >> 12)));
    return t + (long long)((unsigned long long)(long long)h0 << 35);
}

// T 2^k rounded to FP64: round half up on the 64-bit magnitude, whose leading
// bit is normalised to bit 63 (error <= 0.5 ulp of the result).  The common
// cases are T = 0 (every column of a row without coefficients) and a bit set in
// T's upper word with a normal result; the rest (results near the ends of the
// range) is out of line.
__device__ __noinline__ double join_rest(long long T, int k) {
    const unsigned long long sg = (unsigned long long)(T >> 63);
    const unsigned long long a = ((unsigned long long)T ^ sg) - sg;
    if (a == 0) return 0.0;
    const int z = __clzll((long long)a);
    const unsigned long long W = a << z;
    const unsigned long long mant = (W >> 11) + ((W >> 10) & 1);  // 2^52 .. 2^53 (carries into the exponent)
    const int ebm1 = 63 - z + k + 1022;                             // biased exponent - 1
    if ((unsigned)ebm1 > 2044u) {
        if (ebm1 < 0) return sg ? -0.0 : 0.0;  // below the normal range: negligible here
        return sg ? -INFINITY : INFINITY;
    }
    const unsigned long long bits = ((unsigned long long)ebm1 << 52) + mant;
    return __longlong_as_double((long long)(bits | (sg << 63)));
}
__device__ __forceinline__ double join_t(long long T, int k) {
    const unsigned long long sg = (unsigned long long)(T >> 63);
    const unsigned long long a = ((unsigned long long)T ^ sg) - sg;
    const unsigned ah = (unsigned)(a >> 32);
    const int z = __clz((int)ah);
    const int ebm1 = 1085 - z + k;
    if (ah == 0 ? (unsigned)a != 0u : (unsigned)ebm1 > 2044u) return join_rest(T, k);
    // (z < 32 where ah is not 0; the shifts of a row of zeros are not used)
    const unsigned wl = (unsigned)a << (z & 31), wh = __funnelshift_l((unsigned)a, ah, z);
    const unsigned long long mant =
        (((unsigned long long)(wh >> 11) << 32) | __funnelshift_r(wl, wh, 11)) + ((wl >> 10) & 1u);
    const unsigned hi = ah ? (unsigned)(mant >> 32) + ((unsigned)ebm1 << 20) : 0u;
    return __hiloint2double((int)(hi | ((unsigned)sg & 0x80000000u)), (int)(unsigned)mant);
}

// one 32-byte sector per lane and instruction (x and p rows are read and
// written 4 doubles at a time; 16-byte pieces of a sector written by separate
// instructions cost partial-sector traffic)
__device__ __forceinline__ void ld_sector(const double *p, double &a, double &b, double &c, double &d) {
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p));
}
__device__ __forceinline__ void st_sector(double *p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

struct TcArgs {
    const double *V;      // basis [slots][ld]
    size_t ld;
    unsigned n;
    int L;                // slots in use (<= 64)
    const unsigned long long *slot_max;  // bits of max |V[l]| per slot
    const unsigned char *aimg;           // per group: 8 digit slices of the 128 x 64 coefficient block
    const int *rowexp;    // per group: [128]
    const double *rown;   // per group: [128] own-term scalar (xi for x rows, rho for p rows)
    double *X, *Pmat;     // panel-major, m systems
    int m, keep_p;
    const int *live;      // [0]: number of live shifts; [1 ..]: their indices, ascending
    int *err;
};

// live shifts: not converged (conv_k == 0) or converged after iteration
// k_last (the last one the previous flush covered); one warp, index order
__global__ void k_flush_live(const int *__restrict__ conv_k, int m, int k_last, int *live) {
    int cnt = 0;
    for (int base = 0; base < m; base += 32) {
        const int j = base + (int)threadIdx.x;
        bool on = false;
        if (j < m) {
            int c = conv_k ? conv_k[j] : 0;
            c = c < 0 ? -c : c;  // a shift that broke down at k stopped there like a converged one
            on = c == 0 || c > k_last;
        }
        const unsigned b = __ballot_sync(0xffffffffu, on);
        if (on) live[1 + cnt + __popc(b & ((1u << threadIdx.x) - 1u))] = j;
        cnt += __popc(b);
    }
    if (threadIdx.x == 0) live[0] = cnt;
}

// ---- per-slot max |V[l]| (bits of a non-negative double order as integers)
__global__ void __launch_bounds__(NT) k_slot_max(const double *__restrict__ V, size_t ld, unsigned n, int L,
                                                 unsigned long long *slot_max) {
    const int l = blockIdx.y;
    if (l >= L) return;
    const double *v = V + (size_t)l * ld;
    unsigned long long mx = 0;
    for (size_t i = blockIdx.x * (size_t)NT + threadIdx.x; i < n; i += (size_t)gridDim.x * NT) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(v[i]) & 0x7FFFFFFFFFFFFFFFull;
        mx = b > mx ? b : mx;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = t > mx ? t : mx;
    }
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(slot_max + l, mx);
}

// slot maxima from the partial maxima kept by the kernels that wrote the slots
// (one warp per slot)
__global__ void k_fold_slot_max(const unsigned long long *__restrict__ part, int L, unsigned long long *slot_max) {
    const int l = blockIdx.x;
    if (l >= L) return;
    unsigned long long m = part[(size_t)l * HBK_SLOT_SPREAD + threadIdx.x];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
        m = t > m ? t : m;
    }
    if (threadIdx.x == 0) slot_max[l] = m;
}

// TMEM lane / A row r of a group -> (x or p, shift within the group)
__device__ __forceinline__ int row_which(int r) { return (r >> 4) & 1; }
__device__ __forceinline__ int row_shift(int r) { return ((r >> 5) << 4) | (r & 15); }

// ---- coefficient digits: one block per output row, one thread per slot
__global__ void __launch_bounds__(TC_K) k_flush_prep(const double *__restrict__ Xc, const double *__restrict__ Pc,
                                                     int cap, const double *__restrict__ own, int L,
                                                     const unsigned long long *__restrict__ slot_max,
                                                     const int *__restrict__ live, unsigned char *aimg, int *rowexp,
                                                     double *rown) {
    __shared__ unsigned long long s_max[2];
    const int r = blockIdx.x, g = blockIdx.y, l = threadIdx.x;
    const int which = row_which(r), pos = g * 64 + row_shift(r);
    if (g * 64 >= live[0]) return;  // the whole group is idle
    const int j = pos < live[0] ? live[1 + pos] : -1;
    double a = 0.0;
    if (j >= 0 && l < L) {
        const double c = (which ? Pc : Xc)[(size_t)j * cap + l];
        const unsigned long long sm = slot_max[l];
        a = sm ? ldexp(c, exp_of_bits(sm)) : 0.0;  // fold the slot's scale into the coefficient
    }
    unsigned long long b = (unsigned long long)__double_as_longlong(fabs(a));
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o);
        b = t > b ? t : b;
    }
    if ((l & 31) == 0) s_max[l >> 5] = b;
    __syncthreads();
    const unsigned long long rmax = s_max[0] > s_max[1] ? s_max[0] : s_max[1];
    const int E = rmax ? exp_of_bits(rmax) : EXP_NONE;
    int64_t q = (rmax && a != 0.0) ? fixed63((uint64_t)__double_as_longlong(a), E) : 0;
    unsigned char *img = aimg + (size_t)g * A_BYTES;
    const uint32_t off = umma_off(r, l);
#pragma unroll
    for (int s = NDIG - 1; s >= 0; --s) {
        // balanced digit: the low byte in [-128, 127], its borrow to the next
        const int d = s ? (int)(signed char)(q & 255) : (int)q;
        q = (q >> 8) + ((q >> 7) & 1);
        *reinterpret_cast<__half *>(img + (size_t)s * A_SLICE + off) = __int2half_rn(d);
    }
    if (l == 0) {
        rowexp[g * TC_M + r] = E;
        rown[g * TC_M + r] = (j >= 0) ? own[2 * (size_t)j + which] : 0.0;
    }
}

// ---- the tensor-core flush
__global__ void __launch_bounds__(TC_THREADS, 1) k_flush_tc(TcArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *sA = smem;                 // coefficient digit slices 4 .. 7
    unsigned char *sB = smem + A_SMEM_BYTES;  // NBUF basis-digit buffers, tile it in buffer it % 2
    unsigned char *misc = smem + A_SMEM_BYTES + NBUF * B_BYTES;
    // Tiles alternate between the two basis-digit buffers, and the barriers
    // that hand a buffer between the builders and the tensor core come in
    // pairs (one per buffer): a parity wait is only sound while the waiter is
    // at most one phase behind, and the builders now run two tiles ahead.
    uint64_t *bar_a = reinterpret_cast<uint64_t *>(misc);           // coefficient digits landed
    uint64_t *bar_full = reinterpret_cast<uint64_t *>(misc + 8);     // [2] basis digits of a tile written
    uint64_t *bar_mma = reinterpret_cast<uint64_t *>(misc + 24);     // [2] MMAs of a tile done
    uint64_t *bar_ready = reinterpret_cast<uint64_t *>(misc + 40);   // MMAs issued (orders s_F for the epilogue)
    uint64_t *bar_tfree = reinterpret_cast<uint64_t *>(misc + 48);   // accumulators read out
    uint64_t *bar_cexp = reinterpret_cast<uint64_t *>(misc + 56);    // builders' partial exponents written
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(misc + 64);
    int *s_fail = reinterpret_cast<int *>(misc + 68);
    int *s_slotexp = reinterpret_cast<int *>(misc + 128);            // [64]
    int *s_cexp = reinterpret_cast<int *>(misc + 384);               // [2][8][48] per slot octet
    int *s_F = reinterpret_cast<int *>(misc + 3456);                 // [4][48] element exponents, ring
    int *s_rowexp = reinterpret_cast<int *>(misc + 4224);            // [128]
    double *s_rown = reinterpret_cast<double *>(misc + 4736);        // [128], ends at 5760

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = blockIdx.y;
    // live rows of this group; the whole CTA leaves (before any barrier or
    // TMEM allocation) when there are none
    const int n_live = a.live[0];
    const int g_live = n_live - 64 * g;
    if (g_live <= 0) return;
    const int live_quads = g_live >= 64 ? 4 : (g_live + 15) / 16;  // TMEM quadrants with a live row

    if (tid == 0) {
        mbar_init(bar_a, 1);
        mbar_init(bar_full, BUILD_THREADS);
        mbar_init(bar_full + 1, BUILD_THREADS);
        mbar_init(bar_mma, 1);
        mbar_init(bar_mma + 1, 1);
        mbar_init(bar_ready, 1);
        mbar_init(bar_tfree, (EPI_WARPS / 4) * live_quads);
        mbar_init(bar_cexp, BUILD_THREADS);
        *s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid < TC_K) {
        const unsigned long long sm = a.slot_max[tid < a.L ? tid : a.L - 1];  // (past L: slot L - 1 again)
        s_slotexp[tid] = sm ? exp_of_bits(sm) : 0;
    }
    if (tid < TC_M) {
        s_rowexp[tid] = a.rowexp[g * TC_M + tid];
        s_rown[tid] = a.rown[g * TC_M + tid];
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    // coefficient digit slices 0 .. 3 into TMEM: lane r holds row r, each
    // 32-bit column two consecutive k (the lower k in the low half), slice s
    // at columns A_TCOL + 32 s ..  Warps 4-7 each write their own quadrant.
    if (warp >= EPI_WARP0 && warp < EPI_WARP0 + 4) {
        const int r = 32 * (warp & 3) + lane;
        const unsigned char *src = a.aimg + (size_t)g * A_BYTES;
#pragma unroll
        for (int s = 0; s < A_TMEM_SLICES; ++s) {
            uint32_t col[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                const uint32_t lo = *reinterpret_cast<const unsigned short *>(src + s * A_SLICE + umma_off(r, 2 * c));
                const uint32_t hi = *reinterpret_cast<const unsigned short *>(src + s * A_SLICE + umma_off(r, 2 * c + 1));
                col[c] = lo | (hi << 16);
            }
            const uint32_t taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(A_TCOL + 32 * s);
            asm volatile(
                "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
                "r"(col[0]), "r"(col[1]), "r"(col[2]), "r"(col[3]), "r"(col[4]), "r"(col[5]), "r"(col[6]),
                "r"(col[7]), "r"(col[8]), "r"(col[9]), "r"(col[10]), "r"(col[11]), "r"(col[12]), "r"(col[13]),
                "r"(col[14]), "r"(col[15]), "r"(col[16]), "r"(col[17]), "r"(col[18]), "r"(col[19]), "r"(col[20]),
                "r"(col[21]), "r"(col[22]), "r"(col[23]), "r"(col[24]), "r"(col[25]), "r"(col[26]), "r"(col[27]),
                "r"(col[28]), "r"(col[29]), "r"(col[30]), "r"(col[31])
                : "memory");
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    const unsigned n = a.n;
    const unsigned ntiles = (n + TC_N - 1) / TC_N;
    const size_t ld = a.ld;
    bool a_ok = true;
    int issued = 0;  // the MMA thread: MMA batches committed

    if (warp < BUILD_WARPS) {
        // ---- builders: the basis digits of every tile.  They never issue
        // MMAs, so their work for the next tile (loads, exponents) runs while
        // the tensor core works through the current one.
        // item (octet o, element i): slots 8o..8o+7 of element i0 + i
        int io[ITEMS_PER], ii[ITEMS_PER];
#pragma unroll
        for (int u = 0; u < ITEMS_PER; ++u) {
            const int it = tid + BUILD_THREADS * u;
            io[u] = it / TC_N;
            ii[u] = it % TC_N;
        }
        // slots past L read as zero (with slot L - 1's exponent they do not move
        // the element's), elements past n as element n - 1 (never stored)
        double v[ITEMS_PER][8];
        const double *vcol[ITEMS_PER];
        uint32_t wmax[ITEMS_PER];
#pragma unroll
        for (int u = 0; u < ITEMS_PER; ++u) {
            const int l0 = min(8 * io[u], a.L - 1);
            vcol[u] = a.V + (size_t)l0 * ld;
            wmax[u] = (uint32_t)min(7, a.L - 1 - l0);  // (an octet past L: slot L - 1 again, against zero digits)
        }
        const uint32_t ld32 = (uint32_t)ld;
        auto load_item = [&](int u, unsigned t) {
            const double *p = vcol[u] + min(t * TC_N + ii[u], n - 1);
#pragma unroll
            for (uint32_t w = 0; w < 8; ++w) v[u][w] = w <= wmax[u] ? __ldcs(p + (uint64_t)w * ld32) : 0.0;
        };
        int it = 0;
        if (blockIdx.x < ntiles) {
#pragma unroll
            for (int u = 0; u < ITEMS_PER; ++u) load_item(u, blockIdx.x);
        }
        for (unsigned t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
            if (*(volatile int *)s_fail) break;
            // phase A (overlaps the previous tile's MMAs): element exponents;
            // s_cexp alternates between two buffers
            int *cexp = s_cexp + (it & 1) * ITEMS;
            int em[ITEMS_PER];
#pragma unroll
            for (int u = 0; u < ITEMS_PER; ++u) {
                const int4 *sx = reinterpret_cast<const int4 *>(s_slotexp + 8 * io[u]);
                const int4 sa = sx[0], sb = sx[1];
                const int se[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
                int e = EXP_NONE;
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    // |v| < 2^(eb - 1022) for every v, zero and subnormals included
                    const int eb = (__double2hiint(v[u][w]) >> 20) & 0x7ff;
                    e = max(e, eb - se[w]);
                }
                e -= 1022;
                em[u] = e;
                cexp[io[u] * TC_N + ii[u]] = e;
            }
            // (an mbarrier, not a named barrier: a builder that gave up must not hang the others)
            mbar_arrive(bar_cexp);
            if (!mbar_wait(bar_cexp, it & 1, s_fail)) {
                atomicExch(s_fail, 1);
                break;
            }
            int Fv[ITEMS_PER];
#pragma unroll
            for (int u = 0; u < ITEMS_PER; ++u) {
                int F = em[u];
#pragma unroll
                for (int o = 0; o < TC_K / 8; ++o) F = max(F, cexp[o * TC_N + ii[u]]);
                Fv[u] = F;
            }
            // phase B: this tile's digit buffer is free once the MMAs of the
            // tile before the previous one (the same buffer) are done
            if (it >= NBUF && !mbar_wait(bar_mma + (it & 1), ((it >> 1) - 1) & 1, s_fail)) {
                atomicExch(s_fail, 1);
                break;
            }
            unsigned char *sBt = sB + (it & 1) * B_BYTES;
#pragma unroll
            for (int u = 0; u < ITEMS_PER; ++u) {
                const int4 *sx = reinterpret_cast<const int4 *>(s_slotexp + 8 * io[u]);
                const int4 sa = sx[0], sb = sx[1];
                const int se[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
                uint64_t U[8];
#pragma unroll
                for (int w = 0; w < 8; ++w)
                    U[w] = biased62((uint64_t)__double_as_longlong(v[u][w]), Fv[u] + se[w]);
                if (io[u] == 0) s_F[(it & 3) * TC_N + ii[u]] = Fv[u];
                store_digits<0>(sBt, umma_off(ii[u], 8 * io[u]), U);
                // the next tile's values take this item's registers
                if (t + gridDim.x < ntiles) load_item(u, t + gridDim.x);
            }
            // digits written by threads must be visible to the tensor core (async proxy)
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(bar_full + (it & 1));
        }
    } else if (warp == MMA_WARP) {
        // ---- one thread loads the coefficient digits and issues every MMA
        if (lane == 0) {
            // the coefficient digits of this group: one bulk copy per slice
            // the coefficient digit slices kept in shared memory (4 .. 7)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar_a)),
                         "r"((uint32_t)A_SMEM_BYTES)
                         : "memory");
            const unsigned char *src = a.aimg + (size_t)g * A_BYTES;
            for (int s = A_TMEM_SLICES; s < NDIG; ++s)
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        smem_u32(sA + (s - A_TMEM_SLICES) * A_SLICE)),
                    "l"(src + (size_t)s * A_SLICE), "r"((uint32_t)A_SLICE), "r"(smem_u32(bar_a))
                    : "memory");
            a_ok = mbar_wait(bar_a, 0, s_fail);
            if (!a_ok) atomicExch(s_fail, 1);
            const uint64_t ad0 = umma_desc(smem_u32(sA));
            int it = 0;
            for (unsigned t = blockIdx.x; t < ntiles && a_ok; t += gridDim.x, ++it) {
                const uint64_t bd0 = umma_desc(smem_u32(sB + (it & 1) * B_BYTES));
                bool ok = mbar_wait(bar_full + (it & 1), (it >> 1) & 1, s_fail);
                // the previous tile's accumulators must have been read out
                if (ok && it > 0) ok = mbar_wait(bar_tfree, (it - 1) & 1, s_fail);
                if (!ok) {
                    atomicExch(s_fail, 1);
                    break;
                }
                tc_fence_after();
                // diagonal d accumulates in columns [48 d, 48 d + 48).  The basis
                // digit slices lie one after another along N, so one MMA of
                // coefficient slice s against basis rows 0 .. 48 (8 - s) - 1,
                // written from column 48 s on, adds A_s B_t to diagonal s + t
                // for every t <= 7 - s (in two MMAs where N would pass 256).
#pragma unroll
                for (int kk = 0; kk < TC_K / 16; ++kk) {
#pragma unroll
                    for (int s = 0; s < NDIG; ++s) {
                        const int ntot = TC_N * (NDIG - s);
#pragma unroll
                        for (int part = 0; part * 256 < ntot; ++part) {
                            const int nn = ntot - part * 256 < 256 ? ntot - part * 256 : 256;
                            // kind::f16 instruction descriptor: D = F32, A = B = F16 (0), both
                            // K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
                            const uint32_t idesc = (1u << 4) | ((uint32_t)(nn >> 3) << 17) |
                                                   ((uint32_t)(TC_M >> 4) << 24);
                            // start-address field: (offset >> 4) adds without carry (smem < 256 KB)
                            const uint64_t bd = bd0 + (uint64_t)((part * 256 / 8 * 1024 + kk * 256) >> 4);
                            const uint32_t acc = (kk | s) ? 1u : 0u;
                            const uint32_t dt = tmem + (uint32_t)(TC_N * s + 256 * part);
                            if (s < A_TMEM_SLICES) {  // A from TMEM: K = 16 is 8 columns
                                const uint32_t at = tmem + (uint32_t)(A_TCOL + 32 * s + 8 * kk);
                                asm volatile(
                                    "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
                                    " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(dt),
                                    "r"(at), "l"(bd), "r"(idesc), "r"(acc)
                                    : "memory");
                            } else {
                                const uint64_t ad =
                                    ad0 + (uint64_t)(((s - A_TMEM_SLICES) * A_SLICE + kk * 256) >> 4);
                                asm volatile(
                                    "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
                                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dt),
                                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                                    : "memory");
                            }
                        }
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(bar_mma + (it & 1)))
                             : "memory");
                ++issued;
                mbar_arrive(bar_ready);
            }
        }
        __syncwarp();
    } else if ((warp & 3) < live_quads) {
        // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31, columns
        // 16 c .. 16 c + 15 with c = (w - 4) / 4; lane u < 16 holds the x row
        // of live shift 16 (w % 4) + u of the group, lane u + 16 its p row.
        // (Warps of a quadrant without live rows skip this loop; the
        // accumulator-free barrier counts only the others.)
        const int q = warp & 3, cg = (warp - EPI_WARP0) >> 2;
        const int r = 32 * q + lane;
        const int which = row_which(r);
        const int pos = g * 64 + row_shift(r);
        const bool live = pos < n_live;
        const int j = live ? a.live[1 + pos] : 0;
        const bool store = live && (which == 0 || a.keep_p);
        const int E = s_rowexp[r];
        const double own = s_rown[r];
        const uint32_t tbase = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(cg * EPI_COLS);
        // A lane pair (u, u + 16) works on one system's piece of a panel
        // (columns 16 cg .. 16 cg + 15): p row and x row, four 32-byte sectors
        // each, consecutive panels m * 48 values apart.  Both lanes need the
        // old p (one load serves both); the additions to x are shared out, the
        // x lane takes sectors 0 and 2, the p lane 1 and 3, so that an FP64 add
        // is issued for two columns at a time.
        const size_t piece = (size_t)j * TC_N + cg * EPI_COLS;
        const double *const pp = live && a.Pmat ? a.Pmat + piece : nullptr;
        double *const xp = live ? a.X + piece + 4 * which : nullptr;
        const size_t pstride = (size_t)a.m * TC_N;
        // x and p values of a tile, loaded one tile ahead: the loads are in
        // flight while the warp waits for that tile's MMAs and drains them.
        double pv[EPI_COLS], xv[EPI_COLS / 2];
        auto load_pv = [&](unsigned t) {
            const unsigned c0 = t * TC_N + cg * EPI_COLS;
            const double *ps = pp ? pp + (size_t)t * pstride : nullptr;
            const double *xs = xp ? xp + (size_t)t * pstride : nullptr;
            const bool full = c0 + EPI_COLS <= n;
            if (ps && full) {
#pragma unroll
                for (int u = 0; u < EPI_COLS; u += 4) ld_sector(ps + u, pv[u], pv[u + 1], pv[u + 2], pv[u + 3]);
            } else {
#pragma unroll
                for (int u = 0; u < EPI_COLS; ++u) pv[u] = (ps && c0 + u < n) ? ps[u] : 0.0;
            }
            if (xs && full) {
#pragma unroll
                for (int u = 0; u < EPI_COLS / 2; u += 4) ld_sector(xs + 2 * u, xv[u], xv[u + 1], xv[u + 2], xv[u + 3]);
            } else {
#pragma unroll
                for (int u = 0; u < EPI_COLS / 2; ++u) {
                    const int col = 2 * (u & 4) + (u & 3);
                    xv[u] = (xs && c0 + 4 * which + col < n) ? xs[col] : 0.0;
                }
            }
        };
        if (blockIdx.x < ntiles) load_pv(blockIdx.x);
        int it = 0;
        for (unsigned t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
            // the warp decides as one: tcgen05.ld and the shuffles below are warp-collective
            bool bad = *(volatile int *)s_fail != 0;
            if (!bad)
                bad = !mbar_wait(bar_ready, it & 1, s_fail) || !mbar_wait(bar_mma + (it & 1), (it >> 1) & 1, s_fail);
            if (__any_sync(0xffffffffu, bad)) {
                if (lane == 0) atomicExch(s_fail, 1);
                break;
            }
            tc_fence_after();
            // exact diagonal sums -> T / 2^13
            long long T[EPI_COLS];
#pragma unroll
            for (int c2 = 0; c2 < EPI_COLS; c2 += 2) {
                float dv[NDIAG][2];
#pragma unroll
                for (int d = 0; d < NDIAG; ++d)
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
                                 : "=f"(dv[d][0]), "=f"(dv[d][1])
                                 : "r"(tbase + (uint32_t)(d * TC_N + c2)));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    float D[NDIAG];
#pragma unroll
                    for (int d = 0; d < NDIAG; ++d) D[d] = dv[d][u];
                    T[c2 + u] = diag_sum(D);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_tfree);

            const unsigned c0 = t * TC_N + cg * EPI_COLS;
            const bool full = c0 + EPI_COLS <= n;
            const int *Fc = s_F + (it & 3) * TC_N + cg * EPI_COLS;
            double *const pd = store && which && a.Pmat ? a.Pmat + piece + (size_t)t * pstride : nullptr;
            double *const xd = xp ? xp + (size_t)t * pstride : nullptr;
            // one pass per two sectors: round, own-vector terms, store
#pragma unroll
            for (int u = 0; u < EPI_COLS; u += 8) {
                double y[8], xn[4];
#pragma unroll
                for (int h = 0; h < 8; ++h)  // (a row of zero coefficients has T = 0)
                    y[h] = fma(own, pv[u + h], join_t(T[u + h], E + Fc[u + h] - 56));
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const double z = __shfl_xor_sync(0xffffffffu, y[4 + h], 16);
                    xn[h] = xv[u / 2 + h] + (which ? z : y[h]);
                }
                if (full) {
                    if (pd) {
                        st_sector(pd + u, y[0], y[1], y[2], y[3]);
                        st_sector(pd + u + 4, y[4], y[5], y[6], y[7]);
                    }
                    if (xd) st_sector(xd + u, xn[0], xn[1], xn[2], xn[3]);
                } else {
#pragma unroll
                    for (int h = 0; h < 8; ++h)
                        if (pd && c0 + u + h < n) pd[u + h] = y[h];
#pragma unroll
                    for (int h = 0; h < 4; ++h)
                        if (xd && c0 + u + 4 * which + h < n) xd[u + h] = xn[h];
                }
            }
            if (t + gridDim.x < ntiles) load_pv(t + gridDim.x);
        }
    }
    // every path ends here: let copies and MMAs still in flight after a
    // timeout finish (bounded), then free TMEM
    __syncthreads();
    if (tid == 32 * MMA_WARP && *(volatile int *)s_fail) {
        int dummy = 0;
        if (!a_ok) mbar_wait(bar_a, 0, &dummy);
        if (issued > 0) mbar_wait(bar_mma + ((issued - 1) & 1), ((issued - 1) >> 1) & 1, &dummy);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    if (tid == 0 && *s_fail) atomicExch(a.err, 1);
}

}  // namespace

extern "C" {

size_t hbk_flush_tc_workspace_bytes(int m) {
    const int groups = (m + 63) / 64;
    return 256 + 64 * sizeof(unsigned long long) + (size_t)groups * (A_BYTES + TC_M * (sizeof(int) + sizeof(double))) +
           sizeof(int) * ((size_t)(m > 0 ? m : 0) + 1);
}

int hbk_flush_tc_max_slots(void) { return TC_K; }

static int g_test_error = 0;
void hbk_flush_tc_test_error(int on) { g_test_error = on ? 1 : 0; }

// x_j (and p_j when keep_p) from the first L basis slots on the tensor cores,
// for the live shifts only: conv_k[j] == 0 or conv_k[j] > k_last (conv_k
// NULL: every shift).  slot_max: bits of each slot's max |value| (NULL:
// computed here; else [L][HBK_SLOT_SPREAD] partial maxima).  V: [L][ld] slots; X, Pmat: panel-major (HBK_PANEL),
// m systems, 32-byte aligned; ws: device workspace of
// hbk_flush_tc_workspace_bytes(m), err: device int.
int hbk_flush_tc_run_live(const double *V, size_t ld, unsigned n, int L, const double *Xc, const double *Pc, int cap,
                          const double *own, int m, double *X, double *Pmat, int keep_p, const int *conv_k,
                          int k_last, const unsigned long long *slot_max_in, void *ws, int *err, cudaStream_t st) {
    // x and p pieces are accessed in 32-byte sectors: 32-byte aligned arrays
    if (L > TC_K || L < 1 || m < 1 || n == 0 || ld < n || ((uintptr_t)X & 31) || ((uintptr_t)Pmat & 31))
        return (int)cudaErrorInvalidValue;
    const int groups = (m + 63) / 64;
    unsigned char *w = (unsigned char *)ws;
    unsigned long long *slot_max = (unsigned long long *)(w + 256);
    unsigned char *aimg = w + 256 + 64 * sizeof(unsigned long long);
    int *rowexp = (int *)(aimg + (size_t)groups * A_BYTES);
    double *rown = (double *)(rowexp + groups * TC_M);
    int *live = (int *)(rown + (size_t)groups * TC_M);
    cudaError_t e = cudaSuccess;
    k_flush_live<<<1, 32, 0, st>>>(conv_k, m, k_last, live);
    if (slot_max_in) {
        static_assert(HBK_SLOT_SPREAD == 32, "one warp folds a slot's partial maxima");
        k_fold_slot_max<<<L, 32, 0, st>>>(slot_max_in, L, slot_max);
    } else {
        if ((e = cudaMemsetAsync(slot_max, 0, 64 * sizeof(unsigned long long), st))) return (int)e;
        dim3 gs(grid_for(n, 16) < 64 ? grid_for(n, 16) : 64, L);
        k_slot_max<<<gs, NT, 0, st>>>(V, ld, n, L, slot_max);
    }
    k_flush_prep<<<dim3(TC_M, groups), TC_K, 0, st>>>(Xc, Pc, cap, own, L, slot_max, live, aimg, rowexp, rown);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    static unsigned attr_set = 0;  // one bit per device
    if (dev < 32 && !(attr_set & (1u << dev))) {
        e = cudaFuncSetAttribute(k_flush_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e) return (int)e;
        attr_set |= 1u << dev;
    }
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const unsigned ntiles = (n + TC_N - 1) / TC_N;
    const unsigned gx = ntiles < (unsigned)sms ? ntiles : (unsigned)sms;
    TcArgs args{V, ld, n, L, slot_max, aimg, rowexp, rown, X, Pmat, m, keep_p, live, err};
    k_flush_tc<<<dim3(gx, groups), TC_THREADS, SMEM_BYTES, st>>>(args);
    if ((e = cudaGetLastError())) return (int)e;
    if (g_test_error) {
        g_test_error = 0;
        e = cudaMemsetAsync(err, 1, sizeof(int), st);
    }
    return (int)e;
}

// device address of the live-shift count of the last hbk_flush_tc_run_live on ws
const int *hbk_flush_tc_live_count(const void *ws, int m) {
    const int groups = (m + 63) / 64;
    const unsigned char *w = (const unsigned char *)ws + 256 + 64 * sizeof(unsigned long long) + (size_t)groups * A_BYTES;
    return (const int *)(w + (size_t)groups * TC_M * (sizeof(int) + sizeof(double)));
}

// every shift live
int hbk_flush_tc_run(const double *V, size_t ld, unsigned n, int L, const double *Xc, const double *Pc, int cap,
                     const double *own, int m, double *X, double *Pmat, int keep_p, void *ws, int *err,
                     cudaStream_t st) {
    return hbk_flush_tc_run_live(V, ld, n, L, Xc, Pc, cap, own, m, X, Pmat, keep_p, nullptr, 0, nullptr, ws, err, st);
}

}  // extern "C"
