// Products A^H B of tall skinny ComplexF64 matrices on the integer tensor
// cores: an Ozaki-style split of every FP64 entry into 8-bit slices whose
// products are exact in 32-bit integer accumulators, recovered to FP64 with
// power-of-two weights. fb_gram.cu takes this form of gram_accumulate!
// (src/kernels.jl:22-55) where it is the faster one and checks afterwards, on
// the device, that it was also accurate enough (split_sum_kernel).
//
// Output tiles are 64 x 64 columns; a CTA owns one tile and one chunk of rows.
//   Folded tile (A === B, on the diagonal). With G = A^H A the real 64 x 64
//   matrix S = Re G + Im G = V^T W holds all of G (Re and Im are its
//   symmetric and antisymmetric parts): W is the interleaved (re, im) rows of
//   A, V the rows (re - im, re + im).
//   Full tile: [W JW]^T W' = [Re; Im] of A^H B, with JW the rows (-im, re) of
//   A and W' the interleaved rows of B.
//
// Slices. Column j carries a power-of-two scale 2^E with |entries| <
// 2^E (1 - 2^-7); an entry x becomes the integer x_int = rint(x 2^(51 - E)),
// written as seven signed bytes on a grid of 8-bit steps,
//   x_int = sum_{t=1..7} d_t 2^(52 - 8 t),   d_t in [-128, 127],
// the last a multiple of 16. One FMA makes them: m = fma(x, 2^(51 - E),
// 2^52 + 2^51 + B) is exact, its 52 mantissa bits are x_int + B + 2^51 with
// B = 0x80808080808 biasing every digit by half its range, and the bytes of
// m << 4 are the digits, each plus 128: the slices are read out of the
// double's bit pattern. V is twice as large and is scaled by half as much.
// A product of two entries is 2^(E_a + E_b - 102) sum d_t e_u 2^(104 - 8(t+u));
// the 28 terms with t + u <= 8 are kept (a folded tile also gets three of the
// six with t + u = 9), the rest lie below 2^-50 of the leading term.
//
// MMAs (kind::i8, M = 128, K = 32 bytes = 16 complex rows, one stage).
//   Full tile: operand A is slice t of W (rows 0-63) and of JW (rows 64-127),
//   operand B the slices 1..8-t of W' stacked along N; the product lands in
//   the accumulator blocks of the groups t + u = 2..8 (seven blocks of 64
//   columns of tensor memory): 1792 columns of N a stage.
//   Folded tile: S needs 64 rows only, so two slices of V share one operand,
//   t = 2p + 1 in rows 0-63 and t = 2p + 2 in rows 64-127, against slices
//   1..7-2p of W; block c then holds group c + 2 in rows 0-63 and c + 3 in
//   rows 64-127: 1024 columns of N a stage, 0.57 of the full tile's.
//
// Scales adapt as the rows stream: a stage with an entry its column's scale
// cannot hold, or one that would let an int32 accumulator overflow, starts a
// new epoch: the accumulators are first drained into this CTA's FP64 partial
// tile, then the column's scale grows. The scale is the power of two above 1.3
// times the maximum that asked for it, and the first one, set by 16 rows, above
// 2.6 times: for Gaussian rows that is 8 sigma, which no later row passes. More
// room costs accuracy (two more bits on every column: 2.3 times the error),
// less costs epochs (above 2 times: 330 us for 10^6 x 64 instead of 300).
//
// What bounds it and how the work is laid out: a stage of 16 rows costs 512
// cycles of integer MMA for a folded tile, about 600 of 32-bit integer work to
// cut and transpose the slices, 709 of HBM time, and shared memory traffic:
// the tile coming in, its rows read once by the slicers, the W slices written
// and read back by the MMAs. Operand A therefore lives in tensor memory (two
// buffers of it beside the accumulators for a folded tile, one for a full
// one): with A in shared memory too, and separate warps reading every entry
// once more for the scales, that traffic alone took 1190 cycles a stage and
// bound the kernel. Nothing may serialize either: the slicers form GROUPS
// groups that take the stages in turn, so one group's load, cut and store
// chain overlaps the others' and the MMAs; a group publishes its stage's
// column maxima, a decider warp turns them into scales in stage order, and no
// slicer ever waits on another group's slicing. Every wait is bounded; a
// failed one stops the CTA and marks its result invalid. Measured: 2.80 ms for
// 10^7 x 64 folded (5.18 on the FP64 tensor cores), 5.70 ms for 64 x 64 cross
// products (9.20); the integer pipe is 62 % busy, HBM 56 %.
#include <type_traits>

#include "fb_gram_split.cuh"
#include "fb_umma.cuh"

namespace fb {
namespace split {

constexpr int SLICES = 7;
constexpr int ROWS = SPLIT_STAGE_ROWS;          // complex rows per stage: K = 32 bytes
constexpr int FBYTES = ROWS * 64 * 16;          // 16 KB: 16 rows x 64 columns
constexpr int BTILE = SLICES * 64 * 32;         // B: 7 x 64 rows x 32 bytes
constexpr int TMEM_COLS = 512;
// Added to the high word of a maximum, carries into its exponent when the
// mantissa is at least 2 / 1.3.
constexpr uint32_t ROUND_UP = (uint32_t)((2.0 - 2.0 / 1.3) * (1 << 20));
constexpr long long MAGIC_BITS = 0x4338080808080808ll;  // 2^52 + 2^51 + 0x80808080808

template <bool FULL>
struct Cfg {
    static constexpr int SIDES = FULL ? 2 : 1;                 // input tiles per stage
    static constexpr int GROUPS = FULL ? 2 : 4;                // slicer groups = B buffers
    static constexpr int GWARPS = 4 * SIDES;                   // warps of a group: a set of four per input tile
    static constexpr int SLOTS = FULL ? 6 : 10;                // FP64 ring depth
    static constexpr int NA = FULL ? SLICES : 4;               // A operands per stage, 8 columns of tensor memory each
    static constexpr int ABUFS = FULL ? 1 : 2;                 // stages of A operands held
    static constexpr int COLUMNS = 64 * SIDES;                 // input columns
    static constexpr int SLICERS = 32 * GWARPS * GROUPS;
    static constexpr int THREADS = SLICERS + 96;           // and the issuer, producer and decider warps
    // int32 headroom: products are at most 2^14, a block gets 7 (full) or 4
    // (folded) of them per K row and 2 K rows per complex row.
    static constexpr int EPOCH_STAGES = (FULL ? 8192 : 12288) / ROWS;
    struct Stage {                                             // of the stage a group is working on
        uint32_t colmax[64 * SIDES];                           // slicers: high words of the column maxima
        uint16_t colmin[64 * SIDES];                           // and the upper halves of those of the column minima
        int E[64 * SIDES], Eold[64 * SIDES];                   // decider: scales of this stage and the one before
        int fresh, epoch;
        int mma_fresh;                                         // fresh, kept by the slicers until the MMAs are issued
    };
    static constexpr size_t OFF_F = 0;
    static constexpr size_t OFF_B = OFF_F + (size_t)SLOTS * SIDES * FBYTES;
    static constexpr size_t OFF_STAGE = OFF_B + (size_t)GROUPS * BTILE;
    static constexpr size_t OFF_BAR = (OFF_STAGE + GROUPS * sizeof(Stage) + 15) / 16 * 16;
    static constexpr size_t OFF_MISC = OFF_BAR + (2 * SLOTS + 4 * GROUPS) * 8;
    static constexpr size_t SMEM = OFF_MISC + 64 + 1024;       // + alignment slack
};
static_assert(Cfg<false>::SMEM <= 227 * 1024 && Cfg<true>::SMEM <= 227 * 1024, "a CTA's shared memory");
constexpr int A_COL = 64 * SLICES;                             // tensor memory column of the first A operand
static_assert(A_COL + 8 * Cfg<false>::NA * Cfg<false>::ABUFS <= TMEM_COLS, "accumulators and A operands");
static_assert(A_COL + 8 * Cfg<true>::NA * Cfg<true>::ABUFS <= TMEM_COLS, "accumulators and A operands");

__device__ __forceinline__ uint32_t sw32_offset(uint32_t row, uint32_t chunk) {
    return row * 32 + ((chunk ^ ((row >> 2) & 1)) << 4);
}

// 2^e as a double for e in the normal range, 0 below it.
__device__ __forceinline__ double pow2(int e) {
    if (e < -1022) return 0.0;
    if (e > 1023) e = 1023;
    return __longlong_as_double((long long)(e + 1023) << 52);
}

// K-major operand tile with 32-byte rows and the 32-byte swizzle: eight-row
// groups 256 bytes apart, layout type 6 = SWIZZLE_32B.
__device__ __forceinline__ uint64_t desc_sw32(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;           // leading byte offset, unused when swizzled
    d |= (uint64_t)(256 >> 4) << 32;  // stride byte offset: eight 32-byte rows
    d |= (uint64_t)1 << 46;           // version
    d |= (uint64_t)6 << 61;           // SWIZZLE_32B
    return d;
}

// The seven slice words of four FMA results (bit patterns, each shifted
// left by 4): word t holds slice t of each, low to high. Bytes 6..0 of the
// four values are transposed with byte permutes and the bias bit of every
// digit flipped back.
__device__ __forceinline__ void slice_words(const uint64_t (&y)[4], uint32_t (&w)[SLICES]) {
    const uint32_t l0 = (uint32_t)y[0], l1 = (uint32_t)y[1], l2 = (uint32_t)y[2], l3 = (uint32_t)y[3];
    const uint32_t h0 = (uint32_t)(y[0] >> 32), h1 = (uint32_t)(y[1] >> 32);
    const uint32_t h2 = (uint32_t)(y[2] >> 32), h3 = (uint32_t)(y[3] >> 32);
    const uint32_t a01 = __byte_perm(l0, l1, 0x5140), b01 = __byte_perm(l0, l1, 0x7362);
    const uint32_t a23 = __byte_perm(l2, l3, 0x5140), b23 = __byte_perm(l2, l3, 0x7362);
    const uint32_t c01 = __byte_perm(h0, h1, 0x5140), d01 = __byte_perm(h0, h1, 0x7362);
    const uint32_t c23 = __byte_perm(h2, h3, 0x5140), d23 = __byte_perm(h2, h3, 0x7362);
    w[0] = __byte_perm(d01, d23, 0x5410) ^ 0x80808080u;  // byte 6
    w[1] = __byte_perm(c01, c23, 0x7632) ^ 0x80808080u;  // byte 5
    w[2] = __byte_perm(c01, c23, 0x5410) ^ 0x80808080u;  // byte 4
    w[3] = __byte_perm(b01, b23, 0x7632) ^ 0x80808080u;  // byte 3
    w[4] = __byte_perm(b01, b23, 0x5410) ^ 0x80808080u;  // byte 2
    w[5] = __byte_perm(a01, a23, 0x7632) ^ 0x80808080u;  // byte 1
    w[6] = __byte_perm(a01, a23, 0x5410) ^ 0x80808080u;  // byte 0
}

// The largest and the smallest high word over four complex values, each
// counting by the larger of its parts, taken as single-precision magnitudes,
// which order like the words themselves and whose comparison drops the sign for
// free. A word past single precision's range (|x| >= 2^1017, Inf, NaN)
// propagates to the largest as a NaN, 0x7FFFFFFF.
__device__ __forceinline__ void range_hi(const double (&v)[8], uint32_t& largest, uint32_t& smallest) {
    float m[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
        asm("max.NaN.f32 %0, %1, %2;" : "=f"(m[e])
            : "f"(fabsf(__int_as_float(__double2hiint(v[2 * e])))),
              "f"(fabsf(__int_as_float(__double2hiint(v[2 * e + 1])))));
    float mx = m[0];
#pragma unroll
    for (int e = 1; e < 4; ++e) asm("max.NaN.f32 %0, %0, %1;" : "+f"(mx) : "f"(m[e]));
    largest = (uint32_t)__float_as_int(mx);
    smallest = (uint32_t)__float_as_int(fminf(fminf(m[0], m[1]), fminf(m[2], m[3])));
}

// What an operand's K rows are made of, from a complex entry (re, im).
enum Form { FORM_W, FORM_JW, FORM_V };

// Cuts two complex rows of one column (re, im, re, im) into the four K bytes
// of every slice.
template <Form F>
__device__ __forceinline__ void cut(const double* v, double sc, uint32_t (&w)[SLICES]) {
    const double magic = __longlong_as_double(MAGIC_BITS);
    uint64_t y[4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const double re = v[2 * r], im = v[2 * r + 1];
        double a = re, b = im;
        if (F == FORM_JW) { a = -im; b = re; }
        if (F == FORM_V) { a = re - im; b = re + im; }
        y[2 * r] = (uint64_t)__double_as_longlong(fma(a, sc, magic)) << 4;
        y[2 * r + 1] = (uint64_t)__double_as_longlong(fma(b, sc, magic)) << 4;
    }
    slice_words(y, w);
}

// Adds the accumulators into the partial tile P (128 x 64 doubles, column n
// contiguous): this thread's row `prow`, all 64 columns. EA and EB are the
// scale exponents of the operands' columns in the epoch that ends. Kept out
// of line: it runs a few times per CTA and would otherwise hold registers
// across the slicing loop.
template <bool FULL>
__device__ __noinline__ void drain_epoch(uint32_t tmem_lane, const int* EA, const int* EB, int prow, double* P,
                                         bool initialized) {
    const int Em = EA[prow & 63];
    // Weight of block c: 2^(E_a + E_b + 2 - 8 g), V's halved scale one more.
    const int shift = FULL ? 2 : (prow < 64 ? 3 : 3 - 8);
#pragma unroll 1
    for (int cc = 0; cc < 4; ++cc) {
        double acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.0;
#pragma unroll 1
        for (int c = 0; c < SLICES; ++c) {
            uint32_t r[16];
            umma::tmem_ld16(tmem_lane + 64 * c + 16 * cc, r);
            umma::tmem_wait_ld();
            const double w = pow2(-8 * (c + 2));
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = fma((double)(int)r[i], w, acc[i]);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int n = 16 * cc + i;
            const int En = EB[n];
            double v = 0.0;
            if (Em != SPLIT_E_UNSET && En != SPLIT_E_UNSET) v = acc[i] * pow2(Em + En + shift);
            double* dst = P + (size_t)n * 128 + prow;
            *dst = initialized ? *dst + v : v;
        }
    }
    __threadfence_block();
}

// Whether the screen refused any column; by all threads of a block.
__device__ __forceinline__ bool screened_off(const int* __restrict__ refused, const SplitShape& sh) {
    int any = 0;
    for (int c = threadIdx.x; c < SPLIT_SCREEN_PARTS * sh.screened; c += blockDim.x) any |= refused[c];
    return __syncthreads_or(any) != 0;
}

// A look at a sample of every column before its products are formed: 64 rows of
// every chunk, its first 16, its last 16 and two runs of 16 between them, by
// SPLIT_SCREEN_PARTS blocks a column (A's, then those of B) that take every
// SPLIT_SCREEN_PARTS-th chunk. What the verdict would refuse afterwards, or what the
// slicing is slow on, goes to the FP64 kernels at once. A column is refused
//   when a quarter of the runs have an entry under 2^-6 of their chunk's
//   sampled maximum (the verdict asks for 5/8 of the stages within 2^-8 of a
//   scale of 2.6 to 5.2 times that of the first stage);
//   when two of a chunk's four runs have one under 2^-10 of it;
//   when a chunk's later runs exceed its first by 4 or more: a scale set by
//   the first 16 rows holds 2.6 times their maximum, and each time a column
//   outgrows its scale the accumulators are drained;
//   when its real or its imaginary part stays under 2^-5 of the other: one sum of
//   both parts carries Re and Im of a folded tile, and what is left out of it
//   would show in the smaller of them (the Gram of real columns has no Im at all);
//   at numbers that are not finite or whose products could leave the range.
// The choice of the runs depends on the shape alone. Gaussian columns pass with
// a few runs in a hundred under the line and all but never a fourfold maximum.
// Latency-bound, hence the four blocks a column: 6.3 us for 64 columns (one
// block of 512 threads a column: 10). Without it a refused product paid for
// both forms, and for a drain at every growth. Folded, 2e6 x 64, us, FP64 alone
// 1075: columns in Gaussian envelopes 6530 -> 1087, heavy-tailed 3130 -> 1090,
// sin(pi j x) 3190 -> 1090; 3e5 rows, FP64 alone 198: 1780, 1110, 1220 -> 218.
// Accepted: 585 -> 592 and 133 -> 141.
constexpr int SCREEN_THREADS = 256;

__global__ void __launch_bounds__(SCREEN_THREADS)
split_screen_kernel(const z64* __restrict__ A, int64_t lda, const z64* __restrict__ B, int64_t ldb, int64_t rows,
                    SplitShape sh, int kA, int* __restrict__ refused, const ChainStatus* st, int gate) {
    if (gated_off(st, gate)) return;
    constexpr int WARPS = SCREEN_THREADS / 32, BATCH = 5;
    const int c = blockIdx.x / SPLIT_SCREEN_PARTS, part = blockIdx.x % SPLIT_SCREEN_PARTS;
    const int nchunks = (sh.nchunks - part + SPLIT_SCREEN_PARTS - 1) / SPLIT_SCREEN_PARTS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const z64* x = c < kA ? A + (int64_t)c * lda : B + (int64_t)(c - kA) * ldb;
    __shared__ uint32_t most[2];
    __shared__ int low, runs, grown;
    if (threadIdx.x == 0) { most[0] = most[1] = 0; low = runs = grown = 0; }
    __syncthreads();
    uint32_t all[2] = {0, 0};     // the largest real and imaginary part
    int wlow = 0, wruns = 0, wgrown = 0, wgraded = 0;
    for (int k0 = warp; k0 < nchunks; k0 += BATCH * WARPS) {
        z64 v[BATCH][2];
#pragma unroll
        for (int q = 0; q < BATCH; ++q) {
            const int k = SPLIT_SCREEN_PARTS * min(k0 + q * WARPS, nchunks - 1) + part;
            const int64_t row0 = (int64_t)k * sh.chunk_rows;
            const int len = (int)min(rows - row0, sh.chunk_rows), last = max(len - SPLIT_STAGE_ROWS, 0);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // Half a warp a run: the first and one in the first half, then
                // one in the second half and the last.
                const int r = 2 * h + (lane >> 4);
                const uint32_t jump = __umulhi((uint32_t)(4 * k + r) * 2654435761u, (uint32_t)(last / 2));
                const int off = r == 0 ? 0 : r == 3 ? last : (r - 1) * (last / 2) + (int)jump;
                v[q][h] = x[row0 + min(off + (lane & 15), len - 1)];
            }
        }
#pragma unroll
        for (int q = 0; q < BATCH; ++q) {
            if (k0 + q * WARPS >= nchunks) break;
            uint32_t m[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t re = (uint32_t)__double2hiint(v[q][h].x) & 0x7FFFFFFFu;
                const uint32_t im = (uint32_t)__double2hiint(v[q][h].y) & 0x7FFFFFFFu;
                m[h] = max(re, im);
                all[0] = max(all[0], re);
                all[1] = max(all[1], im);
            }
            const uint32_t first = __reduce_max_sync(0xffffffffu, lane < 16 ? m[0] : 0u);
            const uint32_t top = __reduce_max_sync(0xffffffffu, max(m[0], m[1]));
            if (top == 0) continue;   // a chunk of zeros is exact
            const uint32_t line = top > (6u << 20) ? top - (6u << 20) : 1u;
            const uint32_t b0 = __ballot_sync(0xffffffffu, m[0] < line), b1 = __ballot_sync(0xffffffffu, m[1] < line);
            wlow += ((b0 & 0xFFFFu) != 0) + ((b0 >> 16) != 0) + ((b1 & 0xFFFFu) != 0) + ((b1 >> 16) != 0);
            wruns += 4;
            wgrown += top >= first + (2u << 20);
            const uint32_t deep = top > (10u << 20) ? top - (10u << 20) : 1u;
            const uint32_t d0 = __ballot_sync(0xffffffffu, m[0] < deep), d1 = __ballot_sync(0xffffffffu, m[1] < deep);
            wgraded += ((d0 & 0xFFFFu) != 0) + ((d0 >> 16) != 0) + ((d1 & 0xFFFFu) != 0) + ((d1 >> 16) != 0) >= 2;
        }
    }
    for (int p = 0; p < 2; ++p) all[p] = __reduce_max_sync(0xffffffffu, all[p]);
    if (lane == 0) {
        for (int p = 0; p < 2; ++p) atomicMax(&most[p], all[p]);
        atomicAdd(&low, wlow);
        atomicAdd(&runs, wruns);
        atomicAdd(&grown, wgrown + wgraded);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t top = max(most[0], most[1]), other = min(most[0], most[1]);
        const int e = (int)(top >> 20) - 1023;
        refused[blockIdx.x] = top != 0 && (4 * low > runs || grown > 0 || other + (5u << 20) < top || e < -440 || e > 440);
    }
}

template <bool FULL>
__global__ void __launch_bounds__(Cfg<FULL>::THREADS, 1)
split_gram_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int64_t rows,
                  SplitShape sh, double* __restrict__ partial, SplitStat* __restrict__ stats, const ChainStatus* st,
                  int gate, int chunk0, const int* __restrict__ refused, int give_up, int zero) {
    if (gated_off(st, gate)) return;
    if (refused && screened_off(refused, sh)) return;
    using C = Cfg<FULL>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    typename C::Stage* stages = reinterpret_cast<typename C::Stage*>(smem + C::OFF_STAGE);
    uint64_t* fp_full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);   // a stage's rows have landed
    uint64_t* fp_empty = fp_full + C::SLOTS;                              // and are in its slicers' registers
    uint64_t* mx_full = fp_empty + C::SLOTS;                              // a group's column maxima are published
    uint64_t* sc_full = mx_full + C::GROUPS;                              // and its scales
    uint64_t* sl_full = sc_full + C::GROUPS;                              // its slices are written
    uint64_t* sl_empty = sl_full + C::GROUPS;                             // and consumed by the MMAs
    int* misc = reinterpret_cast<int*>(smem + C::OFF_MISC);
    volatile int* abort_flag = misc;
    int* bad_flag = misc + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(misc + 2);

    int ti, tj, tile;
    split_tile_of(sh, FULL, (int)blockIdx.x, ti, tj, tile);
    // Taken from one lane, so that the branches on it are known to be uniform.
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int chunk = chunk0 + (int)blockIdx.y;
    const int64_t row0 = (int64_t)chunk * sh.chunk_rows;
    const int64_t row_end = min(rows, row0 + sh.chunk_rows);
    const int nstages = (int)((row_end - row0 + ROWS - 1) / ROWS);
    double* P = partial + ((size_t)tile * sh.nchunks + chunk) * SPLIT_TILE_DOUBLES;
    SplitStat* stat = stats + (size_t)tile * sh.nchunks + chunk;

    if (threadIdx.x == 0) {
        for (int b = 0; b < C::SLOTS; ++b) {
            mbar_init(&fp_full[b], 1);
            mbar_init(&fp_empty[b], C::GWARPS);
        }
        for (int b = 0; b < C::GROUPS; ++b) {
            mbar_init(&mx_full[b], C::GWARPS);
            mbar_init(&sc_full[b], 1);
            mbar_init(&sl_full[b], C::GWARPS);
            mbar_init(&sl_empty[b], 1);
        }
        *abort_flag = 0;
        *bad_flag = 0;
        mbar_fence_init();
    }
    if (warp == 0) umma::tmem_alloc(tmem_slot, TMEM_COLS);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t taddr = *tmem_slot;
    double sumsq[2] = {0.0, 0.0};                            // of a slicer's two columns

    if (warp == C::SLICERS / 32 + 1) {
        // ---- producer: FP64 tiles, two 8-row boxes per stage and input ----
        if (lane == 0) {
            tma_prefetch_map(&tmA);
            if (FULL) tma_prefetch_map(&tmB);
            int issued = 0, b = 0;
            uint32_t ph = 0;
            for (int s = 0; s < nstages; ++s) {
                if (s >= C::SLOTS && !mbar_wait(&fp_empty[b], ph ^ 1u)) {
                    *abort_flag = 1;
                    break;
                }
                if (*abort_flag) break;
                mbar_arrive_expect_tx(&fp_full[b], C::SIDES * FBYTES);
                const int x = (int)(2 * (row0 + (int64_t)s * ROWS));
                unsigned char* dst = smem + C::OFF_F + (size_t)b * C::SIDES * FBYTES;
                tma_load_2d(dst, &tmA, x, 64 * ti, &fp_full[b]);
                tma_load_2d(dst + FBYTES / 2, &tmA, x + 16, 64 * ti, &fp_full[b]);
                if (FULL) {
                    tma_load_2d(dst + FBYTES, &tmB, x, 64 * tj, &fp_full[b]);
                    tma_load_2d(dst + FBYTES + FBYTES / 2, &tmB, x + 16, 64 * tj, &fp_full[b]);
                }
                issued = s + 1;
                if (++b == C::SLOTS) { b = 0; ph ^= 1u; }
            }
            // After an abort, let the copies still in flight land before the
            // shared memory they write goes away.
            for (int s = issued > C::SLOTS ? issued - C::SLOTS : 0; *abort_flag && s < issued; ++s)
                mbar_wait(&fp_full[s % C::SLOTS], (s / C::SLOTS) & 1);
        }
    } else if (warp == C::SLICERS / 32) {
        // ---- MMA issuer ----
        if (lane == 0) {
            int issued = 0, g = 0;
            uint32_t ph = 0;
            for (int s = 0; s < nstages; ++s) {
                if (!mbar_wait(&sl_full[g], ph) || *abort_flag) {
                    *abort_flag = 1;
                    break;
                }
                umma::fence_after_sync();
                const bool fresh = *(volatile int*)&stages[g].mma_fresh != 0;
                const uint32_t atmem = taddr + A_COL + 8 * C::NA * (s % C::ABUFS);
                const uint32_t bbase = smem_u32(smem + C::OFF_B + (size_t)g * BTILE);
#pragma unroll
                for (int a = 0; a < C::NA; ++a) {
                    const int first = FULL ? a : 2 * a;      // accumulator block of slice 1 of B
                    const int ntot = 64 * (SLICES - first);
#pragma unroll
                    for (int off = 0; off < ntot; off += 256) {
                        const int n = ntot - off < 256 ? ntot - off : 256;
                        umma::mma_s8_tmem_a(taddr + 64 * first + off, atmem + 8 * a, desc_sw32(bbase + off * 32),
                                            umma::idesc_s8s8_s32(128, n), !(fresh && a == 0));
                    }
                }
                umma::commit(&sl_empty[g]);
                issued = s + 1;
                if (++g == C::GROUPS) { g = 0; ph ^= 1u; }
            }
            // After an abort, wait for the MMAs in flight before tensor memory
            // is released.
            if (*abort_flag && issued > 0)
                mbar_wait(&sl_empty[(issued - 1) % C::GROUPS], ((issued - 1) / C::GROUPS) & 1);
        }
    } else if (warp < C::SLICERS / 32) {
        // ---- slicers ----
        // Warp q of a set of four cuts columns 16 q .. 16 q + 15 of its input
        // tile, lane (c8, i) columns m0 = 16 q + c8 and m0 + 8, rows 2 i and
        // 2 i + 1 of both 8-row boxes: words i and 4 + i of a column's 32 K
        // bytes. That is the layout of a 16-lane store to tensor memory,
        // whose lanes c8 and c8 + 8 take the two halves of an A operand (two
        // slices of V, or W and JW) of one column: accumulator lane
        // 32 q + 16 n + c8 (+ 8) belongs to column 16 q + 8 n + c8.
        const int g = warp / C::GWARPS, w = warp - g * C::GWARPS;
        typename C::Stage& stage = stages[g];
        auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity); };
        // Until the MMAs of stage s are done. The barrier is at most one
        // phase behind: this group has waited for its own previous stage,
        // which is later than the one before s on that barrier.
        auto wait_mma = [&](int s) { return wait(&sl_empty[s % C::GROUPS], (s / C::GROUPS) & 1); };
        const int c8 = lane >> 2, i = lane & 3;

        auto slicer = [&](auto side_tag) -> bool {
            constexpr int SIDE = decltype(side_tag)::value;
            constexpr int NC = 2;                             // columns a lane
            constexpr bool TO_B = !FULL || SIDE == 1;         // cuts operand B
            constexpr bool TO_A = SIDE == 0;
            const int q = w & 3, m0 = 16 * q + c8;
            unsigned char* bbuf = smem + C::OFF_B + (size_t)g * BTILE;
            const uint32_t tmem_lane = taddr + ((uint32_t)(32 * q) << 16);
            const int prow = ((lane >> 3) & 1) * 64 + 16 * q + 8 * (lane >> 4) + (lane & 7);
            double v[NC][8];
            // This warp's rows of stage s into registers, and its columns'
            // maxima published: the high word of |x| orders magnitudes by
            // exponent, and Inf and NaN above every finite value. A column of
            // nothing but numbers below the high word's range reports 1.
            auto load = [&](int s) -> bool {
                const int b = s % C::SLOTS;
                if (!wait(&fp_full[b], (s / C::SLOTS) & 1)) return false;
                const unsigned char* f = smem + C::OFF_F + ((size_t)b * C::SIDES + SIDE) * FBYTES;
#pragma unroll
                for (int n = 0; n < NC; ++n)
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int m = m0 + 8 * n, row = 2 * i + (r & 1);
                        const double2 z = *reinterpret_cast<const double2*>(f + (r >> 1) * (FBYTES / 2) + m * 128 +
                                                                            ((row ^ (m & 7)) << 4));
                        v[n][2 * r] = z.x;
                        v[n][2 * r + 1] = z.y;
                    }
                return true;
            };
            auto publish = [&](int s) {
                uint32_t mn[NC];
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    uint32_t mx;
                    range_hi(v[n], mx, mn[n]);
                    if (mx == 0) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) mx |= __double2loint(v[n][e]) != 0 ? 1u : 0u;
                    }
                    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                    if (i == 0) stage.colmax[64 * SIDE + m0 + 8 * n] = mx;
                }
                // Both columns' minima at once, their words' upper halves.
                uint32_t low = __byte_perm(mn[0], mn[1], 0x7632);
                low = __vminu2(low, __shfl_xor_sync(0xffffffffu, low, 1));
                low = __vminu2(low, __shfl_xor_sync(0xffffffffu, low, 2));
                if (i == 0) {
                    stage.colmin[64 * SIDE + m0] = (uint16_t)low;
                    stage.colmin[64 * SIDE + m0 + 8] = (uint16_t)(low >> 16);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&mx_full[g]);
            };
            // Sums of squares of the leading digits, in units of
            // 4^(E - 7) of the scale they were cut with.
            int E[NC], digits[NC];
#pragma unroll
            for (int n = 0; n < NC; ++n) { E[n] = SPLIT_E_UNSET; digits[n] = 0; }
            auto fold = [&](int n) {
                if (E[n] != SPLIT_E_UNSET) sumsq[n] += (double)digits[n] * pow2(2 * (E[n] - 7));
                digits[n] = 0;
            };
            auto drain = [&](int s, const int* EA, const int* EB, bool initialized) -> bool {
                if (!wait_mma(s)) return false;
                umma::fence_after_sync();
                drain_epoch<FULL>(tmem_lane, EA, EB, prow, P, initialized);
                umma::fence_before_sync();
                return true;
            };
            uint32_t gph = 0;                                 // parity of this group's stage count
            int s = g;
            if (s < nstages) {
                if (!load(s)) return false;
                publish(s);
            }
            for (; s < nstages; s += C::GROUPS, gph ^= 1u) {
                if (!wait(&sc_full[g], gph) || __any_sync(0xffffffffu, *abort_flag != 0)) return false;
                const bool fresh = __any_sync(0xffffffffu, stage.fresh != 0);
                // This group's B buffer is free once its previous stage's
                // MMAs are done.
                if (s >= C::GROUPS && !wait(&sl_empty[g], gph ^ 1u)) return false;
                // A new epoch: the MMAs of the one before it all precede this
                // stage's, which wait for this group. (The rows are read
                // again, so that no register holds them across the drain.)
                uint32_t seen = 0;
                if (TO_A && fresh && s > 0) {
                    if (!drain(s - 1, stage.Eold, stage.Eold + (FULL ? 64 : 0), stage.epoch > 1) || !load(s))
                        return false;
#pragma unroll
                    for (int n = 0; n < NC; ++n)
#pragma unroll
                        for (int e = 0; e < 8; ++e) mark_loaded(seen, v[n][e]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&fp_empty[s % C::SLOTS + (seen & zero)]);
                double sc[NC];
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    const int En = stage.E[64 * SIDE + m0 + 8 * n];
                    if (En != E[n] || (s / C::GROUPS) % 4096 == 0) {   // digits: 2^17 a stage at most
                        fold(n);
                        E[n] = En;
                    }
                    sc[n] = En == SPLIT_E_UNSET ? 0.0 : pow2(51 - En);
                }
                if constexpr (TO_B) {
#pragma unroll
                    for (int n = 0; n < NC; ++n) {
                        const int m = m0 + 8 * n;
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            uint32_t wd[SLICES];
                            cut<FORM_W>(v[n] + 4 * x, sc[n], wd);
                            digits[n] = __dp4a((int)wd[0], (int)wd[0], digits[n]);
                            unsigned char* b0 = bbuf + sw32_offset(m, x) + 4 * i;
#pragma unroll
                            for (int t = 0; t < SLICES; ++t) *reinterpret_cast<uint32_t*>(b0 + t * (64 * 32)) = wd[t];
                        }
                    }
                }
                if constexpr (TO_A) {
                    uint32_t lo[NC][2][SLICES], hi[FULL ? NC : 1][2][SLICES];
#pragma unroll
                    for (int n = 0; n < NC; ++n)
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            if constexpr (FULL) {
                                cut<FORM_W>(v[n] + 4 * x, sc[n], lo[n][x]);
                                cut<FORM_JW>(v[n] + 4 * x, sc[n], hi[n][x]);
                                digits[n] = __dp4a((int)lo[n][x][0], (int)lo[n][x][0], digits[n]);
                            } else {
                                cut<FORM_V>(v[n] + 4 * x, 0.5 * sc[n], lo[n][x]);
                            }
                        }
                    if (s >= C::ABUFS && !wait_mma(s - C::ABUFS)) return false;
                    umma::fence_after_sync();
                    const uint32_t at = tmem_lane + A_COL + 8 * C::NA * (s % C::ABUFS);
#pragma unroll
                    for (int n = 0; n < NC; ++n)
#pragma unroll
                        for (int a = 0; a < C::NA; ++a) {
                            const uint32_t col = at + 8 * a + ((uint32_t)(16 * n) << 16);
                            if constexpr (FULL)
                                umma::tmem_st_16x128b_x2(col, lo[n][0][a], hi[n][0][a], lo[n][1][a], hi[n][1][a]);
                            else
                                umma::tmem_st_16x128b_x2(col, lo[n][0][2 * a], a < 3 ? lo[n][0][2 * a + 1] : 0,
                                                         lo[n][1][2 * a], a < 3 ? lo[n][1][2 * a + 1] : 0);
                        }
                    umma::tmem_wait_st();
                }
                if (w == 0 && lane == 0) stage.mma_fresh = fresh ? 1 : 0;
                umma::fence_smem_to_async();
                umma::fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sl_full[g]);
                // The next stage's rows and maxima go out before this group
                // comes back to it, so its scales are settled by then.
                if (s + C::GROUPS < nstages) {
                    if (!load(s + C::GROUPS)) return false;
                    publish(s + C::GROUPS);
                }
            }
#pragma unroll
            for (int n = 0; n < NC; ++n) fold(n);
            // The group of the last stage drains the last epoch.
            if (TO_A && s - C::GROUPS == nstages - 1)
                return drain(nstages - 1, stage.E, stage.E + (FULL ? 64 : 0), stage.epoch > 0);
            return true;
        };
        bool ok;
        if constexpr (FULL) ok = w < 4 ? slicer(std::integral_constant<int, 0>{}) : slicer(std::integral_constant<int, 1>{});
        else ok = slicer(std::integral_constant<int, 0>{});
        if (!ok) *abort_flag = 1;
    } else {
        // ---- decider: the scales, in stage order ----
        // Lane l decides input columns l, l + 32, ... (A's 0-63, then B's).
        // |x| < 2^E (1 - 2^-7) in terms of the high word of x; while the
        // scale is unset every normal number is past it.
        // level[x][j] counts the stages whose smallest entry is 2^(E - 8 + j) or
        // more, by the scale of the time; the levels move down as it grows.
        constexpr int NC = C::COLUMNS / 32, LEVELS = 7;
        int E[NC], level[NC][LEVELS] = {};
        uint32_t limit[NC];
        bool tiny[NC], bad = false;
#pragma unroll
        for (int x = 0; x < NC; ++x) {
            E[x] = SPLIT_E_UNSET;
            limit[x] = 0x00100000u;
            tiny[x] = false;
        }
        // With the FP64 kernels behind it (give_up), a chunk whose scales keep
        // growing is theirs: the rest of it passes with the scales it has.
        const int most = 16 + nstages / 256;
        bool gave_up = false;
        int g = 0, epoch = -1, epoch_start = 0;
        uint32_t ph = 0;
        for (int s = 0; s < nstages; ++s) {
            typename C::Stage& stage = stages[g];
            if (!mbar_wait_warp(&mx_full[g], ph) || __any_sync(0xffffffffu, *abort_flag != 0)) {
                *abort_flag = 1;
                break;
            }
            uint32_t mx[NC];
            int low[NC];
            bool over[NC], mine = false;
#pragma unroll
            for (int x = 0; x < NC; ++x) {
                mx[x] = stage.colmax[32 * x + lane];
                low[x] = (int)(stage.colmin[32 * x + lane] >> 4) - 1023;
                over[x] = mx[x] >= limit[x];
                if (mx[x] >= 0x7FF00000u) { bad = true; over[x] = false; }   // Inf, NaN or next to them
                if (E[x] == SPLIT_E_UNSET && mx[x] != 0 && mx[x] < 0x00100000u) tiny[x] = true;
                mine = mine || over[x];
                stage.Eold[32 * x + lane] = E[x];
            }
            if (give_up && epoch >= most) gave_up = true;
            const bool any_over = __any_sync(0xffffffffu, mine) && !gave_up;
            if (any_over) {
#pragma unroll
                for (int x = 0; x < NC; ++x) {
                    if (!over[x]) continue;
                    // The power of two above 1.3 times the maximum, and once
                    // more that while the maximum is that of 16 rows only.
                    const int spare = E[x] == SPLIT_E_UNSET ? 1 : 0, before = E[x];
                    E[x] = (int)((mx[x] + ROUND_UP) >> 20) - 1023 + 1 + spare;
#pragma unroll 1
                    for (int up = min(E[x] - before, LEVELS); up > 0; --up)
#pragma unroll
                        for (int j = 0; j < LEVELS; ++j) level[x][j] = j + 1 < LEVELS ? level[x][j + 1] : 0;
                    // The limit's exponent stays in range: a scale past it is
                    // refused afterwards by split_sum_kernel anyway.
                    limit[x] = ((uint32_t)min(max(E[x] - 1 + 1023, 1), 0x7FE) << 20) | 0xFC000u;
                }
            }
            const bool fresh = s == 0 || any_over || (s - epoch_start >= C::EPOCH_STAGES && !gave_up);
            if (fresh) {
                ++epoch;
                epoch_start = s;
            }
#pragma unroll
            for (int x = 0; x < NC; ++x) stage.E[32 * x + lane] = E[x];
            if (lane == 0) {
                stage.fresh = fresh ? 1 : 0;
                stage.epoch = epoch;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sc_full[g]);
            if (++g == C::GROUPS) { g = 0; ph ^= 1u; }
#pragma unroll
            for (int x = 0; x < NC; ++x)
#pragma unroll
                for (int j = 0; j < LEVELS; ++j) level[x][j] += E[x] != SPLIT_E_UNSET && low[x] - (E[x] - 8) >= j;
        }
        if (bad) atomicOr(bad_flag, SPLIT_INVALID);
        if (gave_up) atomicOr(bad_flag, SPLIT_INACCURATE);
#pragma unroll
        for (int x = 0; x < NC; ++x) {
            // Fewer than 5/8 of the stages within 2^-8 of the scale.
            if (E[x] != SPLIT_E_UNSET && 8 * level[x][0] < 5 * nstages) atomicOr(bad_flag, SPLIT_INACCURATE);
            stat->E[32 * x + lane] = E[x] == SPLIT_E_UNSET && tiny[x] ? SPLIT_E_TINY : E[x];
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (threadIdx.x == 0) stat->flags = (*abort_flag ? SPLIT_INVALID : 0) | *bad_flag;
    if (warp == 0) umma::tmem_dealloc(taddr, TMEM_COLS);
    // The columns' sums of squares, over the four lanes of a column, then the
    // groups in order (the ring is free by now).
    double* sq = reinterpret_cast<double*>(smem + C::OFF_F);
    if (warp < C::SLICERS / 32) {
        const int g = warp / C::GWARPS, w = warp - g * C::GWARPS;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            sumsq[n] += __shfl_xor_sync(0xffffffffu, sumsq[n], 1);
            sumsq[n] += __shfl_xor_sync(0xffffffffu, sumsq[n], 2);
            if ((lane & 3) == 0) sq[g * C::COLUMNS + 16 * w + 8 * n + (lane >> 2)] = sumsq[n];
        }
    }
    __syncthreads();
    if (threadIdx.x < C::COLUMNS) {
        double t = 0.0;
        for (int g = 0; g < C::GROUPS; ++g) t += sq[g * C::COLUMNS + threadIdx.x];
        stat->sumsq[threadIdx.x] = t;
    }
}

// Blocks 0..127 of a tile: half a column each (a folded tile: a column, its
// two halves added) summed over the chunks in a fixed order, eight interleaved
// runs of chunks, then the eight. Block 128: the tile's verdict. The partial
// tiles are in L2, so the loads' latency is what counts: ten are in flight a
// thread (21 us at 148 chunks with the loads of the sums and of the verdict waiting
// for one another, 7 to 10 now).
//
// The verdict compares what the slices leave out with what the column weighs.
// With scale 2^E an entry is off by at most 2^(E - 51) (V: 2^(E - 50)), which
// reaches G_ij as an error of about 2^(E_j - 50) / sqrt(12) ||a_i||. The
// products left out, digits of standard deviation 74: in a full tile the six
// pairs with t + u = 9 over 2 N K rows, sqrt(12 N) 74^2 2^(E_i + E_j - 70); in a
// folded one three pairs of twice the weight, of which the mean of S_ij and
// S_ji keeps 1 / sqrt(2): the same. Both stay below 2^-54 ||a_i|| ||a_j||,
// under the rounding of the FP64 sums themselves, when
//     ||a_j||^2 >= 4^E_j max(21.4, 0.29 sqrt(N)).
// These are root mean squares of roundings that do not know of one another; a
// column of equal entries rounds alike in every row and is off by up to 4e-15
// of the entry (its FP64 sums: 1e-13 at 3e5 rows, 1.5e-12 at 4e6).
// The kernel knows ||a_j||^2 from the leading digits, whose rounding can raise
// it by a third where they are small, so it checks 1.4 times that (N Gaussian
// rows have at least about 2 N / 576).
// A spike that dwarfs the rest of its column fails it, as do Inf and NaN, a
// scale whose products could leave the FP64 range, and a wait that gave up:
// the caller then computes the tile in FP64 instead.
//
// An error that is small against ||a_i|| ||a_j|| can still be all of an entry
// to which only small parts of the columns contribute (rows graded one way in
// one column and the other way in another, say). FP64 sums are off by little
// against sum_r |a_ri| |a_rj|, and so the chunks report whether every column
// has, in at least 5/8 of the stages, all its entries within 2^-8 of its
// scale (entries count by the larger of their parts; a column that is zero
// throughout a chunk is exact there). Any two columns then share a quarter of
// the stages in which both have, so the sum is at least
// n / 4 2^(E_i + E_j - 16) over a chunk's n rows. Rows alternating by 2^-5, the
// two columns in opposite phase, pass: entries are then off by up to 2e-16 of
// their sum at 3e5 rows, as FP64 sums are; alternating by 2^-48, refused, they
// had no correct digit. Chunks of Gaussian rows pass with 9 of 10 stages or
// more, whatever scale their first 16 rows set.
constexpr int SUM_THREADS = 512;

__global__ void __launch_bounds__(SUM_THREADS)
split_sum_kernel(SplitShape sh, int64_t rows, const double* __restrict__ partial, const SplitStat* __restrict__ stats,
                 double* __restrict__ sums, int* __restrict__ verdict, const ChainStatus* st, int gate,
                 const int* __restrict__ refused) {
    if (gated_off(st, gate)) return;
    if (refused && screened_off(refused, sh)) {
        if (blockIdx.x == 128 && threadIdx.x == 0) verdict[blockIdx.y] = SPLIT_INACCURATE;
        return;
    }
    __shared__ double red[SUM_THREADS];
    __shared__ int redE[SUM_THREADS];
    __shared__ int flags;
    const int tile = blockIdx.y, tid = threadIdx.x;
    const bool full = !sh.hermitian || tile >= sh.nt_a;
    if (blockIdx.x < 128) {
        if (!full && blockIdx.x >= 64) return;
        const int n = full ? blockIdx.x >> 1 : blockIdx.x, half = full ? blockIdx.x & 1 : 0;
        const int m = tid & 63, run = tid >> 6;
        const double* p = partial + (size_t)tile * sh.nchunks * SPLIT_TILE_DOUBLES + n * 128 + half * 64 + m;
        double s = 0.0;
        for (int c0 = run; c0 < sh.nchunks; c0 += 80) {
            double v[10], w[10];
#pragma unroll
            for (int q = 0; q < 10; ++q) {
                const double* c = p + (size_t)min(c0 + 8 * q, sh.nchunks - 1) * SPLIT_TILE_DOUBLES;
                v[q] = c[0];
                w[q] = c[full ? 0 : 64];
            }
#pragma unroll
            for (int q = 0; q < 10; ++q)
                if (c0 + 8 * q < sh.nchunks) s += full ? v[q] : v[q] + w[q];
        }
        red[tid] = s;
        __syncthreads();
        if (tid >= 64) return;
        s = 0.0;
#pragma unroll
        for (int r = 0; r < 8; ++r) s += red[64 * r + tid];
        sums[(size_t)tile * SPLIT_TILE_DOUBLES + n * 128 + half * 64 + m] = s;
        return;
    }
    const int m = tid & 127, part = tid >> 7;
    if (tid == 0) flags = 0;
    __syncthreads();
    const int columns = full ? 128 : 64;
    int E = SPLIT_E_UNSET, mine = 0;
    double s = 0.0;
    const SplitStat* x = stats + (size_t)tile * sh.nchunks;
    for (int c = tid; c < sh.nchunks; c += SUM_THREADS)
        mine |= x[c].flags;
    if (m < columns)
        for (int c0 = part; c0 < sh.nchunks; c0 += 40) {
            double v[10];
            int e[10];
#pragma unroll
            for (int q = 0; q < 10; ++q) {
                const int c = min(c0 + 4 * q, sh.nchunks - 1);   // the last one again past the end
                v[q] = x[c].sumsq[m];
                e[q] = x[c].E[m];
            }
#pragma unroll
            for (int q = 0; q < 10; ++q) {
                s += c0 + 4 * q < sh.nchunks ? v[q] : 0.0;
                if (e[q] == SPLIT_E_TINY) mine |= SPLIT_INACCURATE;
                E = max(E, e[q] == SPLIT_E_TINY ? SPLIT_E_UNSET : e[q]);
            }
        }
    red[tid] = s;
    redE[tid] = E;
    __syncthreads();
    if (tid < columns) {
        s = (red[tid] + red[128 + tid]) + (red[256 + tid] + red[384 + tid]);
        E = max(max(redE[tid], redE[128 + tid]), max(redE[256 + tid], redE[384 + tid]));
        if (E != SPLIT_E_UNSET &&
            !(E >= -450 && E <= 450 && s >= fmax(30.0, 0.41 * sqrt((double)rows)) * pow2(2 * E)))
            mine |= SPLIT_INACCURATE;
    }
    if (mine) atomicOr(&flags, mine);
    __syncthreads();
    if (tid == 0) verdict[tile] = flags;
}

template <bool FULL>
static int launch(const CUtensorMap& ma, const CUtensorMap& mb, int64_t rows, const SplitShape& sh, int ntiles,
                  double* partial, SplitStat* stats, cudaStream_t stream, const ChainStatus* st, int gate, int chunk0,
                  int chunk1, const int* refused, int give_up) {
    using C = Cfg<FULL>;
    FB_ALLOW_SMEM(split_gram_kernel<FULL>, C::SMEM);
    split_gram_kernel<FULL><<<dim3((unsigned)ntiles, (unsigned)(chunk1 - chunk0)), C::THREADS, C::SMEM, stream>>>(
        ma, mb, rows, sh, partial, stats, st, gate, chunk0, refused, give_up, 0);
    FB_LAUNCHED("split_gram_kernel");
    return FB_OK;
}

}  // namespace split

// One chunk per SM for the launch with fewer tiles, in whole stages; of long
// chunks the last one is long too, since the verdict on a column is taken from
// each chunk's stages.
SplitShape split_shape(int64_t rows, int kA, int kB, bool hermitian) {
    SplitShape sh{};
    sh.nt_a = (kA + 63) / 64;
    sh.nt_b = (kB + 63) / 64;
    sh.hermitian = hermitian ? 1 : 0;
    sh.screened = hermitian ? kA : kA + kB;
    sh.ntiles = hermitian ? sh.nt_a * (sh.nt_a + 1) / 2 : sh.nt_a * sh.nt_b;
    int smallest = sh.ntiles;
    if (hermitian && sh.nt_a > 1) smallest = std::min(sh.nt_a, sh.nt_a * (sh.nt_a - 1) / 2);
    const int64_t stages = (rows + SPLIT_STAGE_ROWS - 1) / SPLIT_STAGE_ROWS;
    const int64_t target = std::max<int64_t>(1, sm_count() / smallest);
    int64_t per = std::max<int64_t>(1, (stages + target - 1) / target);
    while (per >= 96 && stages % per != 0 && stages % per < 64) ++per;
    sh.chunk_rows = per * SPLIT_STAGE_ROWS;
    sh.nchunks = (int)((rows + sh.chunk_rows - 1) / sh.chunk_rows);
    return sh;
}

SplitLayout split_layout(const SplitShape& sh) {
    SplitLayout L{};
    const size_t parts = (size_t)sh.ntiles * (size_t)(sh.nchunks > 0 ? sh.nchunks : 1);
    L.verdict = 0;
    L.refused = align_up((size_t)sh.ntiles * sizeof(int), 256);
    L.sums = L.refused + align_up((size_t)SPLIT_SCREEN_PARTS * sh.screened * sizeof(int), 256);
    L.stats = L.sums + (size_t)sh.ntiles * SPLIT_TILE_DOUBLES * sizeof(double);
    L.partial = align_up(L.stats + parts * sizeof(SplitStat), 256);
    L.total = L.partial + parts * SPLIT_TILE_DOUBLES * sizeof(double);
    return L;
}

int split_screen_enqueue(const z64* A, int64_t lda, const z64* B, int64_t ldb, int64_t rows, int kA,
                         const SplitShape& sh, void* workspace, cudaStream_t stream, const ChainStatus* st, int gate) {
    int* refused = reinterpret_cast<int*>(static_cast<char*>(workspace) + split_layout(sh).refused);
    split::split_screen_kernel<<<SPLIT_SCREEN_PARTS * sh.screened, split::SCREEN_THREADS, 0, stream>>>(
        A, lda, B, ldb, rows, sh, kA, refused, st, gate);
    FB_LAUNCHED("split_screen_kernel");
    return FB_OK;
}

int split_partials_enqueue(const z64* A, int64_t lda, const z64* B, int64_t ldb, int64_t rows, int kA, int kB,
                           const SplitShape& sh, void* workspace, cudaStream_t stream, const ChainStatus* st, int gate,
                           int chunk0, int chunk1, bool screened, bool strict) {
    if (chunk0 < 0) chunk0 = 0;
    if (chunk1 > sh.nchunks) chunk1 = sh.nchunks;
    if (chunk0 >= chunk1) return FB_OK;
    const SplitLayout L = split_layout(sh);
    char* ws = static_cast<char*>(workspace);
    double* partial = reinterpret_cast<double*>(ws + L.partial);
    SplitStat* stats = reinterpret_cast<SplitStat*>(ws + L.stats);
    CUtensorMap ma, mb;
    FB_TRY(encode_panel_map(&ma, A, rows, kA, lda, 64));
    if (sh.hermitian) mb = ma;
    else FB_TRY(encode_panel_map(&mb, B, rows, kB, ldb, 64));
    const int* refused = screened ? reinterpret_cast<const int*>(ws + L.refused) : nullptr;
    const int give_up = strict ? 0 : 1;
    const int full = sh.hermitian ? sh.ntiles - sh.nt_a : sh.ntiles;
    if (sh.hermitian)
        FB_TRY(split::launch<false>(ma, mb, rows, sh, sh.nt_a, partial, stats, stream, st, gate, chunk0, chunk1, refused,
                                    give_up));
    if (full > 0)
        FB_TRY(split::launch<true>(ma, mb, rows, sh, full, partial, stats, stream, st, gate, chunk0, chunk1, refused,
                                   give_up));
    return FB_OK;
}

int split_sum_enqueue(int64_t rows, const SplitShape& sh, void* workspace, cudaStream_t stream, const ChainStatus* st,
                      int gate, bool screened) {
    const SplitLayout L = split_layout(sh);
    char* ws = static_cast<char*>(workspace);
    split::split_sum_kernel<<<dim3(129, (unsigned)sh.ntiles), split::SUM_THREADS, 0, stream>>>(
        sh, rows, reinterpret_cast<const double*>(ws + L.partial), reinterpret_cast<const SplitStat*>(ws + L.stats),
        reinterpret_cast<double*>(ws + L.sums), reinterpret_cast<int*>(ws + L.verdict), st, gate,
        screened ? reinterpret_cast<const int*>(ws + L.refused) : nullptr);
    FB_LAUNCHED("split_sum_kernel");
    return FB_OK;
}

}  // namespace fb

