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
// tile, then the column's scale grows with HEADROOM spare bits.
//
// What bounds it and how the work is laid out: a stage of 16 rows costs 512
// cycles of integer MMA for a folded tile, about as many of 32-bit integer
// work to cut and transpose the slices, and 709 cycles of HBM time. So nothing
// may serialize: the decision about scales is made by scanner warps a few
// stages ahead of the slicers (so slicers never vote), and the slicers form
// GROUPS groups of four warps that take the stages in turn, each with a slice
// buffer of its own, so one group's load, cut and store chain overlaps the
// others' and the MMAs. Every wait is bounded; a failed one stops the CTA and
// marks its result invalid.
#include "fb_gram_split.cuh"
#include "fb_umma.cuh"

namespace fb {
namespace split {

constexpr int SLICES = 7;
constexpr int ROWS = SPLIT_STAGE_ROWS;          // complex rows per stage: K = 32 bytes
constexpr int FBYTES = ROWS * 64 * 16;          // 16 KB: 16 rows x 64 columns
constexpr int BTILE = SLICES * 64 * 32;         // B: 7 x 64 rows x 32 bytes
constexpr int ATILE = 128 * 32;                 // one A operand
constexpr int TMEM_COLS = 512;                  // 448 used; the allocation is a power of two
constexpr int HEADROOM = 2;                     // spare exponent bits above the maximum that set a scale
constexpr long long MAGIC_BITS = 0x4338080808080808ll;  // 2^52 + 2^51 + 0x80808080808

template <bool FULL>
struct Cfg {
    static constexpr int SIDES = FULL ? 2 : 1;                 // input tiles per stage
    static constexpr int GROUPS = FULL ? 3 : 4;                // slicer groups of 128 threads = slice buffers
    static constexpr int SLOTS = FULL ? 3 : 6;                 // FP64 ring depth
    static constexpr int NA = FULL ? SLICES : 4;               // A operands per stage
    static constexpr int SCANNERS = 64 * SIDES;                // scanner threads, one per input column
    static constexpr int SLICERS = 128 * GROUPS;
    static constexpr int THREADS = SLICERS + 64 + SCANNERS;
    static constexpr int BUF = NA * ATILE + BTILE;             // one slice buffer: A operands, then B
    // int32 headroom: products are at most 2^14, a block gets 7 (full) or 4
    // (folded) of them per K row and 2 K rows per complex row.
    static constexpr int EPOCH_STAGES = (FULL ? 8192 : 12288) / ROWS;
    struct Slot {                                              // what the scanners say about a stage
        int E[64 * SIDES], Eold[64 * SIDES];
        int fresh, epoch;
    };
    static constexpr size_t OFF_F = 0;
    static constexpr size_t OFF_S = OFF_F + (size_t)SLOTS * SIDES * FBYTES;
    static constexpr size_t OFF_SLOT = OFF_S + (size_t)GROUPS * BUF;
    static constexpr size_t OFF_BAR = (OFF_SLOT + SLOTS * sizeof(Slot) + 15) / 16 * 16;
    static constexpr size_t OFF_MISC = OFF_BAR + (3 * SLOTS + 2 * GROUPS) * 8;
    static constexpr size_t SMEM = OFF_MISC + 64 + 1024;       // + alignment slack
};
static_assert(Cfg<false>::SMEM <= 227 * 1024 && Cfg<true>::SMEM <= 227 * 1024, "a CTA's shared memory");

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

// What an operand's K rows are made of, from a complex entry (re, im).
enum Form { FORM_W, FORM_JW, FORM_V };

// Cuts eight complex rows of one column (v: re, im alternating) into the 16
// K bytes of every slice and stores slice t at base(t).
template <Form F, class Base>
__device__ __forceinline__ void cut(const double (&v)[16], double sc, Base base) {
    const double magic = __longlong_as_double(MAGIC_BITS);
    uint32_t w[4][SLICES];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint64_t y[4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const double re = v[4 * q + 2 * r], im = v[4 * q + 2 * r + 1];
            double a = re, b = im;
            if (F == FORM_JW) { a = -im; b = re; }
            if (F == FORM_V) { a = re - im; b = re + im; }
            y[2 * r] = (uint64_t)__double_as_longlong(fma(a, sc, magic)) << 4;
            y[2 * r + 1] = (uint64_t)__double_as_longlong(fma(b, sc, magic)) << 4;
        }
        slice_words(y, w[q]);
    }
#pragma unroll
    for (int t = 0; t < SLICES; ++t)
        *reinterpret_cast<uint4*>(base(t)) = make_uint4(w[0][t], w[1][t], w[2][t], w[3][t]);
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

template <bool FULL>
__global__ void __launch_bounds__(Cfg<FULL>::THREADS, 1)
split_gram_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int64_t rows,
                  SplitShape sh, double* __restrict__ partial, SplitStat* __restrict__ stats, const ChainStatus* st,
                  int gate, int chunk0) {
    if (gated_off(st, gate)) return;
    using C = Cfg<FULL>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    typename C::Slot* slots = reinterpret_cast<typename C::Slot*>(smem + C::OFF_SLOT);
    uint64_t* fp_full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);   // a stage's rows have landed
    uint64_t* fp_empty = fp_full + C::SLOTS;                              // scanned and loaded by its slicers
    uint64_t* sc_full = fp_empty + C::SLOTS;                              // scanned
    uint64_t* sl_full = sc_full + C::SLOTS;                               // a group's slices are written
    uint64_t* sl_empty = sl_full + C::GROUPS;                             // and consumed by the MMAs
    int* misc = reinterpret_cast<int*>(smem + C::OFF_MISC);
    volatile int* abort_flag = misc;
    int* bad_flag = misc + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(misc + 2);
    volatile int* fresh_flag = misc + 4;   // [GROUPS]

    int ti, tj, tile;
    split_tile_of(sh, FULL, (int)blockIdx.x, ti, tj, tile);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chunk = chunk0 + (int)blockIdx.y;
    const int64_t row0 = (int64_t)chunk * sh.chunk_rows;
    const int64_t row_end = min(rows, row0 + sh.chunk_rows);
    const int nstages = (int)((row_end - row0 + ROWS - 1) / ROWS);
    double* P = partial + ((size_t)tile * sh.nchunks + chunk) * SPLIT_TILE_DOUBLES;
    SplitStat* stat = stats + (size_t)tile * sh.nchunks + chunk;

    if (threadIdx.x == 0) {
        for (int b = 0; b < C::SLOTS; ++b) {
            mbar_init(&fp_full[b], 1);
            mbar_init(&fp_empty[b], 4 + C::SCANNERS / 32);
            mbar_init(&sc_full[b], C::SCANNERS);
        }
        for (int b = 0; b < C::GROUPS; ++b) {
            mbar_init(&sl_full[b], 4);
            mbar_init(&sl_empty[b], 1);
        }
        *abort_flag = 0;
        *bad_flag = 0;
        mbar_fence_init();
    }
    if constexpr (!FULL) {
        // The last A operand of a folded tile has one slice only: its rows
        // 64-127 are zero for good.
        for (int e = threadIdx.x; e < C::GROUPS * (ATILE / 2) / 16; e += blockDim.x) {
            const int b = e / ((ATILE / 2) / 16), o = e - b * ((ATILE / 2) / 16);
            reinterpret_cast<uint4*>(smem + C::OFF_S + (size_t)b * C::BUF + 3 * ATILE + ATILE / 2)[o] =
                make_uint4(0, 0, 0, 0);
        }
    }
    if (warp == 0) umma::tmem_alloc(tmem_slot, TMEM_COLS);
    umma::fence_smem_to_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t taddr = *tmem_slot;

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
                const bool fresh = fresh_flag[g] != 0;
                const uint32_t abase = smem_u32(smem + C::OFF_S + (size_t)g * C::BUF);
                const uint32_t bbase = abase + C::NA * ATILE;
#pragma unroll
                for (int a = 0; a < C::NA; ++a) {
                    const int first = FULL ? a : 2 * a;      // accumulator block of slice 1 of B
                    const int ntot = 64 * (SLICES - first);
#pragma unroll
                    for (int off = 0; off < ntot; off += 256) {
                        const int n = ntot - off < 256 ? ntot - off : 256;
                        umma::mma_s8(taddr + 64 * first + off, desc_sw32(abase + a * ATILE),
                                     desc_sw32(bbase + off * 32), umma::idesc_s8s8_s32(128, n), !(fresh && a == 0));
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
        const int g = warp >> 2, q = warp & 3;
        const int t128 = threadIdx.x & 127;
        const int j = t128 & 63, kq = t128 >> 6;             // this thread's column and 8-row box
        const int prow = 32 * q + lane;                      // its row of the accumulators
        const uint32_t tmem_lane = taddr + ((uint32_t)(32 * q) << 16);
        unsigned char* abuf = smem + C::OFF_S + (size_t)g * C::BUF;
        unsigned char* bbuf = abuf + C::NA * ATILE;
        const uint32_t off_lo = sw32_offset(j, kq), off_hi = sw32_offset(64 + j, kq);
        // Waits are decided by the whole warp together, so that a warp leaves
        // the loop as one.
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0;
        };
        auto load = [&](const unsigned char* tile_base, double (&v)[16]) {
            const unsigned char* col = tile_base + (size_t)kq * (FBYTES / 2) + j * 128;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const double2 z = *reinterpret_cast<const double2*>(col + ((r ^ (j & 7)) << 4));
                v[2 * r] = z.x;
                v[2 * r + 1] = z.y;
            }
        };
        // Drains the accumulators once the MMAs of `stage` have finished.
        auto drain = [&](int stage, const int* EA, const int* EB, bool initialized) {
            if (!wait(&sl_empty[stage % C::GROUPS], (stage / C::GROUPS) & 1)) return false;
            umma::fence_after_sync();
            drain_epoch<FULL>(tmem_lane, EA, EB, prow, P, initialized);
            umma::fence_before_sync();
            return true;
        };
        bool ok = true;
        uint32_t gph = 1;                                     // parity of this group's previous commit
        int s = g;
        for (; s < nstages; s += C::GROUPS) {
            const int b = s % C::SLOTS;
            const uint32_t ph = (s / C::SLOTS) & 1;
            if (!wait(&sc_full[b], ph) || !wait(&fp_full[b], ph) || *abort_flag) { ok = false; break; }
            const typename C::Slot& slot = slots[b];
            const bool fresh = slot.fresh != 0;
            // This group's buffer is free once its previous stage's MMAs are
            // done (waited for before a drain, too: it leaves the barrier of
            // stage s - 1 at most one phase behind).
            if (s >= C::GROUPS && !wait(&sl_empty[g], gph)) { ok = false; break; }
            // A new epoch: the MMAs of the one before it all precede this
            // stage's, which wait for this group.
            if (fresh && s > 0 &&
                !drain(s - 1, slot.Eold, slot.Eold + (FULL ? 64 : 0), slot.epoch > 1)) { ok = false; break; }
            const unsigned char* f = smem + C::OFF_F + (size_t)b * C::SIDES * FBYTES;
            const int EA = slot.E[j], EB = slot.E[(FULL ? 64 : 0) + j];
            const double sca = EA == SPLIT_E_UNSET ? 0.0 : pow2((FULL ? 51 : 50) - EA);
            const double scb = EB == SPLIT_E_UNSET ? 0.0 : pow2(51 - EB);
            auto release = [&]() {
                __syncwarp();
                if (lane == 0) mbar_arrive(&fp_empty[b]);
            };
            double v[16];
            if constexpr (FULL) {
                load(f + FBYTES, v);
                cut<FORM_W>(v, scb, [&](int t) { return bbuf + off_lo + t * (64 * 32); });
                load(f, v);
                release();
                cut<FORM_W>(v, sca, [&](int t) { return abuf + t * ATILE + off_lo; });
                cut<FORM_JW>(v, sca, [&](int t) { return abuf + t * ATILE + off_hi; });
            } else {
                load(f, v);
                release();
                cut<FORM_W>(v, scb, [&](int t) { return bbuf + off_lo + t * (64 * 32); });
                cut<FORM_V>(v, sca, [&](int t) { return abuf + (t >> 1) * ATILE + ((t & 1) ? off_hi : off_lo); });
            }
            if (t128 == 0) fresh_flag[g] = fresh ? 1 : 0;
            umma::fence_smem_to_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sl_full[g]);
            gph ^= 1u;
        }
        if (!ok) *abort_flag = 1;
        // The group of the last stage drains the last epoch.
        if (ok && nstages > 0 && s - C::GROUPS == nstages - 1) {
            const typename C::Slot& slot = slots[(nstages - 1) % C::SLOTS];
            if (!drain(nstages - 1, slot.E, slot.E + (FULL ? 64 : 0), slot.epoch > 0)) *abort_flag = 1;
        }
    } else {
        // ---- scanners: scales, a few stages ahead of the slicers ----
        const int c = (int)threadIdx.x - C::SLICERS - 64;    // input column: A's 0-63, then B's
        auto any = [](bool p) -> bool {
            uint32_t r;
            asm volatile(
                "{\n\t.reg .pred a, b;\n\t"
                "setp.ne.u32 a, %1, 0;\n\t"
                "barrier.cta.red.or.pred b, 1, %2, a;\n\t"
                "selp.u32 %0, 1, 0, b;\n\t}"
                : "=r"(r)
                : "r"((uint32_t)p), "n"(C::SCANNERS)
                : "memory");
            return r != 0;
        };
        int E = SPLIT_E_UNSET;
        // |x| < 2^E (1 - 2^-7) in terms of the high word of x; while the
        // scale is unset every normal number is past it.
        uint32_t limit = 0x00100000u;
        uint32_t tiny = 0;                                   // bits of subnormal entries under an unset scale
        bool bad = false;
        double sq[4] = {0.0, 0.0, 0.0, 0.0};
        int b = 0, epoch = -1, epoch_start = 0;
        uint32_t ph = 0;
        for (int s = 0; s < nstages; ++s) {
            const bool landed = mbar_wait(&fp_full[b], ph);
            const bool stop = !landed || *abort_flag;
            const unsigned char* col =
                smem + C::OFF_F + ((size_t)b * C::SIDES + (c >> 6)) * FBYTES + (c & 63) * 128;
            uint32_t mx = 0, low = 0;
            if (!stop) {
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const double2 z =
                        *reinterpret_cast<const double2*>(col + (r >> 3) * (FBYTES / 2) + (((r & 7) ^ (c & 7)) << 4));
                    mx = max(mx, (uint32_t)__double2hiint(z.x) & 0x7FFFFFFFu);
                    mx = max(mx, (uint32_t)__double2hiint(z.y) & 0x7FFFFFFFu);
                    low |= (uint32_t)__double2loint(z.x) | (uint32_t)__double2loint(z.y);
                    sq[r & 1] = fma(z.x, z.x, sq[r & 1]);
                    sq[2 + (r & 1)] = fma(z.y, z.y, sq[2 + (r & 1)]);
                }
            }
            bool over = mx >= limit;
            if (mx >= 0x7FF00000u) { bad = true; over = false; }   // Inf or NaN
            if (E == SPLIT_E_UNSET && mx < 0x00100000u) tiny |= mx | low;
            const bool epoch_full = s - epoch_start >= C::EPOCH_STAGES;
            const int Eold = E;
            bool any_over = false;
            if (any(over || stop)) {
                if (any(stop)) {
                    *abort_flag = 1;
                    break;
                }
                any_over = true;
                if (over) {
                    // The maximum lies in [2^e, 2^(e + 1)), e = the exponent:
                    // the scale leaves HEADROOM bits above that.
                    E = (int)(mx >> 20) - 1023 + 1 + HEADROOM;
                    // The limit's exponent stays in range: a scale past it is
                    // refused afterwards by split_sum_kernel anyway.
                    limit = ((uint32_t)min(max(E - 1 + 1023, 1), 0x7FE) << 20) | 0xFC000u;
                }
            }
            const bool fresh = s == 0 || any_over || epoch_full;
            if (fresh) {
                ++epoch;
                epoch_start = s;
            }
            slots[b].E[c] = E;
            slots[b].Eold[c] = Eold;
            if (c == 0) {
                slots[b].fresh = fresh ? 1 : 0;
                slots[b].epoch = epoch;
            }
            mbar_arrive(&sc_full[b]);
            __syncwarp();
            if (lane == 0) mbar_arrive(&fp_empty[b]);
            if (++b == C::SLOTS) { b = 0; ph ^= 1u; }
        }
        if (bad) *bad_flag = 1;
        stat->E[c] = E;
        stat->tiny[c] = E == SPLIT_E_UNSET && tiny != 0 ? 1 : 0;
        stat->sumsq[c] = (sq[0] + sq[1]) + (sq[2] + sq[3]);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (threadIdx.x == 0) stat->invalid = (*abort_flag || *bad_flag) ? 1 : 0;
    if (warp == 0) umma::tmem_dealloc(taddr, TMEM_COLS);
}

// Blocks 0..63 of a tile: its columns summed over the chunks in a fixed order
// (four interleaved runs of chunks, then the four), a folded tile's two halves
// added. Block 64: the tile's verdict.
//
// The verdict compares what the slices leave out with what the column weighs.
// With scale 2^E an entry is off by at most 2^(E - 51) (V: 2^(E - 50)), which
// reaches G_ij as an error of about 2^(E_j - 50) / sqrt(12) ||a_i||; the
// products left out (three digit pairs a K row, digits of standard deviation
// 74) add about sqrt(6 N) 74^2 2^(E_i + E_j - 70). Both stay below
// 2^-54 ||a_i|| ||a_j||, under the rounding of the FP64 sums themselves, when
//     ||a_j||^2 >= 4^E_j max(21.4, 0.21 sqrt(N)),
// which the kernel checks per column (N Gaussian rows give about 2 N / 400).
// A spike that dwarfs the rest of its column fails it, as do Inf and NaN, a
// scale whose products could leave the FP64 range, and a wait that gave up:
// the caller then computes the tile in FP64 instead.
constexpr int SUM_THREADS = 512;

__global__ void __launch_bounds__(SUM_THREADS)
split_sum_kernel(SplitShape sh, int64_t rows, const double* __restrict__ partial, const SplitStat* __restrict__ stats,
                 double* __restrict__ sums, int* __restrict__ verdict, const ChainStatus* st, int gate) {
    if (gated_off(st, gate)) return;
    __shared__ double red[SUM_THREADS];
    __shared__ int redE[SUM_THREADS];
    __shared__ int flags;
    const int tile = blockIdx.y, tid = threadIdx.x;
    const int m = tid & 127, part = tid >> 7;
    const bool full = !sh.hermitian || tile >= sh.nt_a;
    if (blockIdx.x < 64) {
        const double* p = partial + (size_t)tile * sh.nchunks * SPLIT_TILE_DOUBLES + blockIdx.x * 128 + m;
        double s = 0.0;
#pragma unroll 8
        for (int c = part; c < sh.nchunks; c += 4) s += p[(size_t)c * SPLIT_TILE_DOUBLES];
        red[tid] = s;
        __syncthreads();
        if (tid >= 128) return;
        s = (red[tid] + red[128 + tid]) + (red[256 + tid] + red[384 + tid]);
        if (!full) {
            __syncthreads();
            red[tid] = s;
            __syncthreads();
            if (tid >= 64) return;
            s += red[64 + tid];
        }
        sums[(size_t)tile * SPLIT_TILE_DOUBLES + blockIdx.x * 128 + m] = s;
        return;
    }
    if (tid == 0) flags = 0;
    __syncthreads();
    const int columns = full ? 128 : 64;
    int E = SPLIT_E_UNSET, mine = 0;
    double s = 0.0;
    for (int c = part; c < sh.nchunks; c += 4) {
        const SplitStat& x = stats[(size_t)tile * sh.nchunks + c];
        if (m == 0 && x.invalid) mine |= SPLIT_INVALID;
        if (m < columns) {
            E = max(E, x.E[m]);
            s += x.sumsq[m];
            if (x.tiny[m]) mine |= SPLIT_INACCURATE;
        }
    }
    red[tid] = s;
    redE[tid] = E;
    __syncthreads();
    if (tid < columns) {
        s = (red[tid] + red[128 + tid]) + (red[256 + tid] + red[384 + tid]);
        E = max(max(redE[tid], redE[128 + tid]), max(redE[256 + tid], redE[384 + tid]));
        if (E != SPLIT_E_UNSET &&
            !(E >= -450 && E <= 450 && s >= fmax(21.4, 0.21 * sqrt((double)rows)) * pow2(2 * E)))
            mine |= SPLIT_INACCURATE;
    }
    if (mine) atomicOr(&flags, mine);
    __syncthreads();
    if (tid == 0) verdict[tile] = flags;
}

template <bool FULL>
static int launch(const CUtensorMap& ma, const CUtensorMap& mb, int64_t rows, const SplitShape& sh, int ntiles,
                  double* partial, SplitStat* stats, cudaStream_t stream, const ChainStatus* st, int gate, int chunk0,
                  int chunk1) {
    using C = Cfg<FULL>;
    FB_CUDA(cudaFuncSetAttribute(split_gram_kernel<FULL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM),
            "cudaFuncSetAttribute(split_gram_kernel)");
    split_gram_kernel<FULL><<<dim3((unsigned)ntiles, (unsigned)(chunk1 - chunk0)), C::THREADS, C::SMEM, stream>>>(
        ma, mb, rows, sh, partial, stats, st, gate, chunk0);
    FB_LAUNCHED("split_gram_kernel");
    return FB_OK;
}

}  // namespace split

// One chunk per SM for the launch with fewer tiles, in whole stages.
SplitShape split_shape(int64_t rows, int kA, int kB, bool hermitian) {
    SplitShape sh{};
    sh.nt_a = (kA + 63) / 64;
    sh.nt_b = (kB + 63) / 64;
    sh.hermitian = hermitian ? 1 : 0;
    sh.ntiles = hermitian ? sh.nt_a * (sh.nt_a + 1) / 2 : sh.nt_a * sh.nt_b;
    int smallest = sh.ntiles;
    if (hermitian && sh.nt_a > 1) smallest = std::min(sh.nt_a, sh.nt_a * (sh.nt_a - 1) / 2);
    const int64_t stages = (rows + SPLIT_STAGE_ROWS - 1) / SPLIT_STAGE_ROWS;
    const int64_t target = std::max<int64_t>(1, sm_count() / smallest);
    sh.chunk_rows = std::max<int64_t>(1, (stages + target - 1) / target) * SPLIT_STAGE_ROWS;
    sh.nchunks = (int)((rows + sh.chunk_rows - 1) / sh.chunk_rows);
    return sh;
}

SplitLayout split_layout(const SplitShape& sh) {
    SplitLayout L{};
    const size_t parts = (size_t)sh.ntiles * (size_t)(sh.nchunks > 0 ? sh.nchunks : 1);
    L.verdict = 0;
    L.sums = align_up((size_t)sh.ntiles * sizeof(int), 256);
    L.stats = L.sums + (size_t)sh.ntiles * SPLIT_TILE_DOUBLES * sizeof(double);
    L.partial = align_up(L.stats + parts * sizeof(SplitStat), 256);
    L.total = L.partial + parts * SPLIT_TILE_DOUBLES * sizeof(double);
    return L;
}

int split_partials_enqueue(const z64* A, int64_t lda, const z64* B, int64_t ldb, int64_t rows, int kA, int kB,
                           const SplitShape& sh, void* workspace, cudaStream_t stream, const ChainStatus* st, int gate,
                           int chunk0, int chunk1) {
    if (chunk0 < 0) chunk0 = 0;
    if (chunk1 > sh.nchunks) chunk1 = sh.nchunks;
    if (chunk0 >= chunk1) return FB_OK;
    const SplitLayout L = split_layout(sh);
    char* ws = static_cast<char*>(workspace);
    double* partial = reinterpret_cast<double*>(ws + L.partial);
    SplitStat* stats = reinterpret_cast<SplitStat*>(ws + L.stats);
    CUtensorMap ma, mb;
    FB_TRY(encode_panel_map(&ma, A, rows, kA, lda, 64));
    FB_TRY(encode_panel_map(&mb, B, rows, kB, ldb, 64));
    const int full = sh.hermitian ? sh.ntiles - sh.nt_a : sh.ntiles;
    if (sh.hermitian)
        FB_TRY(split::launch<false>(ma, mb, rows, sh, sh.nt_a, partial, stats, stream, st, gate, chunk0, chunk1));
    if (full > 0)
        FB_TRY(split::launch<true>(ma, mb, rows, sh, full, partial, stats, stream, st, gate, chunk0, chunk1));
    return FB_OK;
}

int split_sum_enqueue(int64_t rows, const SplitShape& sh, void* workspace, cudaStream_t stream, const ChainStatus* st,
                      int gate) {
    const SplitLayout L = split_layout(sh);
    char* ws = static_cast<char*>(workspace);
    split::split_sum_kernel<<<dim3(65, (unsigned)sh.ntiles), split::SUM_THREADS, 0, stream>>>(
        sh, rows, reinterpret_cast<const double*>(ws + L.partial), reinterpret_cast<const SplitStat*>(ws + L.stats),
        reinterpret_cast<double*>(ws + L.sums), reinterpret_cast<int*>(ws + L.verdict), st, gate);
    FB_LAUNCHED("split_sum_kernel");
    return FB_OK;
}

}  // namespace fb

