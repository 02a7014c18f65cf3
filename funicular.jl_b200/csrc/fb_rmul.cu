// The tensor-core right products (fb_rmul.cuh): D <- beta D + A1 L + A2 C and
// D <- beta D + A C in rmul_dmma_kernel, tall D <- A C in rmul_pair_kernel.
//
// rmul_dmma_kernel: a team of one or two warps owns 8 rows at a time, each warp a contiguous
// share of the output n-tiles. A warp streams the rows' entries one k-step
// (two complex columns) at a time, loading each entry of A1 and A2 once (the
// second warp of a team finds them in L1), and keeps its n-tiles in its
// accumulators, so each output entry is written once. The loads run two
// groups of four k-steps ahead of the products; the group after that waits for
// the products of the current one, which bounds the registers the prefetch
// holds.
#include <algorithm>

#include "fb_rmul.cuh"
#include "fb_tma.cuh"

namespace fb {

constexpr int RM_THREADS = 512;
// Warps that share one 8-row unit, each taking a contiguous share of the
// output n-tiles: wide factors split in two, which halves the accumulators a
// thread holds and lets 16 warps run on an SM instead of 8.
__host__ __device__ constexpr int rm_split(int ntn) { return ntn >= 8 ? 2 : 1; }

template <int NTK, int NTN>
__global__ void __launch_bounds__(RM_THREADS, 1)
rmul_dmma_kernel(z64* D, int64_t ldd, const z64* A1, int64_t lda1, const z64* A2, int64_t lda2, int64_t rows,
                 int K, int n, const double* __restrict__ gdense, const double* __restrict__ glower,
                 const z64* __restrict__ Cm, int64_t ldcm, z64 beta,
                 int use_beta, int zero, int inplace, const ChainStatus* st, int gate) {
    if (gated_off(st, gate)) return;
    constexpr int NS = 2 * NTK;               // k-steps
    constexpr int NT = NTN;                   // output n-tiles
    constexpr int SPLIT = rm_split(NTN);      // warps sharing one 8-row unit
    constexpr int NH = (NT + SPLIT - 1) / SPLIT;  // n-tiles of one warp
    constexpr int G = 4;                      // k-steps whose inputs are loaded together
    constexpr int NG = (NS + G - 1) / G;
    constexpr bool SQUARE = NTK == NTN;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* fd = reinterpret_cast<double*>(smem_raw);
    double* fl = fd + dense_frag_doubles(NTK, NTN);
    const bool lower = SQUARE && A1 != nullptr;
    if (gdense == nullptr) {
        // The factor given as a K x n matrix (the plain product A2 C): every
        // CTA lays out the fragments of the whole template-sized factor
        // itself, zero past K and n.
        for (int e = threadIdx.x; e < dense_frag_doubles(NTK, NTN); e += blockDim.x) {
            const int l = e & 31, q = e >> 5;
            const int s = q / NTN, t = q - s * NTN;
            fd[e] = frag_entry(Cm, ldcm, K, n, s, t, l, 1.0);
        }
    } else {
        const double2* s2 = reinterpret_cast<const double2*>(gdense);
        double2* d2 = reinterpret_cast<double2*>(fd);
        for (int e = threadIdx.x; e < dense_frag_doubles(NTK, NTN) / 2; e += blockDim.x) d2[e] = s2[e];
        if (lower) {
            const double2* l2 = reinterpret_cast<const double2*>(glower);
            double2* dl = reinterpret_cast<double2*>(fl);
            for (int e = threadIdx.x; e < lower_frag_doubles(NTN) / 2; e += blockDim.x) dl[e] = l2[e];
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rr = lane >> 2, cq = lane & 3, acol = cq >> 1;
    const int apart = lane & 1;
    const int64_t units = (rows + 7) / 8;
    const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
    const int t0 = (int)(gw % SPLIT) * NH;    // this warp's first n-tile
    const int64_t teams = (int64_t)gridDim.x * (blockDim.x >> 5) / SPLIT;
    for (int64_t u = gw / SPLIT; u < units; u += teams) {
        const int64_t row = u * 8 + rr;
        const bool live = row < rows;
        const int64_t r0 = live ? row : 0;
        // This lane's entries of k-steps gG .. gG + G - 1 of both inputs.
        auto load_group = [&](int g, double (&b2)[G], double (&b1)[G], const z64* p2, const z64* p1) {
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const int s = g * G + j;
                const int col = 2 * s + acol;
                const bool ok = s < NS && live && col < K;
                b2[j] = ok ? reinterpret_cast<const double*>(p2 + (int64_t)col * lda2)[apart] : 0.0;
                b1[j] = (ok && lower) ? reinterpret_cast<const double*>(p1 + (int64_t)col * lda1)[apart] : 0.0;
            }
        };
        double acc[NH][2];
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            const int col = 4 * (t0 + h) + cq;
            z64 d = zmake(0.0, 0.0);
            if (use_beta && live && col < n) d = zmul(beta, D[r0 + (int64_t)col * ldd]);
            acc[h][0] = d.x;
            acc[h][1] = d.y;
        }
        const z64* p2 = A2 + r0;
        const z64* p1 = lower ? A1 + r0 : A2 + r0;
        double c2[G], c1[G], n2[G], n1[G];
        load_group(0, c2, c1, p2, p1);
        load_group(1, n2, n1, p2, p1);
        // Two groups of loads in flight: group g + 2 is issued once group
        // g's products are done, so its registers are not held any longer.
#pragma unroll
        for (int g = 0; g < NG; ++g) {
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const int s = g * G + j;
                if (s >= NS) break;
                // This step's fragments are read once the previous step's
                // first product is done, not hoisted further ahead.
                const double step_chain = acc[0][0];
                const double* fp = hold(fd + (s * NT + t0) * 32 + lane, step_chain, zero);
#pragma unroll
                for (int h = 0; h < NH; ++h)
                    if (SPLIT == 1 || t0 + h < NT) dmma_884(acc[h][0], acc[h][1], c2[j], fp[h * 32]);
                if (SQUARE && lower) {
                    const double* lp = hold(fl + (lower_step_offset(s) + t0) * 32 + lane, step_chain, zero);
#pragma unroll
                    for (int h = 0; h < NH; ++h)
                        if (t0 + h <= s / 2 && t0 + h < NT) dmma_884(acc[h][0], acc[h][1], c1[j], lp[h * 32]);
                }
            }
#pragma unroll
            for (int j = 0; j < G; ++j) {
                c2[j] = n2[j];
                c1[j] = n1[j];
            }
            if (g + 2 < NG) {
                const double chain = acc[0][0];
                load_group(g + 2, n2, n1, hold(p2, chain, zero), hold(p1, chain, zero));
            }
        }
        // When D is one of the inputs, the other warp of the team may still be
        // reading these rows: both finish reading before either writes.
        if (SPLIT > 1 && inplace) asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / SPLIT), "r"(32 * SPLIT) : "memory");
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            const int col = 4 * (t0 + h) + cq;
            if (live && col < n && t0 + h < NT) D[row + (int64_t)col * ldd] = zmake(acc[h][0], acc[h][1]);
        }
    }
}

// The tall product by a dense factor alone, D <- A C. A warp owns two 8-row
// units at a time and all n-tiles, so a fragment read from shared memory feeds
// two MMAs (with one unit a warp the fragment reads took half of the shared
// memory pipe), and keeps 4 NTN accumulators a lane. The rows come by TMA, 16
// columns of both units a stage, through a ring of the warp's own that its
// lane 0 refills across units. Each accumulator adds the k-steps in order, as
// in rmul_dmma_kernel: the bits are the same.
// Bound at 2500003 x 64 by 64 x 64: the FP64 tensor pipe, 2.23 ms (memory
// 0.78). Measured there, rmul_dmma_kernel / this: 2.74 / 2.42 ms; 64 x 40
// 2.26 / 1.71, 48 x 48 1.92 / 1.44, 32 x 32 1.12 / 0.68, 20 x 50 2.20 / 0.78
// (K runs in steps of two columns here, there in the template's).
// Narrow results leave the registers for twice the warps.
__host__ __device__ constexpr int rp_warps(int ntn) { return ntn <= 4 ? 16 : 8; }
constexpr int RP_STAGE = 4096;                       // 2 units x 8 rows x 16 columns
constexpr size_t RP_SMEM = 227 * 1024 - 2048;        // fragments and rings

template <int NTN>
__global__ void __launch_bounds__(32 * rp_warps(NTN), 1)
rmul_pair_kernel(const __grid_constant__ CUtensorMap tmA, z64* D, int64_t ldd, int64_t rows, int K, int n,
                 const double* __restrict__ gdense, const z64* __restrict__ Cm, int64_t ldcm, int slots, int cwarps,
                 int zero, const ChainStatus* st, int gate) {
    if (gated_off(st, gate)) return;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int WARPS = rp_warps(NTN);
    const int ngroups = (K + 15) / 16;               // stages a unit pair
    const int ksteps = (K + 1) / 2;
    unsigned char* ring = smem + warp * slots * RP_STAGE;
    double* fd = reinterpret_cast<double*>(smem + WARPS * slots * RP_STAGE);
    uint64_t* full = reinterpret_cast<uint64_t*>(fd + ksteps * NTN * 32) + warp * slots;

    const int pairs = (int)((rows + 15) / 16);
    const int stride = (int)gridDim.x * cwarps;
    const int first = warp < cwarps ? (int)blockIdx.x * cwarps + warp : pairs;
    int fu = first, fg = 0;                          // the next stage to ask for
    auto fetch = [&](int b) {
        mbar_arrive_expect_tx(&full[b], RP_STAGE);
        tma_load_2d(ring + b * RP_STAGE, &tmA, fu * 32, fg * 16, &full[b]);
        tma_load_2d(ring + b * RP_STAGE + RP_STAGE / 2, &tmA, fu * 32 + 16, fg * 16, &full[b]);
        if (++fg == ngroups) { fg = 0; fu += stride; }
    };
    if (lane == 0) {
        for (int b = 0; b < slots; ++b) mbar_init(&full[b], 1);
        mbar_fence_init();
        for (int b = 0; b < slots && fu < pairs; ++b) fetch(b);
    }
    // The factor's fragments, zero past K and n, 16 loads in flight a thread.
    const int entries = ksteps * NTN * 32;
    for (int e0 = threadIdx.x; e0 < entries; e0 += 16 * 32 * WARPS) {
        double v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int e = e0 + i * 32 * WARPS;
            const int q = e >> 5, s = q / NTN;
            v[i] = e >= entries ? 0.0 : gdense ? gdense[e] : frag_entry(Cm, ldcm, K, n, s, q - s * NTN, lane, 1.0);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (e0 + i * 32 * WARPS < entries) fd[e0 + i * 32 * WARPS] = v[i];
    }
    __syncthreads();

    const int rr = lane >> 2, cq = lane & 3, acol = cq >> 1, apart = lane & 1;
    // Swizzled offsets of row rr in columns 2 s + acol of a box, s = 0..3 (and
    // the same eight columns further on).
    int off[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) off[s] = (2 * s + acol) * 128 + ((rr ^ (2 * s + acol)) << 4) + apart * 8;
    bool ok = true;
    int b = 0;
    uint32_t phase = 0;
    for (int u = first; u < pairs; u += stride) {
        const int64_t row = (int64_t)u * 16 + rr;
        const bool live0 = row < rows, live1 = row + 8 < rows;
        double acc[2][NTN][2] = {};
        const double* fp = fd + lane;
        for (int g = 0; g < ngroups; ++g) {
            ok = ok && mbar_wait_warp(&full[b], phase);
            const unsigned char* box = ring + b * RP_STAGE;
            double a[2][8];
            uint32_t seen = 0;
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                a[0][s] = *reinterpret_cast<const double*>(box + (s >> 2) * 1024 + off[s & 3]);
                a[1][s] = *reinterpret_cast<const double*>(box + RP_STAGE / 2 + (s >> 2) * 1024 + off[s & 3]);
            }
#pragma unroll
            for (int s = 0; s < 8; ++s) { mark_loaded(seen, a[0][s]); mark_loaded(seen, a[1][s]); }
            __syncwarp();
            if (lane == 0 && ok && fu < pairs) fetch(b + (int)(seen & zero));
            if (++b == slots) { b = 0; phase ^= 1u; }
            // Rows that never arrived come out as NaN.
            if (!ok) a[0][0] = a[1][0] = __longlong_as_double(0x7ff8000000000000ll);
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (8 * g + s >= ksteps) break;
                // A step's fragments are read once the previous step's first
                // product is done, not hoisted further ahead.
                fp = hold(fp, acc[0][0][0], zero);
#pragma unroll
                for (int t = 0; t < NTN; ++t) {
                    const double bv = fp[t * 32];
                    dmma_884(acc[0][t][0], acc[0][t][1], a[0][s], bv);
                    dmma_884(acc[1][t][0], acc[1][t][1], a[1][s], bv);
                }
                fp += NTN * 32;
            }
        }
#pragma unroll
        for (int t = 0; t < NTN; ++t) {
            const int col = 4 * t + cq;
            if (col >= n) continue;
            if (live0) D[row + (int64_t)col * ldd] = zmake(acc[0][t][0], acc[0][t][1]);
            if (live1) D[row + 8 + (int64_t)col * ldd] = zmake(acc[1][t][0], acc[1][t][1]);
        }
    }
}

// The same product on the FP64 pipes, for factors past 64: a thread per row,
// output columns in order, so D may be the same matrix as A1 (column j of the
// result reads columns l >= j of A1 only) but must not overlap A2.
__global__ void __launch_bounds__(128)
rmul_rows_kernel(z64* D, int64_t ldd, const z64* A1, int64_t lda1, const z64* __restrict__ A2, int64_t lda2,
                 int64_t rows, int K, int n, const z64* __restrict__ L, int64_t ldl, const z64* __restrict__ C,
                 int64_t ldc, z64 beta, int use_beta, const ChainStatus* st, int gate) {
    if (gated_off(st, gate)) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += stride) {
        for (int j = 0; j < n; ++j) {
            z64 acc = use_beta ? zmul(beta, D[r + (int64_t)j * ldd]) : zmake(0.0, 0.0);
            if (A1)
                for (int l = j; l < K; ++l) zmac(acc, A1[r + (int64_t)l * lda1], __ldg(L + l + (int64_t)j * ldl));
            for (int l = 0; l < K; ++l) zmac(acc, A2[r + (int64_t)l * lda2], __ldg(C + l + (int64_t)j * ldc));
            D[r + (int64_t)j * ldd] = acc;
        }
    }
}

template <int NTK, int NTN>
static int launch_rmul_dmma(z64* D, int64_t ldd, const z64* A1, int64_t lda1, const z64* A2, int64_t lda2,
                            int64_t rows, int K, int n, const double* fdense, const double* flower, z64 beta,
                            int use_beta, cudaStream_t stream, const ChainStatus* st, int gate,
                            const z64* Cm = nullptr, int64_t ldcm = 0) {
    const bool lower = NTK == NTN && A1 != nullptr;
    const size_t smem = (size_t)(dense_frag_doubles(NTK, NTN) + (lower ? lower_frag_doubles(NTN) : 0)) * sizeof(double);
    FB_ALLOW_SMEM((rmul_dmma_kernel<NTK, NTN>), smem);
    static PerDevice fit[2];
    int per_sm = 0;
    FB_TRY(blocks_per_sm(reinterpret_cast<const void*>(rmul_dmma_kernel<NTK, NTN>), RM_THREADS, smem, fit[lower], &per_sm));
    const int64_t units = (rows + 7) / 8;
    const int teams_per_cta = RM_THREADS / 32 / rm_split(NTN);
    int64_t need = (units + teams_per_cta - 1) / teams_per_cta;
    int64_t grid = (int64_t)sm_count() * per_sm;
    if (grid > need) grid = need;
    if (grid < 1) grid = 1;
    const int inplace = (D == A1 || D == A2) ? 1 : 0;
    rmul_dmma_kernel<NTK, NTN><<<(unsigned)grid, RM_THREADS, smem, stream>>>(
        D, ldd, lower ? A1 : nullptr, lda1, A2, lda2, rows, K, n, fdense, flower, Cm, ldcm, beta, use_beta, 0, inplace,
        st, gate);
    FB_LAUNCHED("rmul_dmma_kernel");
    return FB_OK;
}

template <int NTN>
static int launch_rmul_pair(z64* D, int64_t ldd, const z64* A, int64_t lda, int64_t rows, int K, int n,
                            const double* fdense, cudaStream_t stream, const ChainStatus* st, int gate, const z64* Cm,
                            int64_t ldcm) {
    constexpr int WARPS = rp_warps(NTN);
    const size_t frags = (size_t)(K + 1) / 2 * NTN * 32 * sizeof(double);
    const int slots = (int)std::min<size_t>((RP_SMEM - frags) / (WARPS * RP_STAGE), 4);
    const size_t smem = frags + (size_t)WARPS * slots * (RP_STAGE + sizeof(uint64_t)) + 1024;
    FB_ALLOW_SMEM(rmul_pair_kernel<NTN>, RP_SMEM + 2048);
    // The loads' coordinates are 32-bit: more rows than 2^30 go in slices.
    constexpr int64_t SLICE = (int64_t)1 << 30;
    for (int64_t r = 0; r < rows; r += SLICE) {
        const int64_t m = rows - r < SLICE ? rows - r : SLICE;
        CUtensorMap map;
        FB_TRY(encode_panel_map(&map, A + r, m, K, lda, 16));
        // A short panel spreads over the SMs before it fills them.
        const int64_t pairs = (m + 15) / 16, sms = sm_count();
        const int warps = (int)std::min<int64_t>((pairs + sms - 1) / sms, WARPS);
        const int64_t grid = std::min<int64_t>((pairs + warps - 1) / warps, sms);
        rmul_pair_kernel<NTN><<<(unsigned)grid, 32 * WARPS, smem, stream>>>(
            map, D + r, ldd, m, K, n, fdense, Cm, ldcm, slots, warps, 0, st, gate);
        FB_LAUNCHED("rmul_pair_kernel");
    }
    return FB_OK;
}

// D <- A C with the factor as fragments or as a matrix.
static int rmul_pair_enqueue(z64* D, int64_t ldd, const z64* A, int64_t lda, int64_t rows, int K, int n,
                             const double* fdense, cudaStream_t stream, const ChainStatus* st, int gate, const z64* Cm,
                             int64_t ldcm) {
    switch ((n + 3) / 4) {
#define FB_RP_CASE(t) \
    case t: return launch_rmul_pair<t>(D, ldd, A, lda, rows, K, n, fdense, stream, st, gate, Cm, ldcm);
        FB_RP_CASE(1) FB_RP_CASE(2) FB_RP_CASE(3) FB_RP_CASE(4) FB_RP_CASE(5) FB_RP_CASE(6) FB_RP_CASE(7) FB_RP_CASE(8)
        FB_RP_CASE(9) FB_RP_CASE(10) FB_RP_CASE(11) FB_RP_CASE(12) FB_RP_CASE(13) FB_RP_CASE(14) FB_RP_CASE(15)
        FB_RP_CASE(16)
#undef FB_RP_CASE
    }
    set_error(FB_EINVAL, "rmul: no template for a %d x %d factor", K, n);
    return FB_EINVAL;
}

// Whether the product by a dense factor runs in rmul_pair_kernel. Its units
// are twice as long and leave the last wave emptier, so short panels stay in
// rmul_dmma_kernel, and so do the narrowest, whose stages would be mostly
// padding, and those that add to D, whose loads only more warps can hide.
// Microseconds, rmul_dmma_kernel / rmul_pair_kernel: 64 x 64: 5000 rows 23 / 31,
// 1e5 rows 132 / 140, 2.6e5 rows 308 / 290; 8 x 20: 2.6e5 rows 46 / 31; 4 x 4:
// 2.6e5 rows 8 / 12, 2.5e6 rows 65 / 64; adding to D, 2^20 x 64 by 64 x 64: the
// whole adjoint it is part of 10.6 / 11.3 ms.
// TMA wants A on a 16-byte boundary.
static bool rmul_takes_pairs(const z64* A, int64_t rows, int K, int use_beta) {
    return rows >= (int64_t)1 << 18 && K >= 8 && !use_beta && ((uintptr_t)A & 15) == 0;
}

// D <- beta D (when use_beta) + A C for a K x n factor C given as a matrix,
// K, n <= 64, on the tensor cores. The template is the smallest one that
// holds the factor: square when K and n take the same number of 4-column
// tiles or K takes fewer (K padded with zeros), 64 rows of K otherwise.
int rmul_matrix_enqueue(z64* D, int64_t ldd, const z64* A, int64_t lda, int64_t rows, int K, int n, const z64* C,
                        int64_t ldc, z64 beta, int use_beta, cudaStream_t stream) {
    if (rows == 0 || n == 0) return FB_OK;
    if (K < 1 || K > RM_KMAX || n > RM_KMAX) {
        set_error(FB_EINVAL, "rmul: a %d x %d factor is past the 64 x 64 the tensor-core product takes", K, n);
        return FB_EINVAL;
    }
    if (rmul_takes_pairs(A, rows, K, use_beta))
        return rmul_pair_enqueue(D, ldd, A, lda, rows, K, n, nullptr, stream, nullptr, GATE_ALWAYS, C, ldc);
    const int ntk = (K + 3) / 4, ntn = (n + 3) / 4;
    if (ntk <= ntn) {
        switch (ntn) {
#define FB_RM_MSQ(t) \
    case t: return launch_rmul_dmma<t, t>(D, ldd, nullptr, 0, A, lda, rows, K, n, nullptr, nullptr, beta, use_beta, stream, nullptr, GATE_ALWAYS, C, ldc);
            FB_RM_MSQ(1) FB_RM_MSQ(2) FB_RM_MSQ(3) FB_RM_MSQ(4) FB_RM_MSQ(5) FB_RM_MSQ(6) FB_RM_MSQ(7) FB_RM_MSQ(8)
            FB_RM_MSQ(9) FB_RM_MSQ(10) FB_RM_MSQ(11) FB_RM_MSQ(12) FB_RM_MSQ(13) FB_RM_MSQ(14) FB_RM_MSQ(15)
            FB_RM_MSQ(16)
#undef FB_RM_MSQ
        }
    } else {
        switch (ntn) {
#define FB_RM_MWIDE(t) \
    case t: return launch_rmul_dmma<16, t>(D, ldd, nullptr, 0, A, lda, rows, K, n, nullptr, nullptr, beta, use_beta, stream, nullptr, GATE_ALWAYS, C, ldc);
            FB_RM_MWIDE(1) FB_RM_MWIDE(2) FB_RM_MWIDE(3) FB_RM_MWIDE(4) FB_RM_MWIDE(5) FB_RM_MWIDE(6) FB_RM_MWIDE(7)
            FB_RM_MWIDE(8) FB_RM_MWIDE(9) FB_RM_MWIDE(10) FB_RM_MWIDE(11) FB_RM_MWIDE(12) FB_RM_MWIDE(13)
            FB_RM_MWIDE(14) FB_RM_MWIDE(15)
#undef FB_RM_MWIDE
        }
    }
    set_error(FB_EINVAL, "rmul: no template for a %d x %d factor", K, n);
    return FB_EINVAL;
}

int rmul_enqueue(z64* D, int64_t ldd, const z64* A1, int64_t lda1, const z64* A2, int64_t lda2, int64_t rows,
                 int K, int n, const z64* L, int64_t ldl, const z64* C, int64_t ldc, const double* fdense,
                 const double* flower, z64 beta, int use_beta, cudaStream_t stream, const ChainStatus* st, int gate) {
    if (rows == 0 || n == 0) return FB_OK;
    if (A1 && K != n) { set_error(FB_EINVAL, "rmul: a lower triangular factor is square, got %d x %d", K, n); return FB_EINVAL; }
    const int ntk = (K + 3) / 4, ntn = (n + 3) / 4;
    if (K <= RM_KMAX && n <= RM_KMAX && (ntk == ntn || ntk == RM_KMAX / 4)) {
        if (A1 == nullptr && rmul_takes_pairs(A2, rows, K, use_beta))
            return rmul_pair_enqueue(D, ldd, A2, lda2, rows, K, n, fdense, stream, st, gate, nullptr, 0);
        if (ntk == ntn) {
            switch (ntn) {
#define FB_RM_SQ(t) \
    case t: return launch_rmul_dmma<t, t>(D, ldd, A1, lda1, A2, lda2, rows, K, n, fdense, flower, beta, use_beta, stream, st, gate);
                FB_RM_SQ(1) FB_RM_SQ(2) FB_RM_SQ(3) FB_RM_SQ(4) FB_RM_SQ(5) FB_RM_SQ(6) FB_RM_SQ(7) FB_RM_SQ(8)
                FB_RM_SQ(9) FB_RM_SQ(10) FB_RM_SQ(11) FB_RM_SQ(12) FB_RM_SQ(13) FB_RM_SQ(14) FB_RM_SQ(15) FB_RM_SQ(16)
#undef FB_RM_SQ
            }
        } else {
            switch (ntn) {
#define FB_RM_WIDE(t) \
    case t: return launch_rmul_dmma<16, t>(D, ldd, nullptr, 0, A2, lda2, rows, K, n, fdense, nullptr, beta, use_beta, stream, st, gate);
                FB_RM_WIDE(1) FB_RM_WIDE(2) FB_RM_WIDE(3) FB_RM_WIDE(4) FB_RM_WIDE(5) FB_RM_WIDE(6) FB_RM_WIDE(7)
                FB_RM_WIDE(8) FB_RM_WIDE(9) FB_RM_WIDE(10) FB_RM_WIDE(11) FB_RM_WIDE(12) FB_RM_WIDE(13)
                FB_RM_WIDE(14) FB_RM_WIDE(15)
#undef FB_RM_WIDE
            }
        }
    }
    int64_t grid = (int64_t)sm_count() * 8;
    int64_t need = (rows + 127) / 128;
    if (grid > need) grid = need;
    if (grid < 1) grid = 1;
    rmul_rows_kernel<<<(unsigned)grid, 128, 0, stream>>>(D, ldd, A1, lda1, A2, lda2, rows, K, n, L, ldl, C, ldc, beta,
                                                         use_beta, st, gate);
    FB_LAUNCHED("rmul_rows_kernel");
    return FB_OK;
}

}  // namespace fb
