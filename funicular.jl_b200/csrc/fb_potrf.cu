// cholesky_upper (src/panelblas.jl:148-155) as one CTA on the device: the
// k x k Cholesky of a Hermitian Gram matrix, the shifted retry, and the
// R2 * R product of cholqr2! (src/panelblas.jl:133,136), all FP64.
//
// The factor is held in shared memory: for k <= 64 in the solve plan's layout,
// so that the orthonormalization chain gets the plan of its next triangular
// solve from the same launch; as a packed upper triangle up to k = 160; in
// workspace memory beyond. Pivot test as LAPACK's zpotrf makes it: the
// factorization fails as soon as a pivot is not > 0 (this also catches NaN).
// On failure the matrix is reloaded with s = 11 N k eps(Float64) ||G||_F added
// to the diagonal and factored again; a second failure is reported, not
// shifted further.
//
// The shifted CholeskyQR3 of Fukaya, Kannan, Nakatsukasa, Zhang and Yamamoto
// (SIAM J. Sci. Comput. 2020) shifts its first pass unconditionally: with a
// unit roundoff u > 0 the kernel factors G + s I once, s = 11 (N k + k (k+1))
// u ||G||_F (||G||_F bounds ||Y||_2^2 from above, which keeps s inside the
// range the analysis allows for the condition numbers it targets).
#include "fb_factor.cuh"

namespace fb {

constexpr int POTRF_THREADS = 512;
constexpr int POTRF_PACKED_MAX_K = 160;

// Where the factor lives while it is made.
enum FactorStore { STORE_PLAN, STORE_PACKED, STORE_GLOBAL };

template <FactorStore S>
__global__ void __launch_bounds__(POTRF_THREADS, 1)
potrf_kernel(const z64* __restrict__ G, int64_t ldg, int k, int64_t N,
             z64* __restrict__ U, int64_t ldu, z64* __restrict__ gwork,
             ChainStatus* st, int pass, int gate, double forced_u, TrsmPlan* plan, double* __restrict__ frag,
             const z64* Rin, int64_t ldrin, z64* Rout, int64_t ldrout) {
    if (gated_off(st, gate)) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red_scratch[33];
    constexpr int LD = TR_PREP_LD;
    z64* W = S == STORE_GLOBAL ? gwork : reinterpret_cast<z64*>(smem_raw);
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
    auto at = [&](int i, int j) -> z64& {
        if (S == STORE_PLAN) return W[i * LD + j];
        if (S == STORE_PACKED) return W[i * k - i * (i + 1) / 2 + j];
        return W[(int64_t)i * k + j];
    };
    auto g = [&](int i, int j) { return G[i + (int64_t)j * ldg]; };
    double gnorm = 0.0, shift = 0.0;
    bool shifted = false;
    const bool ok = factor_shifted(g, k, N, forced_u, at, red_scratch, gnorm, shifted, shift);

    if (tid == 0 && st) {
        st->shifted[pass] = shifted ? 1 : 0;
        st->shift[pass] = shift;
        st->norm[pass] = gnorm;
        if (!ok) st->failed = pass;
    }
    if (!ok) return;

    for (int j = warp; j < k; j += nwarps)
        for (int i = lane; i < k; i += 32) U[i + (int64_t)j * ldu] = (i <= j) ? at(i, j) : zmake(0.0, 0.0);
    if (Rout) {
        // R = U Rin (U without Rin) over the caller's U, from the factor held
        // here: what the stores above left there is not read again.
        __syncthreads();
        for (int j = warp; j < k; j += nwarps)
            for (int i = lane; i < k; i += 32) {
                z64 acc = zmake(0.0, 0.0);
                if (!Rin && i <= j) acc = at(i, j);
                if (Rin)
                    for (int m = i; m <= j; ++m) zmac(acc, at(i, m), Rin[m + (int64_t)j * ldrin]);
                Rout[i + (int64_t)j * ldrout] = acc;
            }
    }
    if (S == STORE_PLAN && plan) {
        __syncthreads();
        z64* Xs = W + TR_KMAX * LD;
        const int KP = (k + TR_NB - 1) / TR_NB * TR_NB;
        for (int i = warp; i < KP; i += nwarps)
            for (int j = lane; j < KP; j += 32) {
                if (j >= k || i >= k || i > j) W[i * LD + j] = zmake(i == j ? 1.0 : 0.0, 0.0);
                Xs[i * LD + j] = zmake(0.0, 0.0);
            }
        __syncthreads();
        solve_plan(W, Xs, k, plan, frag);
    }
}

// R = U3 U2 U1 column by column: the product of the passes' factors, run once
// after the last pass instead of inside each pass's one-CTA factor step. A
// block per column; 32 rows a warp and, where that leaves warps, the sum over
// the columns of U cut into `parts` interleaved runs, added in order. U3
// counts only if a third pass ran, U1 may be NULL (R = U2); two_passes_only
// leaves R alone when a third pass is still to come. Latency-bound: eight
// loads a thread in flight.
constexpr int COMPOSE_THREADS = 512;

__global__ void __launch_bounds__(COMPOSE_THREADS)
compose_r_kernel(z64* __restrict__ R, int64_t ldr, int k, const z64* __restrict__ U1, int64_t ldu1,
                 const z64* __restrict__ U2, int64_t ldu2, const z64* __restrict__ U3, int64_t ldu3,
                 const ChainStatus* st, int two_passes_only) {
    if (st->failed) return;
    const bool shifted = (st->shifted[1] | st->shifted[2]) != 0;
    if (two_passes_only && shifted) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    z64* t = reinterpret_cast<z64*>(smem_raw);   // the column so far
    z64* red = t + k;                            // COMPOSE_THREADS partial sums
    const int j = blockIdx.x;
    if (!U1) {
        for (int i = threadIdx.x; i < k; i += blockDim.x) R[i + (int64_t)j * ldr] = U2[i + (int64_t)j * ldu2];
        return;
    }
    const bool third = U3 != nullptr && shifted;
    const int span = k < COMPOSE_THREADS ? (k + 31) / 32 * 32 : COMPOSE_THREADS;
    const int parts = COMPOSE_THREADS / span;
    const int part = threadIdx.x / span, lane = threadIdx.x - part * span;
    for (int i = threadIdx.x; i < k; i += blockDim.x) t[i] = U1[i + (int64_t)j * ldu1];
    __syncthreads();
    for (int f = 0; f < (third ? 2 : 1); ++f) {
        const z64* U = f ? U3 : U2;
        const int64_t ldu = f ? ldu3 : ldu2;
        for (int i0 = 0; i0 < k; i0 += span) {
            const int i = i0 + lane;
            z64 acc = zmake(0.0, 0.0);
            if (part < parts && i < k)
                for (int m0 = part; m0 <= j; m0 += 8 * parts) {
                    z64 u[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) u[q] = U[i + (int64_t)min(m0 + q * parts, j) * ldu];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int m = m0 + q * parts;
                        if (m >= i && m <= j) zmac(acc, u[q], t[m]);
                    }
                }
            // Rows i0 .. i0 + span of the result need t's rows from i0 on
            // only, so t can be overwritten strip by strip.
            red[threadIdx.x] = acc;
            __syncthreads();
            if (part == 0 && i < k) {
                for (int p = 1; p < parts; ++p) {
                    acc.x += red[p * span + lane].x;
                    acc.y += red[p * span + lane].y;
                }
                t[i] = acc;
                if (f == (third ? 1 : 0)) R[i + (int64_t)j * ldr] = acc;
            }
            __syncthreads();
        }
    }
}

int compose_r_enqueue(z64* R, int64_t ldr, int k, const z64* U1, int64_t ldu1, const z64* U2, int64_t ldu2,
                      const z64* U3, int64_t ldu3, const ChainStatus* st, int two_passes_only, cudaStream_t stream) {
    const size_t smem = (size_t)(k + COMPOSE_THREADS) * sizeof(z64);
    FB_ALLOW_SMEM(compose_r_kernel, smem);
    compose_r_kernel<<<k, COMPOSE_THREADS, smem, stream>>>(R, ldr, k, U1, ldu1, U2, ldu2, U3, ldu3, st,
                                                            two_passes_only);
    FB_LAUNCHED("compose_r_kernel");
    return FB_OK;
}

size_t potrf_gwork_bytes(int k) { return k > POTRF_PACKED_MAX_K ? (size_t)k * k * sizeof(z64) : 0; }

// plan and frag, when given (k <= 64 only), also receive the solve plan of U:
// what trsm_prepare_enqueue would make of it. Rout, when given, receives U Rin
// (U without Rin) from the same launch.
static int potrf_launch(const z64* G, int64_t ldg, int k, int64_t N, z64* U, int64_t ldu, z64* gwork,
                        ChainStatus* st, int pass, int gate, cudaStream_t stream, double forced_u, TrsmPlan* plan,
                        double* frag, const z64* Rin, int64_t ldrin, z64* Rout, int64_t ldrout) {
#define FB_POTRF(store, smem)                                                                                  \
    do {                                                                                                       \
        FB_ALLOW_SMEM(potrf_kernel<store>, smem);                                                              \
        potrf_kernel<store><<<1, POTRF_THREADS, (smem), stream>>>(G, ldg, k, N, U, ldu, gwork, st, pass, gate, \
                                                                  forced_u, plan, frag, Rin, ldrin, Rout,      \
                                                                  ldrout);                                     \
    } while (0)
    if (k <= TR_KMAX) FB_POTRF(STORE_PLAN, (size_t)2 * TR_KMAX * TR_PREP_LD * sizeof(z64));
    else if (k <= POTRF_PACKED_MAX_K) FB_POTRF(STORE_PACKED, (size_t)k * (k + 1) / 2 * sizeof(z64));
    else FB_POTRF(STORE_GLOBAL, 0);
#undef FB_POTRF
    FB_LAUNCHED("potrf_kernel");
    return FB_OK;
}

int potrf_enqueue(const z64* G, int64_t ldg, int k, int64_t N, z64* U, int64_t ldu, z64* gwork,
                  ChainStatus* st, int pass, int gate, cudaStream_t stream, double forced_u, TrsmPlan* plan,
                  double* frag) {
    return potrf_launch(G, ldg, k, N, U, ldu, gwork, st, pass, gate, stream, forced_u, plan, frag, nullptr, 0, nullptr,
                        0);
}

}  // namespace fb

using namespace fb;

extern "C" {

int fb_zpotrf_workspace_size(int k, size_t* bytes) {
    if (!bytes || k < 0) { set_error(FB_EINVAL, "fb_zpotrf_workspace_size: bad argument"); return FB_EINVAL; }
    *bytes = align_up(sizeof(ChainStatus), 256) + align_up(potrf_gwork_bytes(k), 256);
    return FB_OK;
}

static int potrf_call(fb_z128* U, int64_t ldu, const fb_z128* G, int64_t ldg, int k, int64_t N,
                      const fb_z128* Rin, int64_t ldrin, fb_z128* Rout, int64_t ldrout,
                      int* shifted, double* shift, void* workspace, size_t workspace_bytes, fb_queue_t queue,
                      double forced_u) {
    if (k < 0 || N < 0) { set_error(FB_EINVAL, "fb_zpotrf_shifted: negative size"); return FB_EINVAL; }
    if (k == 0) {
        if (shifted) *shifted = 0;
        if (shift) *shift = 0.0;
        return FB_OK;
    }
    if (!U || !G || (Rin && !Rout)) { set_error(FB_EINVAL, "fb_zpotrf_shifted: NULL matrix"); return FB_EINVAL; }
    if (ldu < k || ldg < k || (Rin && ldrin < k) || (Rout && ldrout < k)) {
        set_error(FB_EDIM, "fb_zpotrf_shifted: leading dimension smaller than k=%d", k);
        return FB_EDIM;
    }
    if (Rin && Rout && Rin == Rout) {
        set_error(FB_EINVAL, "fb_zpotrf_shifted: Rout must not alias Rin");
        return FB_EINVAL;
    }
    size_t need = 0;
    fb_zpotrf_workspace_size(k, &need);
    if (!workspace || workspace_bytes < need) {
        set_error(FB_ENOMEM, "fb_zpotrf_shifted: workspace of %zu bytes, need %zu", workspace_bytes, need);
        return FB_ENOMEM;
    }
    cudaStream_t stream = stream_of(queue);
    ChainStatus* st = static_cast<ChainStatus*>(workspace);
    z64* gwork = reinterpret_cast<z64*>(static_cast<char*>(workspace) + align_up(sizeof(ChainStatus), 256));
    FB_CUDA(cudaMemsetAsync(st, 0, sizeof(ChainStatus), stream), "cudaMemsetAsync");
    z64* Uz = reinterpret_cast<z64*>(U);
    const z64* Ri = reinterpret_cast<const z64*>(Rin);
    z64* Ro = reinterpret_cast<z64*>(Rout);
    // The composition's blocks read U while others write R, so where the two
    // share memory the factor's own CTA forms the product.
    const bool shared = Ro && Uz < Ro + ((int64_t)(k - 1) * ldrout + k) && Ro < Uz + ((int64_t)(k - 1) * ldu + k);
    FB_TRY(potrf_launch(reinterpret_cast<const z64*>(G), ldg, k, N, Uz, ldu, gwork, st, 1, GATE_ALWAYS, stream, forced_u,
                        nullptr, nullptr, Ri, ldrin, shared ? Ro : nullptr, ldrout));
    if (Ro && !shared) FB_TRY(compose_r_enqueue(Ro, ldrout, k, Ri, ldrin, Uz, ldu, nullptr, 0, st, 0, stream));
    ChainStatus host{};
    FB_CUDA(cudaMemcpyAsync(&host, st, sizeof host, cudaMemcpyDeviceToHost, stream), "cudaMemcpyAsync");
    FB_CUDA(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
    if (shifted) *shifted = host.shifted[1];
    if (shift) *shift = host.shift[1];
    if (host.failed) {
        set_error(FB_ENOTSPD,
                  "the %dx%d Gram matrix is not positive definite even after a shift of %.17g, so the columns are "
                  "numerically dependent: a zero column, a duplicated one, or a condition number past 4.5e15. "
                  "Drop the dependent columns before orthonormalizing",
                  k, k, host.shift[1]);
        return FB_ENOTSPD;
    }
    return FB_OK;
}

int fb_zpotrf_shifted(fb_z128* U, int64_t ldu, const fb_z128* G, int64_t ldg, int k, int64_t N,
                      const fb_z128* Rin, int64_t ldrin, fb_z128* Rout, int64_t ldrout,
                      int* shifted, double* shift, void* workspace, size_t workspace_bytes, fb_queue_t queue) {
    return potrf_call(U, ldu, G, ldg, k, N, Rin, ldrin, Rout, ldrout, shifted, shift, workspace, workspace_bytes,
                      queue, 0.0);
}

int fb_zpotrf_forced_shift(fb_z128* U, int64_t ldu, const fb_z128* G, int64_t ldg, int k, int64_t N,
                           const fb_z128* Rin, int64_t ldrin, fb_z128* Rout, int64_t ldrout, double unit_roundoff,
                           double* shift, void* workspace, size_t workspace_bytes, fb_queue_t queue) {
    if (!(unit_roundoff > 0.0 && unit_roundoff < 1.0)) {
        set_error(FB_EINVAL, "fb_zpotrf_forced_shift: the unit roundoff must lie in (0, 1), got %g", unit_roundoff);
        return FB_EINVAL;
    }
    return potrf_call(U, ldu, G, ldg, k, N, Rin, ldrin, Rout, ldrout, nullptr, shift, workspace, workspace_bytes,
                      queue, unit_roundoff);
}

}  // extern "C"
