// The k x k steps of one cholqr2! pass, as device functions that one CTA of
// any size runs: ||G||_F, the Cholesky of the Gram matrix with the shifted
// retry of cholesky_upper (src/panelblas.jl:148-155), and the solve plan of
// the triangular solve (inv(R), the conditioning, the path and its B
// fragments). The chain's one-CTA kernels and the persistent batch kernel
// both call them, so a factor is computed the same way in either.
#pragma once

#include "fb_solve.cuh"

namespace fb {

// Fixed-order sum over the CTA: warp shuffle tree, then warp 0 over the
// warps. scratch: 33 doubles of shared memory.
__device__ inline double block_sum(double v, double* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    double total = 0.0;
    if (warp == 0) {
        double w = lane < nwarps ? scratch[lane] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) w += __shfl_down_sync(0xffffffffu, w, off);
        if (lane == 0) scratch[32] = w;
    }
    __syncthreads();
    total = scratch[32];
    return total;
}

// Cholesky of the Hermitian matrix g (upper triangle read) into the upper
// triangle of `at`, at(i, j) a reference to entry (i, j), i <= j. Pivot test as
// LAPACK's zpotrf makes it: the factorization fails as soon as a pivot is not
// > 0 (this also catches NaN). On failure the matrix is reloaded with
// s = 11 N k eps ||G||_F added to the diagonal and factored again; a second
// failure is reported, not shifted further. forced_u > 0 instead shifts once,
// unconditionally, by s = 11 (N k + k (k+1)) forced_u ||G||_F (the shifted
// CholeskyQR3). Returns whether a factor was found; gnorm is ||G||_F, shifted
// and shift say which matrix the factor is of. scratch: 33 doubles of shared
// memory.
//
// Right-looking by blocks of 8 columns. What bounds it is latency, so the
// dependent steps are kept inside one warp: warp 0 factors the 8 x 8 diagonal
// block alone (28 trailing entries on 28 lanes), then a thread per column solves the block row
// in registers, then the trailing triangle takes a rank-8 update, a 2 x 2 tile
// of it a thread: three block barriers a block of 8 columns instead of two a
// column. With the plan below, one launch: k = 16 24 -> 12 us, k = 64 121 ->
// 51 us; k = 128 (packed in shared memory instead of in global memory) 224 ->
// 106 us without a plan.
template <class LoadG, class At>
__device__ bool factor_shifted(LoadG g, int k, int64_t N, double forced_u, At at, double* scratch, double& gnorm,
                               bool& shifted, double& shift) {
    __shared__ double invd[8];
    __shared__ int failed;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
    shifted = false;
    shift = 0.0;
    // This lane's entry (m, l) of a diagonal block's trailing triangle.
    int em = 1, el = lane;
    while (em < 8 && el >= 8 - em) { el -= 8 - em; ++em; }
    el += em;
    bool ok = false;
    for (int attempt = 0; attempt < 2 && !ok; ++attempt) {
        __syncthreads();
        double part = 0.0;
        // Warps over the columns, lanes over 32 rows of one, four columns in
        // flight a warp.
        for (int i0 = 0; i0 < k; i0 += 32) {
            const int i = i0 + lane;
            for (int j0 = warp; j0 < k; j0 += 4 * nwarps) {
                z64 v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int j = j0 + q * nwarps;
                    v[q] = (j < k && i <= j) ? g(i, j) : zmake(0.0, 0.0);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int j = j0 + q * nwarps;
                    const double a2 = fma(v[q].x, v[q].x, v[q].y * v[q].y);
                    part += (i == j) ? a2 : 2.0 * a2;
                    if (j < k && i <= j) at(i, j) = i == j ? zmake(v[q].x + shift, 0.0) : v[q];
                }
            }
        }
        if (attempt == 0) {
            gnorm = sqrt(block_sum(part, scratch));
            if (forced_u > 0.0) {
                shifted = true;
                shift = 11.0 * ((double)N * (double)k + (double)k * (double)(k + 1)) * forced_u * gnorm;
                for (int j = tid; j < k; j += nt) at(j, j).x += shift;
            }
        }
        if (tid == 0) failed = 0;
        __syncthreads();
        for (int j0 = 0; j0 < k; j0 += 8) {
            const int nb = k - j0 < 8 ? k - j0 : 8;
            if (warp == 0) {
                // Rows stay unscaled until the end and the next pivot travels
                // by shuffle from the lane that holds it: a step's critical
                // path is one reciprocal square root.
                double mine = 1.0, mine_inv = 1.0;
                const bool live = el < nb;
                z64 w = live ? at(j0 + em, j0 + el) : zmake(0.0, 0.0);
                double d = at(j0, j0).x;
#pragma unroll 1
                for (int jj = 0; jj < nb; ++jj) {
                    const int j = j0 + jj;
                    if (!(d > 0.0)) {
                        if (lane == 0) failed = 1;
                        break;
                    }
                    const double inv = rsqrt(d);
                    if (lane == jj) {
                        mine = d;
                        mine_inv = inv;
                    }
                    if (em > jj && live) {
                        // w -= conj(a) * b, a and b the scaled row's entries
                        const z64 ra = at(j, j0 + em), rb = at(j, j0 + el);
                        const z64 a = zmake(ra.x * inv, ra.y * inv), b = zmake(rb.x * inv, rb.y * inv);
                        w.x = fma(-a.x, b.x, w.x);
                        w.x = fma(-a.y, b.y, w.x);
                        w.y = fma(-a.x, b.y, w.y);
                        w.y = fma(a.y, b.x, w.y);
                        at(j0 + em, j0 + el) = w;
                    }
                    d = __shfl_sync(0xffffffffu, w.x, jj < 7 ? jj * (15 - jj) / 2 : 0);   // entry (jj + 1, jj + 1)
                    __syncwarp();
                }
                if (lane < nb) {
                    invd[lane] = mine_inv;
                    for (int l = lane + 1; l < nb; ++l) {
                        const z64 v = at(j0 + lane, j0 + l);
                        at(j0 + lane, j0 + l) = zmake(v.x * mine_inv, v.y * mine_inv);
                    }
                    at(j0 + lane, j0 + lane) = zmake(sqrt(mine), 0.0);
                }
            }
            __syncthreads();
            if (failed) break;
            const int first = j0 + 8;
            if (first >= k) break;
            // The block row: x_r = (a_r - sum_{m<r} conj(u_mr) x_m) / u_rr.
            for (int c = first + tid; c < k; c += nt) {
                z64 x[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) x[r] = at(j0 + r, c);
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    x[r] = zmake(x[r].x * invd[r], x[r].y * invd[r]);
#pragma unroll
                    for (int m = r + 1; m < 8; ++m) {
                        const z64 u = at(j0 + r, j0 + m);
                        x[m].x = fma(-u.x, x[r].x, x[m].x);
                        x[m].x = fma(-u.y, x[r].y, x[m].x);
                        x[m].y = fma(-u.x, x[r].y, x[m].y);
                        x[m].y = fma(u.y, x[r].x, x[m].y);
                    }
                }
#pragma unroll
                for (int r = 0; r < 8; ++r) at(j0 + r, c) = x[r];
            }
            __syncthreads();
            // The trailing triangle: row pairs over the warps, column pairs
            // over the lanes.
            const int rest = k - first, pairs = (rest + 1) / 2;
            for (int a = warp; a < pairs; a += nwarps) {
                const int m0 = first + 2 * a;
                const bool m1ok = m0 + 1 < k;
                for (int b = a + lane; b < pairs; b += 32) {
                    const int l0 = first + 2 * b;
                    const bool l1ok = l0 + 1 < k;
                    z64 w[2][2];
                    w[0][0] = at(m0, l0);
                    w[0][1] = l1ok ? at(m0, l0 + 1) : zmake(0.0, 0.0);
                    w[1][0] = (m1ok && a < b) ? at(m0 + 1, l0) : zmake(0.0, 0.0);
                    w[1][1] = (m1ok && l1ok) ? at(m0 + 1, l0 + 1) : zmake(0.0, 0.0);
#pragma unroll 4
                    for (int r = 0; r < 8; ++r) {
                        z64 u[2], v[2];
                        u[0] = at(j0 + r, m0);
                        u[1] = m1ok ? at(j0 + r, m0 + 1) : zmake(0.0, 0.0);
                        v[0] = at(j0 + r, l0);
                        v[1] = l1ok ? at(j0 + r, l0 + 1) : zmake(0.0, 0.0);
#pragma unroll
                        for (int p = 0; p < 2; ++p)
#pragma unroll
                            for (int q = 0; q < 2; ++q) {
                                w[p][q].x = fma(-u[p].x, v[q].x, w[p][q].x);
                                w[p][q].x = fma(-u[p].y, v[q].y, w[p][q].x);
                                w[p][q].y = fma(-u[p].x, v[q].y, w[p][q].y);
                                w[p][q].y = fma(u[p].y, v[q].x, w[p][q].y);
                            }
                    }
                    at(m0, l0) = w[0][0];
                    if (l1ok) at(m0, l0 + 1) = w[0][1];
                    if (m1ok && a < b) at(m0 + 1, l0) = w[1][0];
                    if (m1ok && l1ok) at(m0 + 1, l0 + 1) = w[1][1];
                }
            }
            __syncthreads();
        }
        __syncthreads();
        ok = failed == 0;
        if (ok || forced_u > 0.0) break;
        if (attempt == 0) {
            shifted = true;
            shift = 11.0 * (double)N * (double)k * 2.220446049250313e-16 * gnorm;
        }
    }
    __syncthreads();
    return ok;
}

// Row stride of the prep's KP x KP matrices in shared memory (one complex
// of padding against bank conflicts).
constexpr int TR_PREP_LD = TR_KMAX + 1;

// |z|; the squares are safe in the middle of the range.
__device__ __forceinline__ double zabs(z64 z) {
    const double m = fmax(fabs(z.x), fabs(z.y));
    const double h = sqrt(fma(z.x, z.x, z.y * z.y));
    if (m == 0.0 || (m > 0x1p-500 && m < 0x1p500)) return h;
    return hypot(z.x, z.y);
}

// The solve plan of an upper triangular R, k <= 64: Rs holds R padded with
// the identity to KP x KP (KP = k rounded up to 8), row stride TR_PREP_LD;
// Xs is zeroed, same shape; both are complete (the caller synchronized).
// Computes inv(R) into Xs, the 1-norm condition numbers of R and of its 8 x 8
// diagonal blocks, the path, and the chosen path's B fragments into frag.
//
// inv(R): the 8 x 8 diagonal blocks by substitution, a thread per column in
// registers, all blocks at once; then block inverses of twice the size from
// pairs of them, [A B; 0 D]^-1 = [A^-1, -A^-1 B D^-1; 0, D^-1], three times:
// eight block barriers instead of one a row. The code is kept short (few loops
// unrolled): it runs once a launch, so fetching it is part of its time (k = 16:
// 23 -> 14 us for factor and plan). k = 64 alone: 62 -> 22 us.
__device__ inline void solve_plan(const z64* Rs, z64* Xs, int k, TrsmPlan* plan, double* __restrict__ frag) {
    constexpr int LD = TR_PREP_LD;
    __shared__ z64 dinv[TR_KMAX];
    __shared__ double colr[TR_KMAX], coli[TR_KMAX];
    __shared__ double bcolr[TR_KMAX], bcoli[TR_KMAX];
    __shared__ int path;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
    const int KP = (k + TR_NB - 1) / TR_NB * TR_NB;
    const int NBLK = KP / TR_NB;
    for (int e = tid; e < KP; e += nt) dinv[e] = zrecip_d(Rs[e * LD + e]);
    __syncthreads();
    for (int e = tid; e < KP; e += nt) {
        const int o = e & ~7, c = e & 7;
        z64 x[TR_NB];
#pragma unroll
        for (int i = TR_NB - 1; i >= 0; --i) {
            z64 s = zmake(i == c ? 1.0 : 0.0, 0.0);
#pragma unroll
            for (int l = TR_NB - 1; l > i; --l)
                if (l <= c) zmsub(s, Rs[(o + i) * LD + o + l], x[l]);
            x[i] = zmul(s, dinv[o + i]);
        }
#pragma unroll
        for (int i = 0; i < TR_NB; ++i)
            if (i <= c) Xs[(o + i) * LD + o + c] = x[i];
    }
    __syncthreads();
    for (int s = TR_NB, lg = 3; s < KP; s *= 2, ++lg) {
        // Pairs (a, b = a + s): entries (i, j) of the s x s block between
        // them, the last pair's block as wide as is left, a 2 x 2 tile of them
        // a thread (shared memory's reads bound this). B D^-1 goes,
        // transposed, to the block's mirror image below the diagonal, which
        // nothing else uses.
        const int tiles = ((KP + s - 1) / (2 * s)) << (2 * lg - 2);
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
#pragma unroll 1
            for (int e = tid; e < tiles; e += nt) {
                const int a = (e >> (2 * lg - 2)) * 2 * s, b = a + s;
                const int i = 2 * ((e >> (lg - 1)) & (s / 2 - 1)), j = 2 * (e & (s / 2 - 1));
                if (b + j >= KP) continue;
                // Row i of the left factor, column j of the right one.
                const z64* x = half ? Xs + (a + i) * LD + a : Rs + (a + i) * LD + b;
                const z64* y = half ? Xs + (b + j) * LD + a : Xs + b * LD + b + j;
                const int step = half ? 1 : LD, next = half ? LD : 1;
                const int l0 = half ? i : 0, l1 = half ? s : j + 2;
                z64 t[2][2];
#pragma unroll
                for (int q = 0; q < 4; ++q) t[q >> 1][q & 1] = zmake(0.0, 0.0);
#pragma unroll 2
                for (int l = l0; l < l1; ++l) {
                    const z64 x0 = x[l], x1 = x[LD + l], y0 = y[l * step], y1 = y[l * step + next];
                    // The triangles' own edges: inv(D) ends at l = j (j + 1
                    // for the second column), inv(A) starts at l = i.
                    if (half || l <= j) {
                        zmac(t[0][0], x0, y0);
                        if (!half || l > i) zmac(t[1][0], x1, y0);
                    }
                    zmac(t[0][1], x0, y1);
                    if (!half || l > i) zmac(t[1][1], x1, y1);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int ii = i + (q >> 1), jj = j + (q & 1);
                    const z64 v = t[q >> 1][q & 1];
                    if (half) Xs[(a + ii) * LD + b + jj] = zmake(-v.x, -v.y);
                    else Xs[(b + jj) * LD + a + ii] = v;
                }
            }
            __syncthreads();
        }
    }
    // 1-norms of R's own columns and of inv(R)'s, and of the columns of
    // their 8 x 8 diagonal blocks: a warp per column.
    for (int c = warp; c < KP; c += nwarps) {
        // R's and inv(R)'s entries of two rows a lane, their square roots
        // side by side.
        double h[2][2];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = lane + 32 * (q & 1);
            const z64 v = i <= c ? ((q >> 1) ? Xs : Rs)[i * LD + c] : zmake(0.0, 0.0);
            h[q >> 1][q & 1] = zabs(v);
        }
        double sums[4];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int first = TR_NB * (c / TR_NB);
            sums[q] = h[q][0] + h[q][1];
            sums[2 + q] = (lane >= first ? h[q][0] : 0.0) + (lane + 32 >= first ? h[q][1] : 0.0);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int q = 0; q < 4; ++q) sums[q] += __shfl_down_sync(0xffffffffu, sums[q], off);
        if (lane == 0) {
            colr[c] = c < k ? sums[0] : 0.0;
            coli[c] = c < k ? sums[1] : 0.0;
            bcolr[c] = sums[2];
            bcoli[c] = sums[3];
        }
    }
    __syncthreads();
    if (warp == 0) {
        double nr = 0.0, ni = 0.0, worst = 0.0;
        for (int c = lane; c < TR_KMAX; c += 32) {
            const bool in = c < KP;
            nr = fmax(nr, in ? colr[c] : 0.0);
            ni = fmax(ni, in ? coli[c] : 0.0);
            double br = in ? bcolr[c] : 0.0, bi = in ? bcoli[c] : 0.0;
#pragma unroll
            for (int off = 4; off > 0; off >>= 1) {   // the block's eight columns
                br = fmax(br, __shfl_xor_sync(0xffffffffu, br, off));
                bi = fmax(bi, __shfl_xor_sync(0xffffffffu, bi, off));
            }
            worst = fmax(worst, br * bi);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            nr = fmax(nr, __shfl_xor_sync(0xffffffffu, nr, off));
            ni = fmax(ni, __shfl_xor_sync(0xffffffffu, ni, off));
            worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, off));
        }
        if (lane == 0) {
            const double cond = nr * ni;
            int p = PATH_SUBSTITUTE;
            if (cond <= TR_INV_COND_LIMIT) p = PATH_INVERSE;
            else if (worst <= TR_COND_LIMIT) p = PATH_BLOCKED;
            path = p;
            plan->path = p;
            plan->cond = cond;
            plan->cond_blocks = worst;
        }
    }
    __syncthreads();
    // The fragments: a warp per n-tile of inv(R), or per 16 x 16 pair.
    if (path == PATH_INVERSE) {
        const int p = lane & 1, o = (lane >> 2) & 1;
        for (int t = warp; t < (k + 3) / 4; t += nwarps)
#pragma unroll 4
            for (int s = 0; s < 2 * t + 2; ++s) {
                const int i = 2 * s + ((lane & 3) >> 1), j = 4 * t + ((lane >> 2) >> 1);
                frag[(t * (t + 1) + s) * 32 + lane] = (i <= j) ? real_form(Xs[i * LD + j], p, o) : 0.0;
            }
    } else if (path == PATH_BLOCKED) {
        for (int pr = warp; pr < NBLK * (NBLK + 1) / 2; pr += nwarps) {
            int b = 0;
            while (pair_index(0, b + 1) <= pr) ++b;
            const int c = pr - pair_index(0, b);
            // -R_cb off the diagonal; inv(R_bb), which is inv(R)'s own diagonal block, on it.
            const z64* M = c < b ? Rs : Xs;
            const double sign = c < b ? -1.0 : 1.0;
#pragma unroll 4
            for (int st_ = 0; st_ < TR_FRAG / 32; ++st_) {
                const int s = st_ >> 1, t = st_ & 1;
                const int kr = 4 * s + (lane & 3), nr = 8 * t + (lane >> 2);
                const int i = TR_NB * c + (kr >> 1), p = kr & 1, j = TR_NB * b + (nr >> 1), o = nr & 1;
                const z64 m = (c == b && i > j) ? zmake(0.0, 0.0) : M[i * LD + j];
                frag[(pr * (TR_FRAG / 32) + st_) * 32 + lane] = sign * real_form(m, p, o);
            }
        }
    }
}

}  // namespace fb
