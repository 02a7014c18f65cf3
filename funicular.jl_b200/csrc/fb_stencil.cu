// The matrix-free operator of the streamed range finder (a complex-shifted
// 3-D Laplacian on a 342^3 grid): G = -Lap_7 + shift I on an nx x ny x nz grid, applied to the columns of a
// device panel, the panel-capable mul! that apply_operator! hands a whole
// resident panel to (src/operator.jl:80-87). Grid point (x, y, z) is row
// x + nx (y + ny z); the 7-point Laplacian has unit spacing and zero
// (Dirichlet) values outside the grid:
//   (G v)_p = (6 + shift) v_p - sum of the six neighbours of p.
// HBM-bound: 32 bytes per entry (read once, write once) when the neighbours
// are read from DRAM once. Two kernels: by 2.5-D tiles (the default), and a
// thread per output entry for column counts past the grid limit.
#include "fb_common.cuh"
#include "fb_tma.cuh"

namespace fb {

// Blocks walk grid lines (fixed y, z) and threads the points of a line, so
// the index arithmetic is one 32-bit division per line.
__global__ void __launch_bounds__(128) laplace7_kernel(z64* __restrict__ Y, int64_t ldy, const z64* __restrict__ X,
                                                       int64_t ldx, int nx, int ny, int nz, int cols, z64 shift) {
    const int64_t plane = (int64_t)nx * ny;
    const int lines = ny * nz;
    const double dr = 6.0 + shift.x, di = shift.y;
    for (int c = blockIdx.y; c < cols; c += gridDim.y) {
        const z64* x = X + (int64_t)c * ldx;
        z64* y = Y + (int64_t)c * ldy;
        for (int line = blockIdx.x; line < lines; line += gridDim.x) {
            const int zi = line / ny, yi = line - zi * ny;
            const int64_t base = (int64_t)line * nx;
            for (int xi = threadIdx.x; xi < nx; xi += blockDim.x) {
                const int64_t p = base + xi;
                const z64 v = x[p];
                z64 s = zmake(0.0, 0.0);
                if (xi > 0) { const z64 u = x[p - 1]; s.x += u.x; s.y += u.y; }
                if (xi < nx - 1) { const z64 u = x[p + 1]; s.x += u.x; s.y += u.y; }
                if (yi > 0) { const z64 u = x[p - nx]; s.x += u.x; s.y += u.y; }
                if (yi < ny - 1) { const z64 u = x[p + nx]; s.x += u.x; s.y += u.y; }
                if (zi > 0) { const z64 u = x[p - plane]; s.x += u.x; s.y += u.y; }
                if (zi < nz - 1) { const z64 u = x[p + plane]; s.x += u.x; s.y += u.y; }
                y[p] = zmake(dr * v.x - di * v.y - s.x, dr * v.y + di * v.x - s.y);
            }
        }
    }
}

// The same operator by 2.5-D tiles: a block owns a 32 x 16 tile of an x-y
// plane of one column and marches it along a range of z. A producer warp keeps
// a ring of planes in flight with TMA, each the tile with a one-point halo (a
// 4-D box at (x0 - 1, y0 - 1, z, column); points outside the grid read as zero,
// which is the boundary condition); a thread takes its four neighbours in the
// plane from there and its own point of the planes below and above from
// registers. Every input is read from DRAM about once: the halos come from L2,
// where the neighbouring tiles marching beside this one have brought them.
// HBM-bound, so what counts is bytes in flight: the ring holds 78 KB a block
// and two blocks run on an SM, against one 16-byte load a thread and two block
// barriers a plane when each thread loaded its own points. 64 columns on the
// 215^3 grid: 3.86 ms, 5280 GB/s (5.31 ms, 3830 before); 3 columns on 342^3:
// 0.66 ms, 5780 GB/s. Three blocks with six slots (0.74 ms, 32 registers a
// thread) and 8-row tiles (0.70 ms, more halo) were slower. The z range of a
// column is cut into zchunks pieces, enough for the grid to fill the GPU when
// there are few columns.
constexpr int LT_X = 32, LT_Y = 16, LT_SLOTS = 8;
constexpr int LT_ROW = LT_X + 2;
constexpr int LT_PLANE = (LT_ROW * (LT_Y + 2) * 16 + 127) / 128 * 128;   // bytes of a ring slot
constexpr int LT_BOX_BYTES = LT_ROW * (LT_Y + 2) * 16;
constexpr int LT_WARPS = LT_X * LT_Y / 32;
constexpr size_t LT_SMEM = (size_t)LT_SLOTS * LT_PLANE + 2 * LT_SLOTS * sizeof(uint64_t) + 128;

__global__ void __launch_bounds__(LT_X * LT_Y + 32, 2)
laplace7_tiled_kernel(const __grid_constant__ CUtensorMap tm, z64* __restrict__ Y, int64_t ldy, int nx, int ny, int nz,
                      z64 shift, int zchunks, int zero) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)LT_SLOTS * LT_PLANE);
    uint64_t* empty = full + LT_SLOTS;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), tx = threadIdx.x & 31;
    const int c = blockIdx.z / zchunks, zc = blockIdx.z - c * zchunks;
    const int z0 = (int)((int64_t)nz * zc / zchunks), z1 = (int)((int64_t)nz * (zc + 1) / zchunks);
    if (threadIdx.x == 0) {
        for (int b = 0; b < LT_SLOTS; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&empty[b], LT_WARPS);
        }
        mbar_fence_init();
    }
    __syncthreads();
    // Planes z0 - 1 .. z1, plane z0 - 1 + i in slot i % LT_SLOTS.
    const int planes = z1 - z0 + 2;
    if (warp == LT_WARPS) {
        if (tx == 0) {
            tma_prefetch_map(&tm);
            int b = 0, issued = 0;
            uint32_t ph = 0;
            for (int i = 0; i < planes; ++i) {
                if (i >= LT_SLOTS && !mbar_wait(&empty[b], ph ^ 1u)) break;
                mbar_arrive_expect_tx(&full[b], LT_BOX_BYTES);
                tma_load_4d(smem + (size_t)b * LT_PLANE, &tm, 2 * ((int)blockIdx.x * LT_X - 1),
                            (int)blockIdx.y * LT_Y - 1, z0 - 1 + i, c, &full[b]);
                if (++b == LT_SLOTS) { b = 0; ph ^= 1u; }
                issued = i + 1;
            }
            // The block's shared memory must not go away under a copy that
            // the other warps gave up on.
            for (int i = issued > LT_SLOTS ? issued - LT_SLOTS : 0; i < issued; ++i)
                mbar_wait(&full[i % LT_SLOTS], (i / LT_SLOTS) & 1);
        }
        return;
    }
    const int gx = blockIdx.x * LT_X + tx, gy = blockIdx.y * LT_Y + warp;
    const bool inside = gx < nx && gy < ny;
    const int64_t plane = (int64_t)nx * ny;
    z64* y = Y + (int64_t)c * ldy + (int64_t)z0 * plane + (int64_t)gy * nx + gx;
    const double dr = 6.0 + shift.x, di = shift.y;
    const unsigned char* mine = smem + (((warp + 1) * LT_ROW + tx + 1) << 4);
    auto point = [&](int b, int off) { return *reinterpret_cast<const z64*>(mine + b * LT_PLANE + (off << 4)); };
    z64 below, cur;
    bool ok = mbar_wait_warp(&full[0], 0) && mbar_wait_warp(&full[1], 0);
    below = point(0, 0);
    cur = point(1, 0);
    uint32_t seen = 0;
    mark_loaded(seen, below.x);
    mark_loaded(seen, cur.x);
    __syncwarp();
    if (tx == 0) mbar_arrive(&empty[seen & zero]);
    int b = 1, nb = 2;
    uint32_t ph = 0;
    for (int z = z0; z < z1; ++z) {
        ok = ok && mbar_wait_warp(&full[nb], ph);
        const z64 above = point(nb, 0);
        const z64 l = point(b, -1), r = point(b, 1), d = point(b, -LT_ROW), u = point(b, LT_ROW);
        double sx = l.x + r.x + d.x + u.x + below.x + above.x;
        double sy = l.y + r.y + d.y + u.y + below.y + above.y;
        mark_loaded(seen, l.x);
        mark_loaded(seen, r.x);
        mark_loaded(seen, d.x);
        mark_loaded(seen, u.x);
        mark_loaded(seen, above.x);
        __syncwarp();
        if (tx == 0) mbar_arrive(&empty[b + (seen & zero)]);
        if (!ok) sx = __longlong_as_double(0x7ff8000000000000ll);   // a plane never came: no silent wrong answer
        if (inside) *y = zmake(dr * cur.x - di * cur.y - sx, dr * cur.y + di * cur.x - sy);
        y += plane;
        below = cur;
        cur = above;
        b = nb;
        if (++nb == LT_SLOTS) { nb = 0; ph ^= 1u; }
    }
}

}  // namespace fb

using namespace fb;

extern "C" {

int fb_zlaplace7_apply(fb_z128* Y, int64_t ldy, const fb_z128* X, int64_t ldx, int nx, int ny, int nz, int cols,
                       fb_z128 shift, fb_queue_t queue) {
    if (nx < 1 || ny < 1 || nz < 1 || cols < 0) {
        set_error(FB_EINVAL, "fb_zlaplace7_apply: the grid needs positive sizes and cols >= 0, got %d x %d x %d, "
                  "%d columns", nx, ny, nz, cols);
        return FB_EINVAL;
    }
    const int64_t n = (int64_t)nx * ny * nz;
    if (cols == 0) return FB_OK;
    if (!Y || !X) { set_error(FB_EINVAL, "fb_zlaplace7_apply: NULL matrix"); return FB_EINVAL; }
    if (ldy < n || ldx < n) {
        set_error(FB_EDIM, "fb_zlaplace7_apply: leading dimensions %lld, %lld below the %lld grid points",
                  (long long)ldy, (long long)ldx, (long long)n);
        return FB_EDIM;
    }
    if (((uintptr_t)Y | (uintptr_t)X) & 15) { set_error(FB_EINVAL, "fb_zlaplace7_apply: pointers must be 16-byte aligned"); return FB_EINVAL; }
    // Y and X must not overlap: every output reads seven inputs.
    const char* y0 = reinterpret_cast<const char*>(Y);
    const char* x0 = reinterpret_cast<const char*>(X);
    const size_t ybytes = ((size_t)(cols - 1) * ldy + n) * 16, xbytes = ((size_t)(cols - 1) * ldx + n) * 16;
    if (y0 < x0 + xbytes && x0 < y0 + ybytes) {
        set_error(FB_EINVAL, "fb_zlaplace7_apply: the output overlaps the input");
        return FB_EINVAL;
    }
    if ((int64_t)ny * nz > INT32_MAX) { set_error(FB_ENOTSUP, "fb_zlaplace7_apply: ny * nz must fit in 32 bits"); return FB_ENOTSUP; }
    const int64_t tiles = (int64_t)((nx + LT_X - 1) / LT_X) * ((ny + LT_Y - 1) / LT_Y);
    // z pieces: enough blocks for three rounds of two a SM, each piece at
    // least 16 planes (a piece reads two planes more than it writes).
    int64_t zchunks = ((int64_t)sm_count() * 6 + tiles * cols - 1) / (tiles * cols);
    if (zchunks > nz / 16) zchunks = nz / 16;
    if (zchunks < 1) zchunks = 1;
    if (cols * zchunks <= 65535 && (ny + LT_Y - 1) / LT_Y <= 65535 && nx < (1 << 30)) {
        CUtensorMap tm;
        FB_TRY(encode_grid_map(&tm, X, nx, ny, nz, cols, ldx, LT_ROW, LT_Y + 2));
        FB_ALLOW_SMEM(laplace7_tiled_kernel, LT_SMEM);
        const dim3 grid((unsigned)((nx + LT_X - 1) / LT_X), (unsigned)((ny + LT_Y - 1) / LT_Y),
                        (unsigned)(cols * zchunks));
        laplace7_tiled_kernel<<<grid, LT_X * LT_Y + 32, LT_SMEM, stream_of(queue)>>>(
            tm, reinterpret_cast<z64*>(Y), ldy, nx, ny, nz, zmake(shift.re, shift.im), (int)zchunks, 0);
        FB_LAUNCHED("laplace7_tiled_kernel");
        return FB_OK;
    }
    // Sixteen blocks per SM, every block walking the columns in the same order
    // and the lines of a column in a grid-strided sweep: the lines in flight
    // at one time span a few planes of one column, so the z neighbours of a
    // line are still in L2 when it is computed.
    const int64_t gy = 1;
    int64_t gx = (int64_t)sm_count() * 16;
    if (gx > (int64_t)ny * nz) gx = (int64_t)ny * nz;
    if (gx < 1) gx = 1;
    laplace7_kernel<<<dim3((unsigned)gx, (unsigned)gy), 128, 0, stream_of(queue)>>>(
        reinterpret_cast<z64*>(Y), ldy, reinterpret_cast<const z64*>(X), ldx, nx, ny, nz, cols,
        zmake(shift.re, shift.im));
    FB_LAUNCHED("laplace7_kernel");
    return FB_OK;
}

}  // extern "C"
