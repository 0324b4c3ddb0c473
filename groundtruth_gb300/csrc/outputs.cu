// Post-solve outputs on the device, from dense FP64 solutions (GroundTruth: Solution.node_field,
// peec.py:1151-1203, copper=False; PlaneStack.moment, peec.py:2668-2700, the plane's part).
#include "kernels.h"

namespace gt {

// Rows of the grid one block walks: a thread keeps its column j and carries the x strip below from row to row, so that
// every strip is read once, and a row's index arithmetic is the row's, not each node's.
constexpr int OUT_ROWS = 8;

// (Kx, Ky) at every node of every sheet: each node averages the strips of each direction that touch it and
// carry current, per cell width d.  kx / ky: [col][S][nx][ny].  Bound by its bytes: the two factors 1 / count / d are made
// once (an FP64 division takes some tens of instructions of a pipe that retires two a clock).
__global__ void __launch_bounds__(256) node_field_kernel(Geo g, const c64* __restrict__ x, int64_t ld, double d,
                                                         c64* __restrict__ kx, c64* __restrict__ ky) {
    const int S = g.S, nx = g.nx, ny = g.ny;
    const int k = blockIdx.y, col = blockIdx.z;
    const c64* X = x + (int64_t)col * ld + g.off_x + (int64_t)k * (nx - 1) * ny;
    const c64* Y = x + (int64_t)col * ld + g.off_y + (int64_t)k * nx * (ny - 1);
    c64* ox = kx + ((int64_t)col * S + k) * nx * ny;
    c64* oy = ky + ((int64_t)col * S + k) * nx * ny;
    const double w1 = 1.0 / 1.0 / d, w2 = 1.0 / 2.0 / d;
    const int i0 = blockIdx.x * OUT_ROWS, i1 = min(nx, i0 + OUT_ROWS);
    auto on = [](c64 v) { return v.re != 0 || v.im != 0; };
    for (int j = threadIdx.x; j < ny; j += blockDim.x) {
        c64 below = i0 > 0 ? X[(int64_t)(i0 - 1) * ny + j] : zero<double>();
#pragma unroll 4
        for (int i = i0; i < i1; ++i) {
            const c64 above = i < nx - 1 ? X[(int64_t)i * ny + j] : zero<double>();
            const c64 left = j > 0 ? Y[(int64_t)i * (ny - 1) + j - 1] : zero<double>();
            const c64 right = j < ny - 1 ? Y[(int64_t)i * (ny - 1) + j] : zero<double>();
            ox[(int64_t)i * ny + j] = (on(below) && on(above) ? w2 : w1) * (below + above);
            oy[(int64_t)i * ny + j] = (on(left) && on(right) ? w2 : w1) * (left + right);
            below = above;
        }
    }
}

void launch_node_field(const Geo& g, const c64* x, int64_t ld, int ncol, double d, c64* kx, c64* ky, cudaStream_t st) {
    const int threads = g.ny >= 256 ? 256 : std::max(32, (g.ny + 31) / 32 * 32);
    node_field_kernel<<<dim3(ceil_div(g.nx, OUT_ROWS), g.S, ncol), threads, 0, st>>>(g, x, ld, d, kx, ky);
    GT_LAUNCH_CHECK();
}

// m = 1/2 sum r x I dl over the plane's strips, capacitances and branches, per column (the signal segments'
// own part is the caller's), in two steps: partial sums of MOM_ROWS grid rows per block, [col][block][3], then one block
// per column adds them in order.  Row weights multiply a row's sum: two or four FP64 instructions an entry, which at the
// pipe's rate is about the time of the bytes.  (One block per column for everything took 1.1 ms for 32 columns of the
// 256 x 256 pair, 10 MB each.)
constexpr int MOM_ROWS = 16;
static __host__ __device__ int mom_blocks(const Geo& g) {
    const int rows = g.S * (g.nx - 1) + g.S * g.nx + g.np * g.nx;
    return (rows + MOM_ROWS - 1) / MOM_ROWS + 1;          // and one for the branches
}
int moment_blocks(const Geo& g) { return mom_blocks(g); }

__device__ __forceinline__ void block_sum3(const c64 (&v)[3], c64* out) {
    __shared__ c64 red[3][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = 0; c < 3; ++c) {
        double re = v[c].re, im = v[c].im;
        for (int o = 16; o > 0; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (lane == 0) red[c][warp] = mk<double>(re, im);
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        c64 s = zero<double>();
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
        out[threadIdx.x] = s;
    }
}

__global__ void __launch_bounds__(256) moment_rows_kernel(Geo g, const c64* __restrict__ x, int64_t ld, SheetZ zs, double d,
                                                          c64* __restrict__ part) {
    const int S = g.S, nx = g.nx, ny = g.ny, col = blockIdx.y;
    const int nX = S * (nx - 1), nY = S * nx, rows = nX + nY + g.np * nx;
    const c64* xc = x + (int64_t)col * ld;
    c64 a[3] = {zero<double>(), zero<double>(), zero<double>()};
    if (blockIdx.x == gridDim.x - 1) {                     // branches a -> b: r_a x r_b
        const int64_t nxy = (int64_t)nx * ny;
        for (int b = threadIdx.x; b < g.nbr; b += blockDim.x) {
            const int na = g.branch_nodes[2 * b], nb = g.branch_nodes[2 * b + 1];
            const double ax = (double)((na % nxy) / ny) * d, ay = (double)((na % nxy) % ny) * d, az = zs.z[na / nxy];
            const double bx = (double)((nb % nxy) / ny) * d, by = (double)((nb % nxy) % ny) * d, bz = zs.z[nb / nxy];
            const c64 I = xc[g.off_b + b];
            a[0] += (ay * bz - az * by) * I;
            a[1] += (az * bx - ax * bz) * I;
            a[2] += (ax * by - ay * bx) * I;
        }
    } else {
        const int r0 = blockIdx.x * MOM_ROWS, r1 = min(rows, r0 + MOM_ROWS);
        for (int j = threadIdx.x; j < ny; j += blockDim.x) {
            // this thread's entries of the rows, in runs of rows that share sheet and kind: sum and row-weighted sum
            for (int r = r0; r < r1;) {
                const bool isx = r < nX, isy = !isx && r < nX + nY;
                const int per = isx ? nx - 1 : nx, q = isx ? r : isy ? r - nX : r - nX - nY;
                const int k = q / per, i0 = q - k * per, n = min(r1 - r, per - i0), len = isy ? ny - 1 : ny;
                const c64* row = xc + (isx ? g.off_x : isy ? g.off_y : g.off_c) + (int64_t)q * len + j;
                r += n;
                if (j >= len) continue;
                c64 s = zero<double>(), t = zero<double>();
                if (isx) {
#pragma unroll 8
                    for (int e = 0; e < n; ++e) s += row[(int64_t)e * len];
                } else {
#pragma unroll 8
                    for (int e = 0; e < n; ++e) {
                        const c64 v = row[(int64_t)e * len];
                        s += v;
                        t.re = fma((double)(i0 + e), v.re, t.re);
                        t.im = fma((double)(i0 + e), v.im, t.im);
                    }
                }
                if (isx) {                                 // x strips (k, i, j): r = (., j d, z_k)
                    a[1] += (zs.z[k] * d) * s;
                    a[2] += (-(double)j * d * d) * s;
                } else if (isy) {                          // y strips (k, i, j): r = (i d, ., z_k)
                    a[0] += (-zs.z[k] * d) * s;
                    a[2] += (d * d) * t;
                } else {                                   // capacitances, upper -> lower
                    const double dz = zs.z[g.pair_layers[2 * k + 1]] - zs.z[g.pair_layers[2 * k]];
                    a[0] += ((double)j * d * dz) * s;
                    a[1] += (-d * dz) * t;
                }
            }
        }
    }
    block_sum3(a, part + ((int64_t)col * gridDim.x + blockIdx.x) * 3);
}

__global__ void __launch_bounds__(128) moment_sum_kernel(const c64* __restrict__ part, int nblk, c64* __restrict__ m) {
    const int col = blockIdx.x;
    c64 a[3] = {zero<double>(), zero<double>(), zero<double>()};
    for (int b = threadIdx.x; b < nblk; b += blockDim.x)
        for (int c = 0; c < 3; ++c) a[c] += part[((int64_t)col * nblk + b) * 3 + c];
    __shared__ c64 out[3];
    block_sum3(a, out);
    if (threadIdx.x < 3) m[(int64_t)col * 3 + threadIdx.x] = 0.5 * out[threadIdx.x];
}

// part: [ncol][moment_blocks][3] scratch
void launch_moment(const Geo& g, const c64* x, int64_t ld, int ncol, const SheetZ& zs, double d, c64* part, c64* m,
                   cudaStream_t st) {
    const int nb = mom_blocks(g);
    constexpr int MOST = 65535;                            // of a grid's second dimension
    for (int c = 0; c < ncol; c += MOST) {
        moment_rows_kernel<<<dim3(nb, std::min(MOST, ncol - c)), 256, 0, st>>>(g, x + c * ld, ld, zs, d, part + (int64_t)c * nb * 3);
        GT_LAUNCH_CHECK();
    }
    moment_sum_kernel<<<ncol, 128, 0, st>>>(part, nb, m);
    GT_LAUNCH_CHECK();
}

}  // namespace gt
