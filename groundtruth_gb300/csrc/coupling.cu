// The signal path's coupling to the strips (GroundTruth: PlaneStack.strip_coupling, peec.py:2615-2656, with
// kernel.segment_vector_potential, kernel.py:297-312): psi of every strip, the flux per ampere of signal current
// along it, in FP64 on the device.
//
// For a strip of orientation `axis` on sheet k (centre of its cell at the sheet face nearer the segment) and a
// horizontal signal segment a -> b with a component along the axis, the segment's vector potential
//     A(p) = mu0 / (4 pi) [asinh((L - p.u) / rho) + asinh(p.u / rho)],  rho = max(dist(p, line), r_min)
// is taken at the centre, or averaged over the cell with a 3 x 3 Gauss rule when the centre lies within
// 3 d + 2 w of the segment; psi = d * sum_segments current * (b - a)[axis] / L * A.
#include "kernels.h"

namespace gt {

namespace {

constexpr double MU0_4PI = 1e-7;     // mu0 / (4 pi)
constexpr int SEG_TILE = 128;

struct Seg {
    double a[3], b[3], width, cur;
    double u[3], L, iL2, rmin2, lim, zm;     // direction, length, 1 / L^2, r_min^2, the cell average's reach, mean height
};

// A(p) of a segment.  The two terms asinh(a / rho) + asinh(b / rho), a = L - p.u, b = p.u, are one asinh by its addition
// theorem: sinh of the sum is (a rb + b ra) / rho^2 with ra, rb the distances to the ends, and for ends on either side of
// the foot (a, b of opposite sign), where that would cancel, L (a - b) / (a rb - b ra).  Half the transcendental work of
// the sum of two: the kernel is bound by the FP64 pipe (two operations a clock and SM).
__device__ __forceinline__ double vec_pot(const Seg& s, double px, double py, double pz) {
    const double dx = px - s.a[0], dy = py - s.a[1], dz = pz - s.a[2];
    const double pu = dx * s.u[0] + dy * s.u[1] + dz * s.u[2];
    const double h2 = fmax(dx * dx + dy * dy + dz * dz - pu * pu, s.rmin2);
    const double a = s.L - pu;
    const double ra = sqrt(a * a + h2), rb = sqrt(pu * pu + h2);
    const bool within = a >= 0 && pu >= 0;
    const double num = within ? a * rb + pu * ra : s.L * (a - pu);
    const double den = within ? h2 : a * rb - pu * ra;
    return MU0_4PI * asinh(num / den);
}

__device__ __forceinline__ double dist_to_segment(const Seg& s, double px, double py, double pz) {
    const double ab[3] = {s.b[0] - s.a[0], s.b[1] - s.a[1], s.b[2] - s.a[2]};
    const double L2 = ab[0] * ab[0] + ab[1] * ab[1] + ab[2] * ab[2];
    double t = 0.0;
    if (L2 > 0) t = fmin(fmax(((px - s.a[0]) * ab[0] + (py - s.a[1]) * ab[1] + (pz - s.a[2]) * ab[2]) / L2, 0.0), 1.0);
    const double qx = px - (s.a[0] + t * ab[0]), qy = py - (s.a[1] + t * ab[1]), qz = pz - (s.a[2] + t * ab[2]);
    return sqrt(qx * qx + qy * qy + qz * qz);
}

__global__ void __launch_bounds__(256) strip_coupling_kernel(Geo g, const int64_t* __restrict__ c2d, int64_t ns,
                                                             SheetZ sheet_z, SheetZ sheet_t, double d,
                                                             const double* __restrict__ segs, int nseg,
                                                             double* __restrict__ psi) {
    __shared__ Seg sh[SEG_TILE];
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool act = c < ns;
    int axis = 0, k = 0;
    double cx = 0, cy = 0;
    if (act) {
        const int64_t pos = c2d[c];
        const int nx = g.nx, ny = g.ny;
        if (pos < g.off_y) {
            const int64_t q = pos - g.off_x, plane = (int64_t)(nx - 1) * ny;
            k = int(q / plane);
            const int64_t ij = q - k * plane;
            const int i = int(ij / ny), j = int(ij - (int64_t)i * ny);
            cx = i * d + 0.5 * d;
            cy = j * d;
        } else {
            axis = 1;
            const int64_t q = pos - g.off_y, plane = (int64_t)nx * (ny - 1);
            k = int(q / plane);
            const int64_t ij = q - k * plane;
            const int i = int(ij / (ny - 1)), j = int(ij - (int64_t)i * (ny - 1));
            cx = i * d;
            cy = j * d + 0.5 * d;
        }
    }
    const double zk = act ? sheet_z.z[k] : 0.0, half = act ? 0.5 * sheet_t.z[k] : 0.0;
    // the 3-point Gauss-Legendre rule on [-1/2, 1/2]
    const double gq[3] = {-0.5 * sqrt(0.6), 0.0, 0.5 * sqrt(0.6)};
    const double gw[3] = {5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0};
    double acc = 0.0;
    for (int t0 = 0; t0 < nseg; t0 += SEG_TILE) {
        const int nt = min(SEG_TILE, nseg - t0);
        __syncthreads();
        for (int q = threadIdx.x; q < nt; q += blockDim.x) {
            const double* r = segs + (int64_t)(t0 + q) * 8;
            Seg s{{r[0], r[1], r[2]}, {r[3], r[4], r[5]}, r[6], r[7]};
            const double ab[3] = {r[3] - r[0], r[4] - r[1], r[5] - r[2]};
            const double L2 = ab[0] * ab[0] + ab[1] * ab[1] + ab[2] * ab[2];
            s.L = sqrt(L2);
            for (int c = 0; c < 3; ++c) s.u[c] = ab[c] / s.L;
            s.iL2 = 1.0 / L2;
            const double rmin = fmax(0.5 * r[6], 1e-7);
            s.rmin2 = rmin * rmin;
            s.lim = 3 * d + 2 * r[6];
            s.zm = 0.5 * (r[2] + r[5]);
            sh[q] = s;
        }
        __syncthreads();
        if (!act) continue;
        for (int q = 0; q < nt; ++q) {
            const Seg& s = sh[q];
            const double ab[3] = {s.b[0] - s.a[0], s.b[1] - s.a[1], s.b[2] - s.a[2]};
            if (ab[0] == 0.0 && ab[1] == 0.0) continue;                  // vertical: not a horizontal segment
            if (fabs(ab[axis]) < 1e-15 * s.L) continue;
            const double cz = zk + (s.zm > zk ? half : -half);
            // near: the centre within lim of the segment; by the squared distance, and by the distance itself where the
            // two are too close for that
            const double dx = cx - s.a[0], dy = cy - s.a[1], dz = cz - s.a[2];
            const double tt = fmin(fmax((dx * ab[0] + dy * ab[1] + dz * ab[2]) * s.iL2, 0.0), 1.0);
            const double qx = dx - tt * ab[0], qy = dy - tt * ab[1], qz = dz - tt * ab[2];
            const double d2 = qx * qx + qy * qy + qz * qz, l2 = s.lim * s.lim;
            const bool near = fabs(d2 - l2) > 1e-9 * l2 ? d2 < l2 : dist_to_segment(s, cx, cy, cz) < s.lim;
            double a;
            if (near) {
                a = 0.0;
                for (int m = 0; m < 3; ++m)
                    for (int n = 0; n < 3; ++n) {
                        const double da = (axis == 0 ? gq[m] : gq[n]) * d, dl = (axis == 0 ? gq[n] : gq[m]) * d;
                        a += vec_pot(s, cx + da, cy + dl, cz) * (gw[m] * gw[n] / 4.0);
                    }
            } else {
                a = vec_pot(s, cx, cy, cz);
            }
            acc += (s.cur * s.u[axis]) * a;
        }
    }
    if (act) psi[c] = d * acc;
}

}  // namespace

void launch_strip_coupling(const Geo& g, const int64_t* c2d, int64_t ns, const SheetZ& sheet_z, const SheetZ& sheet_t,
                           double d, const double* segs, int nseg, double* psi, cudaStream_t st) {
    if (ns <= 0) return;
    strip_coupling_kernel<<<ceil_div(ns, 256), 256, 0, st>>>(g, c2d, ns, sheet_z, sheet_t, d, segs, nseg, psi);
    GT_LAUNCH_CHECK();
}

}  // namespace gt
