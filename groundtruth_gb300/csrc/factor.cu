// The Schur complement S = Ar^T D^-1 Ar of the preconditioner (peec.py:2379), its factorisation and its
// solves, on the device.  The reference factorises S with SuperLU (peec.py:2423, MMD ordering) and applies
// it with SuperLU's triangular solves every iteration (peec.py:3071, on the CPU also in gpu.py:566-573);
// here S (complex symmetric) is factorised as L D L^T by the multifrontal method along a nested-dissection
// elimination tree, one batched launch per tree level for all fronts of the level and all frequencies:
//
//   assemble   S values = sum of coef * admittance table entries (a fixed sparse map, per frequency)
//   front      F = own columns of S + children's update matrices (extend-add)
//   eliminate  the own columns of F; L and D go to the front's panel (nf x nown, column-major, D on its diagonal),
//              the trailing block is the front's update matrix
//
// FP64 throughout (a floating plane coupled only by plane-pair capacitance makes S nearly singular in one
// mode whose pivot is ~1e-10 of the strips' admittance); the panels are also rounded to FP32 for the
// inner iterations' solves.  The solves run level by level: leaves up for L z = s (each front gathers its
// children's update vectors, eliminates its own rows and passes its boundary rows up), z /= D, root down
// for L^T y = z (each front reads its ancestors' finished y).
#include "kernels.h"
#include "pivot.h"

namespace gt {

// Complex multiply-accumulate as four explicit FMAs (acc += a u): written out, the
// product and the sum round as separate operations (six instructions instead of four on the FP64 pipe).
__device__ __forceinline__ void cfma(c64& acc, c64 a, c64 u) {
    acc.re = __fma_rn(a.re, u.re, acc.re);
    acc.re = __fma_rn(-a.im, u.im, acc.re);
    acc.im = __fma_rn(a.re, u.im, acc.im);
    acc.im = __fma_rn(a.im, u.re, acc.im);
}
__global__ void assemble_s_kernel(const int64_t* __restrict__ ptr, const int* __restrict__ tab_idx,
                                  const double* __restrict__ coef, int64_t nsv, const c64* __restrict__ table, int ntab,
                                  c64* __restrict__ svals) {
    pdl_enter();
    const int op = blockIdx.y;
    const c64* T = table + (int64_t)op * ntab;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nsv; e += (int64_t)gridDim.x * blockDim.x) {
        c64 acc = zero<double>();
        for (int64_t q = ptr[e]; q < ptr[e + 1]; ++q) acc += coef[q] * T[tab_idx[q]];
        svals[(int64_t)op * nsv + e] = acc;
    }
}

void launch_assemble_s(const int64_t* ptr, const int* tab_idx, const double* coef, int64_t nsv, const c64* table,
                       int ntab, c64* svals, int nops, cudaStream_t st) {
    int blocks = (int)std::min<int64_t>((nsv + 255) / 256, 2048);
    pdl_launch(assemble_s_kernel, dim3(std::max(blocks, 1), nops), 256, 0, st, ptr, tab_idx, coef, nsv, table, ntab, svals);
    GT_LAUNCH_CHECK();
}

// Front entry (r, c), r >= c: own columns in the panel, the trailing block in the update matrix.
struct FrontView {
    c64* panel;
    c64* upd;
    int nf, nown, nbnd;
    __device__ __forceinline__ c64& at(int r, int c) const {
        return c < nown ? panel[(int64_t)c * nf + r] : upd[(int64_t)(c - nown) * nbnd + (r - nown)];
    }
};

__device__ __forceinline__ c64 pivot_inverse(c64 d, int* status) {
    if (!pivot_recip(d.re, d.im)) atomicOr(status, 1);
    return d;
}

__device__ __forceinline__ FrontView front_view(const Fronts& F, int f, int op, c64* panel, c64* upd) {
    const int nown = (int)F.nown[f], nbnd = (int)F.nbnd[f];
    return FrontView{panel + (int64_t)op * F.panel_total + F.panel_off[f], upd + (int64_t)op * F.upd_total + F.upd_off[f],
                     nown + nbnd, nown, nbnd};
}

// tile t of the lower triangle of a T x T tile grid: (bi, bj), bj <= bi
__device__ __forceinline__ void lower_tile(int t, int& bi, int& bj) {
    int b = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
    while ((int64_t)b * (b + 1) / 2 > t) --b;
    while ((int64_t)(b + 1) * (b + 2) / 2 <= t) ++b;
    bi = b;
    bj = t - b * (b + 1) / 2;
}

// The sweeps' copies of a front's finished panel P = [Linv_own; -L_bnd Linv_own] (unit diagonal, zeros above it):
// element (i, k) into its FP32 forward tile (rows gH .., inner k < min(nown, (g + 1) H)) and backward tile (columns
// tC .., inner i >= tC), see sweep.cu.
struct SweepTiles {
    int nf, nown, H, C;
    c32 *tf, *tb;
    __device__ SweepTiles(const SweepPlan& S, int f, int op, int nf_, int nown_, c32* pf, c32* pb)
        : nf(nf_), nown(nown_), H(S.hf[f]), C(S.hb[f]), tf(pf + (int64_t)op * S.ptotal + S.offf[f]),
          tb(pb + (int64_t)op * S.ptotal + S.offb[f]) {}
    __device__ __forceinline__ void fwd(int i, int k, c32 v) const {
        const int g = i / H;
        if (k >= min(nown, (g + 1) * H)) return;
        const int m = min(g, nown / H), h = min(H, nf - g * H);
        tf[(int64_t)H * H * m * (m + 1) / 2 + (int64_t)H * nown * (g - m) + (int64_t)k * ((h + 1) & ~1) + (i - g * H)] = v;
    }
    __device__ __forceinline__ void bwd(int i, int k, c32 v) const {
        const int t = k / C;
        if (i < t * C) return;
        const int h = min(C, nown - t * C);
        tb[(int64_t)C * ((int64_t)t * nf - (int64_t)C * t * (t - 1) / 2) + (int64_t)(i - t * C) * ((h + 1) & ~1) + (k - t * C)] = v;
    }
};

// Small fronts: one CTA per (front, operator) with the front's own columns in shared memory from assembly to the finished
// solve panel.  An SM of GB300 retires two FP64 FMAs a clock, a warp's instruction holding its quarter of the pipe for 64
// cycles however few lanes it has, so the work is laid out flat over the threads (the elimination column by column as dot
// products over row x segment, the update matrix and the inverse entry by entry), with no complex product in the inner
// loops but the FMAs themselves:
//   assemble   own columns of S plus the children's entries; what falls into the update matrix goes to global memory
//   column k   a(i,k) - sum_{m<k} l(i,m) w(k,m), w = l d held unscaled in the upper triangle; l = that / d_k
//   update     U(i,j) -= sum_k l(i,k) w(j,k)
//   inverse    X = L_own^-1 row by row in place, M = -L_bnd X
// and the sweeps' copies are written straight from shared memory.  Rank-1 updates in global memory and three passes for the
// inversion and the copies took 41 of the 127 ms of four factorisations of the 256 x 256 pair.
constexpr int SF_THREADS = 256;
constexpr size_t SF_SMEM_MAX = 224 * 1024;

size_t small_front_smem(int nown, int nbnd) {
    const size_t ldp = (size_t)(nown + nbnd) | 1, ldb = (size_t)nbnd | 1;
    return ((size_t)nown * (ldp + ldb + 1) + SF_THREADS) * sizeof(c64);
}
bool small_front_fits(int nown, int nbnd) { return small_front_smem(nown, nbnd) <= SF_SMEM_MAX; }

__global__ void __launch_bounds__(SF_THREADS) small_front_kernel(Fronts F, SweepPlan S, const int64_t* __restrict__ front_list,
                                                                 const c64* __restrict__ svals, c64* __restrict__ panel,
                                                                 c64* __restrict__ upd, c64* __restrict__ r64,
                                                                 c64* __restrict__ d64, c32* __restrict__ d32,
                                                                 c32* __restrict__ pf, c32* __restrict__ pb,
                                                                 int* __restrict__ status) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int f = (int)front_list[blockIdx.x], op = blockIdx.y, tid = threadIdx.x;
    const FrontView Fv = front_view(F, f, op, panel, upd);
    const int nf = Fv.nf, nown = Fv.nown, nbnd = Fv.nbnd, ldp = nf | 1, ldb = nbnd | 1;
    c64* P = reinterpret_cast<c64*>(smem_raw);            // [k][i]: L, the unscaled rows above its diagonal; then the inverse
    c64* W = P + nown * ldp;                              // [k][j]: the boundary rows unscaled (l d); then M
    c64* di = W + nown * ldb;                             // 1 / d
    c64* red = di + nown;
    const int64_t ch0 = F.child_ptr[f], ch1 = F.child_ptr[f + 1];
    const bool kids = ch1 > ch0;
    for (int q = tid; q < nown * ldp; q += SF_THREADS) P[q] = zero<double>();
    if (kids)
        for (int q = tid; q < nbnd * nbnd; q += SF_THREADS) Fv.upd[q] = zero<double>();
    __syncthreads();
    {
        const c64* sv = svals + (int64_t)op * F.nsv;
        for (int64_t e = F.ent_ptr[f] + tid; e < F.ent_ptr[f + 1]; e += SF_THREADS)
            P[F.ent_col[e] * ldp + F.ent_row[e]] += sv[F.ent_s[e]];
    }
    __syncthreads();
    for (int64_t ci = ch0; ci < ch1; ++ci) {
        const int c = (int)F.child_idx[ci], nb = (int)F.nbnd[c];
        const int64_t* map = F.cmap_idx + F.cmap_ptr[ci];
        const c64* U = upd + (int64_t)op * F.upd_total + F.upd_off[c];
        for (int q = tid; q < nb * nb; q += SF_THREADS) {
            const int j = q / nb, i = q - j * nb;
            if (i < j) continue;
            const int mi = (int)map[i], mj = (int)map[j];
            if (mj < nown) P[mj * ldp + mi] += U[q];
            else Fv.upd[(mj - nown) * nbnd + (mi - nown)] += U[q];
        }
        __syncthreads();
    }
    // the own columns
    for (int k = 0; k < nown; ++k) {
        const int R = nf - k, nseg = R >= SF_THREADS ? 1 : min(SF_THREADS / R, max(1, k / 4));
        c64* pk = P + k * ldp;
        for (int t0 = 0; t0 < R; t0 += SF_THREADS) {       // (a front of more rows than threads takes them in turns)
            const int seg = nseg > 1 ? tid / R : 0, i = k + t0 + tid - seg * R;
            c64 acc = zero<double>();
            const bool act = seg < nseg && i < nf;
            if (act)
                for (int m = seg; m < k; m += nseg) cfma(acc, P[m * ldp + i], pk[m]);
            if (nseg > 1) {
                red[tid] = acc;
                __syncthreads();
                if (act && seg == 0)
                    for (int q = 1; q < nseg; ++q) acc += red[q * R + tid];
            }
            if (act && seg == 0) {
                const c64 v = pk[i] - acc;
                pk[i] = v;
                if (i == k) di[k] = pivot_inverse(v, status);
            }
        }
        __syncthreads();
        const c64 dk = di[k];
        for (int i = k + 1 + tid; i < nf; i += SF_THREADS) {
            const c64 v = pk[i];
            if (i < nown) P[i * ldp + k] = v;              // w(i, k), above the diagonal of column i
            else W[k * ldb + i - nown] = v;
            pk[i] = v * dk;
        }
        __syncthreads();
    }
    // the update matrix, lower triangle; threads run down its columns
    const int ntri = nbnd * (nbnd + 1) / 2;
    for (int e = tid; e < ntri; e += SF_THREADS) {
        int a, b;
        lower_tile(e, a, b);
        const int i = nbnd - 1 - b, j = nbnd - 1 - a;
        c64 acc = zero<double>();
        for (int k = 0; k < nown; ++k) cfma(acc, P[k * ldp + nown + i], W[k * ldb + j]);
        c64& u = Fv.upd[j * nbnd + i];
        u = (kids ? u : zero<double>()) - acc;
    }
    // X = L_own^-1, row i from the rows above it: X(i,c) = -(L(i,c) + sum_{c<m<i} L(i,m) X(m,c))
    __syncthreads();
    for (int i = 1; i < nown; ++i) {
        const int nseg = i >= SF_THREADS ? 1 : min(SF_THREADS / i, max(1, i / 4));
        c64 keep = zero<double>();
        for (int t0 = 0; t0 < i; t0 += SF_THREADS) {
            const int seg = nseg > 1 ? tid / i : 0, c = t0 + tid - seg * i;
            const bool act = seg < nseg && c < i;
            c64 acc = zero<double>();
            if (act)
                for (int m = c + 1 + seg; m < i; m += nseg) cfma(acc, P[m * ldp + i], P[c * ldp + m]);
            if (nseg > 1) {
                red[tid] = acc;
                __syncthreads();
                if (act && seg == 0)
                    for (int q = 1; q < nseg; ++q) acc += red[q * i + tid];
            }
            if (act && seg == 0) {
                acc += P[c * ldp + i];
                keep = mk<double>(-acc.re, -acc.im);
            }
        }
        __syncthreads();                                   // every term has read row i of L (nown <= SF_THREADS here)
        if (tid < i) P[tid * ldp + i] = keep;
        __syncthreads();
    }
    // M = -L_bnd X, over the unscaled rows
    for (int e = tid; e < nown * nbnd; e += SF_THREADS) {
        const int c = e / nbnd, j = e - c * nbnd;
        c64 acc = P[c * ldp + nown + j];
        for (int m = c + 1; m < nown; ++m) cfma(acc, P[m * ldp + nown + j], P[c * ldp + m]);
        W[c * ldb + j] = mk<double>(-acc.re, -acc.im);
    }
    __syncthreads();
    auto at = [&](int i, int k) {
        return i < k ? zero<double>() : i == k ? mk<double>(1.0, 0.0) : i < nown ? P[k * ldp + i] : W[k * ldb + i - nown];
    };
    const SweepTiles T(S, f, op, nf, nown, pf, pb);
    const int64_t base = (int64_t)op * F.panel_total + F.panel_off[f], dbase = (int64_t)op * F.nfac + F.own_start[f];
    for (int q = tid; q < nf * nown; q += SF_THREADS) {
        const int k = q / nf, i = q - k * nf;
        const c64 v = at(i, k);
        if (r64) Fv.panel[q] = v;
        T.fwd(i, k, cvt<float>(v));
    }
    for (int q = tid; q < nf * nown; q += SF_THREADS) {
        const int i = q / nown, k = q - i * nown;
        const c64 v = at(i, k);
        if (r64) r64[base + q] = v;
        T.bwd(i, k, cvt<float>(v));
    }
    for (int k = tid; k < nown; k += SF_THREADS) {
        d64[dbase + k] = di[k];
        d32[dbase + k] = cvt<float>(di[k]);
    }
}

void launch_small_fronts(const Fronts& F, const SweepPlan& S, const int64_t* front_list, int nfront, size_t smem,
                         const c64* svals, c64* panel, c64* upd, c64* r64, c64* d64, c32* d32, c32* pf, c32* pb, int nops,
                         int* status, cudaStream_t st) {
    raise_smem((const void*)small_front_kernel, smem);
    pdl_launch(small_front_kernel, dim3(nfront, nops), SF_THREADS, smem, st, F, S, front_list, svals, panel, upd, r64, d64, d32, pf, pb,
                                                                     status);
    GT_LAUNCH_CHECK();
}

// Large fronts: blocked elimination, FB own columns per step, every step over many CTAs (the top of the tree
// has a few fronts per operator, and an SM's FP64 rate is 1/152 of the GPU's):
//   diag   one CTA per (front, operator) factors the FB x FB diagonal block in shared memory and inverts its L11
//   rows   W21 = A21 L11^-T as a product with the inverse, L21 = W21 D^-1, 32 rows per CTA
//   trail  A22 -= L21 D L21^T over FT x FT tiles of the trailing lower triangle, one tile per CTA
// Tiles of 32 x 32 (32 us of an SM's FP64 pipe each; 64 x 64 took 127): the last steps of a top front have a few tiles
// for 152 SMs.  A warp's FP64 instruction holds its quarter of the pipe for 64 cycles whatever its active lanes, so no step
// leaves a product chain to one thread: rows by substitution, a thread a row, took 90 us a step.
constexpr int FB = FACTOR_BLOCK, FT = 32;

// the inverses of the diagonal blocks' L11: [op][first block of the front + kb / FB][FB x FB], row-major
struct DiagInv {
    c64* x;
    const int* first;          // [nfront] first block of each large front
    int64_t total;             // blocks per operator
    __device__ __forceinline__ c64* of(int f, int op, int kb) const {
        return x + ((int64_t)op * total + first[f] + kb / FB) * (FB * FB);
    }
};

// A large front's entries before elimination: the own columns of S and the children's update matrices, one child
// at a time (their boundaries overlap).  The panels start zeroed (one memset before the first level); the
// update matrix's slot is shared with matrices of other levels (its last owner's was assembled into its
// parent at an earlier level) and is cleared here.
__global__ void assemble_fronts_kernel(Fronts F, const int64_t* __restrict__ front_list, const c64* __restrict__ svals,
                                       c64* __restrict__ panel, c64* __restrict__ upd) {
    pdl_enter();
    const int f = (int)front_list[blockIdx.x], op = blockIdx.y;
    const FrontView Fv = front_view(F, f, op, panel, upd);
    const int tid = threadIdx.x, nth = blockDim.x;
    for (int64_t q = tid; q < (int64_t)Fv.nbnd * Fv.nbnd; q += nth) Fv.upd[q] = zero<double>();
    __syncthreads();
    const c64* sv = svals + (int64_t)op * F.nsv;
    for (int64_t e = F.ent_ptr[f] + tid; e < F.ent_ptr[f + 1]; e += nth) Fv.at(F.ent_row[e], F.ent_col[e]) += sv[F.ent_s[e]];
    __syncthreads();
    for (int64_t ci = F.child_ptr[f]; ci < F.child_ptr[f + 1]; ++ci) {
        const int c = (int)F.child_idx[ci];
        const int nb = (int)F.nbnd[c];
        const int64_t* map = F.cmap_idx + F.cmap_ptr[ci];
        const c64* U = upd + (int64_t)op * F.upd_total + F.upd_off[c];
        const int warp = tid >> 5, lane = tid & 31;
        for (int j = warp; j < nb; j += nth >> 5) {
            const int mj = (int)map[j];
            for (int i = j + lane; i < nb; i += 32) Fv.at((int)map[i], mj) += U[(int64_t)j * nb + i];
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) tiled_diag_kernel(Fronts F, const int64_t* __restrict__ front_list, int kb,
                                                         c64* __restrict__ panel, c64* __restrict__ upd, DiagInv X,
                                                         int* __restrict__ status) {
    pdl_enter();
    __shared__ c64 a[FB][FB + 1];
    __shared__ c64 x[FB][FB + 1];
    __shared__ c64 red[256];
    __shared__ c64 sd;
    const int f = (int)front_list[blockIdx.x], op = blockIdx.y;
    const FrontView Fv = front_view(F, f, op, panel, upd);
    const int nb = min(FB, Fv.nown - kb);
    if (nb <= 0) return;
    const int tid = threadIdx.x;
    for (int q = tid; q < FB * FB; q += 256) {
        const int j = q / FB, i = q - j * FB;
        a[i][j] = (i < nb && j <= i) ? Fv.panel[(int64_t)(kb + j) * Fv.nf + kb + i] : zero<double>();
    }
    __syncthreads();
    for (int k = 0; k < nb; ++k) {
        // column k as dot products over the columns before it; w = l d unscaled in the upper triangle
        const int R = nb - k, nseg = min(256 / R, max(1, k / 4)), seg = tid / R, i = k + tid - seg * R;
        c64 acc = zero<double>();
        if (seg < nseg)
            for (int m = seg; m < k; m += nseg) cfma(acc, a[i][m], a[m][k]);
        red[tid] = acc;
        __syncthreads();
        if (tid < R) {
            for (int q = 1; q < nseg; ++q) acc += red[q * R + tid];
            const c64 v = a[i][k] - acc;
            a[i][k] = v;
            if (i == k) sd = pivot_inverse(v, status);
        }
        __syncthreads();
        if (tid < R && i > k) {
            const c64 v = a[i][k];
            a[k][i] = v;
            a[i][k] = v * sd;
        }
        __syncthreads();
    }
    for (int q = tid; q < FB * FB; q += 256) {
        const int j = q / FB, i = q - j * FB;
        if (i < nb && j <= i) Fv.panel[(int64_t)(kb + j) * Fv.nf + kb + i] = a[i][j];
        x[i][j] = i == j ? mk<double>(1.0, 0.0) : zero<double>();
    }
    __syncthreads();
    for (int i = 1; i < nb; ++i) {                        // X(i,c) = -sum_{c<=m<i} L(i,m) X(m,c)
        const int nseg = min(256 / i, max(1, i / 4)), seg = tid / i, c = tid - seg * i;
        c64 acc = zero<double>();
        if (seg < nseg)
            for (int m = c + seg; m < i; m += nseg) cfma(acc, a[i][m], x[m][c]);
        red[tid] = acc;
        __syncthreads();
        if (tid < i) {
            for (int q = 1; q < nseg; ++q) acc += red[q * i + tid];
            x[i][c] = mk<double>(-acc.re, -acc.im);
        }
        __syncthreads();
    }
    c64* out = X.of(f, op, kb);
    for (int q = tid; q < FB * FB; q += 256) out[q] = x[q / FB][q % FB];
}

// rows of the front below the block: 32 per CTA
__global__ void __launch_bounds__(256) tiled_rows_kernel(Fronts F, const int64_t* __restrict__ front_list, int kb,
                                                         c64* __restrict__ panel, c64* __restrict__ upd, DiagInv X) {
    pdl_enter();
    __shared__ c64 x[FB][FB];
    __shared__ c64 ar[FB][FB + 1];                        // [row][column]
    __shared__ c64 dv[FB];
    const int f = (int)front_list[blockIdx.y], op = blockIdx.z;
    const FrontView Fv = front_view(F, f, op, panel, upd);
    const int nb = min(FB, Fv.nown - kb);
    if (nb <= 0) return;
    const int i0 = kb + nb + blockIdx.x * 32, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (i0 >= Fv.nf) return;
    const c64* xi = X.of(f, op, kb);
    for (int q = tid; q < FB * FB; q += 256) {
        x[q / FB][q % FB] = xi[q];
        const int m = q / FB, r = q - m * FB;
        ar[r][m] = m < nb && i0 + r < Fv.nf ? Fv.panel[(int64_t)(kb + m) * Fv.nf + i0 + r] : zero<double>();
    }
    if (tid < FB) {
        const c64 d = tid < nb ? Fv.panel[(int64_t)(kb + tid) * Fv.nf + kb + tid] : mk<double>(1.0, 0.0);
        dv[tid] = cdiv(mk<double>(1.0, 0.0), d);
    }
    __syncthreads();
    if (i0 + lane >= Fv.nf) return;
#pragma unroll
    for (int e = 0; e < FB / 8; ++e) {
        // columns e, 15 - e ... of the warp: the short and the long sums mixed
        const int k = (e & 1) ? FB - 1 - warp - 8 * (e >> 1) : warp + 8 * (e >> 1);
        if (k >= nb) continue;
        c64 w = ar[lane][k];
        for (int m = 0; m < k; ++m) cfma(w, ar[lane][m], x[k][m]);
        Fv.panel[(int64_t)(kb + k) * Fv.nf + i0 + lane] = w * dv[k];
    }
}

// 2 x 2 outputs per thread of a 32 x 32 tile: acc += A(m, 2 tx ..) B(m, 2 ty ..) over m < nb
__device__ __forceinline__ void tile_mac(const c64* As, const c64* Bs, int nb, int tx, int ty, c64 (&acc)[2][2]) {
    for (int m = 0; m < nb; ++m) {
        const c64 a0 = As[m * FT + tx], a1 = As[m * FT + tx + 16], b0 = Bs[m * FT + ty], b1 = Bs[m * FT + ty + 16];
        cfma(acc[0][0], a0, b0);
        cfma(acc[0][1], a0, b1);
        cfma(acc[1][0], a1, b0);
        cfma(acc[1][1], a1, b1);
    }
}

__global__ void __launch_bounds__(256) tiled_trail_kernel(Fronts F, const int64_t* __restrict__ front_list, int kb,
                                                          c64* __restrict__ panel, c64* __restrict__ upd) {
    pdl_enter();
    __shared__ c64 As[FB * FT], Bs[FB * FT];             // [m][r]: L(i0 + r, kb + m); [m][c]: L(j0 + c, kb + m) d_m
    const int f = (int)front_list[blockIdx.y];
    const FrontView Fv = front_view(F, f, blockIdx.z, panel, upd);
    const int nb = min(FB, Fv.nown - kb);
    if (nb <= 0) return;
    const int t0 = kb + nb, n2 = Fv.nf - t0;
    const int T = (n2 + FT - 1) / FT;
    if ((int64_t)blockIdx.x >= (int64_t)T * (T + 1) / 2) return;
    int bi, bj;
    lower_tile(blockIdx.x, bi, bj);
    const int i0 = t0 + bi * FT, j0 = t0 + bj * FT;
    for (int q = threadIdx.x; q < FB * FT; q += 256) {
        const int m = q / FT, r = q - m * FT;
        c64 a = zero<double>(), b = zero<double>();
        if (m < nb) {
            const c64* col = Fv.panel + (int64_t)(kb + m) * Fv.nf;
            if (i0 + r < Fv.nf) a = col[i0 + r];
            if (j0 + r < Fv.nf) b = col[j0 + r] * col[kb + m];
        }
        As[q] = a;
        Bs[q] = b;
    }
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    c64 acc[2][2] = {{zero<double>(), zero<double>()}, {zero<double>(), zero<double>()}};
    tile_mac(As, Bs, nb, tx, ty, acc);
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int i = i0 + tx + 16 * r, j = j0 + ty + 16 * c;
            if (i < Fv.nf && j <= i) Fv.at(i, j) -= acc[r][c];
        }
}

void launch_factor_tiled(const Fronts& F, const int64_t* front_list, int nf_level, int max_nf, int max_nown,
                         const c64* svals, c64* panel, c64* upd, c64* xinv, const int* xfirst, int64_t xtotal, int nops,
                         int* status, cudaStream_t st) {
    const DiagInv X{xinv, xfirst, xtotal};
    pdl_launch(assemble_fronts_kernel, dim3(nf_level, nops), 512, 0, st, F, front_list, svals, panel, upd);
    GT_LAUNCH_CHECK();
    for (int kb = 0; kb < max_nown; kb += FB) {
        pdl_launch(tiled_diag_kernel, dim3(nf_level, nops), 256, 0, st, F, front_list, kb, panel, upd, X, status);
        GT_LAUNCH_CHECK();
        const int below = max_nf - kb - 1;              // rows below the block (at least this front's nb of them)
        if (below <= 0) continue;
        pdl_launch(tiled_rows_kernel, dim3(ceil_div(below, 32), nf_level, nops), 256, 0, st, F, front_list, kb, panel, upd, X);
        GT_LAUNCH_CHECK();
        const int T = ceil_div(below, FT);
        pdl_launch(tiled_trail_kernel, dim3((unsigned)((int64_t)T * (T + 1) / 2), nf_level, nops), 256, 0, st, F, front_list, kb, panel,
                                                                                                     upd);
        GT_LAUNCH_CHECK();
    }
}

// Selective inversion of large fronts, blocked.  The inverted panel [Linv_own; -L_bnd Linv_own] is the first
// nown columns of the inverse of the unit lower triangular T = [L_own 0; L_bnd I], so it is computed in place
// as the forward substitution T Y = [I; 0], FB rows of T per step (kb = FB k, nb = the step's rows):
//   inv_rows   Y[kb.., c] = L_kk^-1 Y[kb.., c] for columns c < kb (their right-hand sides accumulated so far), with
//              the inverses the elimination left; the block's own entries become that inverse (D stays on the diagonal)
//   inv_trail  Y[i, c] -= L[i, kb..] Y[kb.., c] for the rows i below the block: first the columns c < kb,
//              then the block's own columns, whose Y takes the place of the L it is made from (each tile
//              reads its rows of L before it writes; the c < kb pass has read them all by then).
// The panel's upper triangle stays zero; the diagonal keeps D for panel_convert.
__global__ void __launch_bounds__(256) inv_rows_kernel(Fronts F, const int64_t* __restrict__ front_list, int kb,
                                                       c64* __restrict__ panel, DiagInv X) {
    pdl_enter();
    __shared__ c64 x[FB][FB];
    __shared__ c64 y[FB][FB + 1];                         // [column][row]
    const int f = (int)front_list[blockIdx.y], op = blockIdx.z;
    const int nown = (int)F.nown[f], nf = nown + (int)F.nbnd[f];
    const int nb = min(FB, nown - kb);
    const int c0 = blockIdx.x * 32, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (nb <= 0 || c0 > kb) return;
    c64* P = panel + (int64_t)op * F.panel_total + F.panel_off[f];
    const c64* xi = X.of(f, op, kb);
    if (c0 == kb) {                                       // the block's own columns
        for (int q = tid; q < FB * FB; q += 256) {
            const int k = q / FB, i = q - k * FB;
            if (i < nb && k < i) P[(int64_t)(kb + k) * nf + kb + i] = xi[i * FB + k];
        }
        return;
    }
    for (int q = tid; q < FB * FB; q += 256) {
        x[q / FB][q % FB] = xi[q];
        const int c = q / FB, r = q - c * FB;
        y[c][r] = r < nb ? P[(int64_t)(c0 + c) * nf + kb + r] : zero<double>();
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < FB / 8; ++e) {
        const int r = (e & 1) ? FB - 1 - warp - 8 * (e >> 1) : warp + 8 * (e >> 1);
        if (r >= nb) continue;
        c64 t = y[lane][r];
        for (int m = 0; m < r; ++m) cfma(t, x[r][m], y[lane][m]);
        P[(int64_t)(c0 + lane) * nf + kb + r] = t;
    }
}

// rows i >= kb + nb of the front; mode 0: columns c < kb (tile grid rt x ct), mode 1: the block's columns
__global__ void __launch_bounds__(256) inv_trail_kernel(Fronts F, const int64_t* __restrict__ front_list, int kb,
                                                        c64* __restrict__ panel, int mode) {
    pdl_enter();
    __shared__ c64 As[FB * FT], Bs[FB * FT];             // [m][r]: L(i0 + r, kb + m); [m][c]: Y(kb + m, c0 + c)
    const int f = (int)front_list[blockIdx.y];
    const int op = blockIdx.z;
    const int nown = (int)F.nown[f], nf = nown + (int)F.nbnd[f];
    const int nb = min(FB, nown - kb);
    if (nb <= 0) return;
    const int t0 = kb + nb, n2 = nf - t0;
    if (n2 <= 0) return;
    const int rt = (n2 + FT - 1) / FT;
    const int ncols = mode == 0 ? kb : nb;
    if (ncols <= 0) return;
    const int ct = (ncols + FT - 1) / FT;
    if ((int)blockIdx.x >= rt * ct) return;
    const int bi = blockIdx.x % rt, bj = blockIdx.x / rt;
    const int i0 = t0 + bi * FT, c0 = (mode == 0 ? 0 : kb) + bj * FT;
    const int c1 = mode == 0 ? kb : kb + nb;             // columns c0 .. min(c0 + FT, c1)
    c64* P = panel + (int64_t)op * F.panel_total + F.panel_off[f];
    for (int q = threadIdx.x; q < FB * FT; q += 256) {
        const int m = q / FT, r = q - m * FT;
        As[q] = m < nb && i0 + r < nf ? P[(int64_t)(kb + m) * nf + i0 + r] : zero<double>();
        // Y(kb + m, c), read down the columns: the block row's solved entries; in mode 1 the block's inverse, unit diagonal
        const int cl = q / FB, mm = q - cl * FB, c = c0 + cl;
        c64 b = zero<double>();
        if (mm < nb && c < c1) b = mode == 0 || c - kb < mm ? P[(int64_t)c * nf + kb + mm]
                                   : c - kb == mm ? mk<double>(1.0, 0.0) : zero<double>();
        Bs[mm * FT + cl] = b;
    }
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    c64 acc[2][2] = {{zero<double>(), zero<double>()}, {zero<double>(), zero<double>()}};
    tile_mac(As, Bs, nb, tx, ty, acc);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int j = c0 + ty + 16 * c;
        if (j >= c1) continue;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int i = i0 + tx + 16 * r;
            if (i >= nf) continue;
            c64& y = P[(int64_t)j * nf + i];
            y = (mode == 1 ? zero<double>() : y) - acc[r][c];
        }
    }
}

// the large fronts of all levels in a launch: they stand in the grid's second dimension, which ends at 65,535 (six planes of
// 1024 x 1024 have 31,000 of them)
template <typename L>
static void in_parts(int nfront, L&& launch) {
    constexpr int MOST = 65535;
    for (int f = 0; f < nfront; f += MOST) launch(f, std::min(MOST, nfront - f));
}

void launch_invert_tiled(const Fronts& F, const int64_t* front_list, const InvertPlan& plan, c64* panel, const c64* xinv,
                         const int* xfirst, int64_t xtotal, int nops, cudaStream_t st) {
    const DiagInv X{const_cast<c64*>(xinv), xfirst, xtotal};
    for (size_t s = 0; s < plan.count.size(); ++s) {
        const int kb = (int)s * FB;
        const int below = plan.max_nf[s] - kb - 1, rt = ceil_div(std::max(below, 0), FT);
        in_parts(plan.count[s], [&](int first, int n) {
            const int64_t* fr = front_list + first;
            pdl_launch(inv_rows_kernel, dim3(kb / 32 + 1, n, nops), 256, 0, st, F, fr, kb, panel, X);
            GT_LAUNCH_CHECK();
            if (below <= 0) return;
            if (kb > 0) {
                pdl_launch(inv_trail_kernel, dim3(rt * ceil_div(kb, FT), n, nops), 256, 0, st, F, fr, kb, panel, 0);
                GT_LAUNCH_CHECK();
            }
            pdl_launch(inv_trail_kernel, dim3(rt, n, nops), 256, 0, st, F, fr, kb, panel, 1);
            GT_LAUNCH_CHECK();
        });
    }
}

// Finish the large fronts' solve panels: an explicit unit diagonal (the pivots go to dinv as 1/D) and the copies the sweeps
// read: the FP32 forward and backward tiles and the FP64 row-major panel.
// r64 (the FP64 row-major copy) may be null: operators that keep their FP32 panels only
__global__ void panel_convert_kernel(Fronts F, SweepPlan S, const int64_t* __restrict__ front_list, c64* __restrict__ p64,
                                     c32* __restrict__ pf, c32* __restrict__ pb, c64* __restrict__ r64, c64* __restrict__ d64,
                                     c32* __restrict__ d32) {
    pdl_enter();
    const int f = (int)front_list[blockIdx.y];
    const int op = blockIdx.z;
    const int nown = (int)F.nown[f], nf = nown + (int)F.nbnd[f];
    const int64_t base = (int64_t)op * F.panel_total + F.panel_off[f];
    const int64_t dbase = (int64_t)op * F.nfac + F.own_start[f];
    const SweepTiles T(S, f, op, nf, nown, pf, pb);
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < (int64_t)nf * nown; q += (int64_t)gridDim.x * blockDim.x) {
        const int k = int(q / nf), i = int(q - (int64_t)k * nf);      // column-major element (i, k)
        c64 v = i < k ? zero<double>() : p64[base + q];
        if (i == k) {
            const c64 dv = cdiv(mk<double>(1.0, 0.0), v);
            d64[dbase + i] = dv;
            d32[dbase + i] = cvt<float>(dv);
            v = mk<double>(1.0, 0.0);
            p64[base + q] = v;
        }
        T.fwd(i, k, cvt<float>(v));
        T.bwd(i, k, cvt<float>(v));
        if (r64) r64[base + (int64_t)i * nown + k] = v;
    }
}

void launch_panel_convert(const Fronts& F, const SweepPlan& S, const int64_t* front_list, int nfront, c64* p64, c32* pf, c32* pb,
                          c64* r64, c64* d64, c32* d32, int nops, cudaStream_t st) {
    in_parts(nfront, [&](int first, int n) {
        pdl_launch(panel_convert_kernel, dim3(16, n, nops), 256, 0, st, F, S, front_list + first, p64, pf, pb, r64, d64, d32);
        GT_LAUNCH_CHECK();
    });
}

// ------------------------------------------------------------------------------------------ solves
// z, y: [col][nfac] in factor order; uvec: [col][vec_total] update vectors; sd: [col][S*nx*ny] in node order.
// After the factorisation each front's panel holds P = [Linv_own; -L_bnd Linv_own] (nf x nown, unit
// diagonal, zeros above it) and dinv = 1/D of its pivots (selective inversion), so that a front's solves are
// two dense matrix-vector products without a sequential chain:
//   forward   out = P w_own: own rows z_own = dinv * out, boundary rows w_bnd + out go up as the update
//   backward  y_own = P^T [z_own; y_bnd]   (y_bnd: the ancestors' results, final)
// A task is (front, group of <= 8 columns sharing its operator, block of rows / columns); its warps split
// the block into 32-row (32-column) tiles and the product's inner dimension into segments whose partial sums
// meet in shared memory.  The launch shape is chosen per level so that the top of the tree, with few fronts,
// still spreads over every SM.  Panel elements are read once per task by consecutive lanes, LB loads in flight.
constexpr int LB = 8;
constexpr int SOLVE_THREADS = 512;

// acc[c] += a * x[c] over all GC columns of one k-major shared row x (unused columns hold zeros)
template <int GC>
__device__ __forceinline__ void mac_row(c64* acc, c64 a, const c64* x) {
#pragma unroll
    for (int c = 0; c < GC; ++c) cfma(acc[c], a, x[c]);
}

// acc[c] += sum_{t < cnt} A[t * lda] x[t * xs + c]: A a strided run of panel elements (part of one row or
// column of a front's panel), x the matching k-major shared rows.  The first LB elements were loaded into
// l ahead of time (prefetch_run, issued before the shared rows were staged); LB loads in flight after that.
__device__ __forceinline__ void prefetch_run(const c64* __restrict__ A, int lda, int cnt, c64* l) {
#pragma unroll
    for (int u = 0; u < LB; ++u) l[u] = u < cnt ? A[u * lda] : zero<double>();
}

template <int GC>
__device__ __forceinline__ void sweep(const c64* __restrict__ A, int lda, const c64* x, int xs, int cnt,
                                      const c64* l0, c64* acc) {
#pragma unroll
    for (int u = 0; u < LB; ++u)
        if (u < cnt) mac_row<GC>(acc, l0[u], x + u * xs);
    A += LB * lda;
    x += LB * xs;
    int t = LB;
    for (; t + LB <= cnt; t += LB) {
        c64 l[LB];
#pragma unroll
        for (int u = 0; u < LB; ++u) l[u] = A[u * lda];
#pragma unroll
        for (int u = 0; u < LB; ++u) mac_row<GC>(acc, l[u], x + u * xs);
        A += LB * lda;
        x += LB * xs;
    }
    for (; t < cnt; ++t) {
        mac_row<GC>(acc, *A, x);
        A += lda;
        x += xs;
    }
}

// The forward rows of front f for a group: own rows of w (s in factor order plus the children's updates)
// into ws (k-major, ldw = GC) and boundary rows r0 <= p < r1 into wt ([c][TR]).  Loads are issued four
// at a time per thread ahead of their stores.
template <int GC>
__device__ __forceinline__ void fwd_gather(const Fronts& F, int f, const int* gs, int gc, const c64* __restrict__ sf,
                                           const c64* __restrict__ uvec, c64* ws, c64* wt, int TR, int r0, int r1) {
    const int nown = (int)F.nown[f];
    const int64_t own0 = F.own_start[f];
    const int tid = threadIdx.x, nth = blockDim.x;
    const int tot = gc * nown;
    for (int q = tot + tid; q < GC * nown; q += nth) ws[(q % nown) * GC + q / nown] = zero<double>();
    for (int q0 = tid; q0 < tot; q0 += 4 * nth) {
        c64 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = min(q0 + u * nth, tot - 1), c = q / nown;
            v[u] = sf[(int64_t)gs[c] * F.nfac + own0 + (q - c * nown)];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = q0 + u * nth;
            if (q < tot) ws[(q % nown) * GC + q / nown] = v[u];
        }
    }
    __syncthreads();
    for (int64_t ci = F.child_ptr[f]; ci < F.child_ptr[f + 1]; ++ci) {
        const int ch = (int)F.child_idx[ci];
        const int nb = (int)F.nbnd[ch], tc = gc * nb;
        const int64_t* map = F.cmap_idx + F.cmap_ptr[ci];
        const int64_t voff = F.vec_off[ch];
        for (int q0 = tid; q0 < tc; q0 += 4 * nth) {
            int p[4];
            c64 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int q = min(q0 + u * nth, tc - 1), c = q / nb, i = q - c * nb;
                p[u] = (int)map[i];
                v[u] = uvec[(int64_t)gs[c] * F.vec_total + voff + i];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int q = q0 + u * nth;
                if (q >= tc) break;
                const int c = q / nb;
                if (p[u] < nown) ws[p[u] * GC + c] += v[u];
                else if (p[u] >= r0 && p[u] < r1) wt[c * TR + p[u] - r0] += v[u];
            }
        }
        __syncthreads();
    }
}

// Forward assembly of a front split over several blocks, once per (front, group): w_own to wasm (factor
// order), the children's updates of the boundary rows to the front's own update-vector slots.
template <int GC>
__global__ void __launch_bounds__(256) fwd_assemble_kernel(Fronts F, const int64_t* __restrict__ front_list,
                                                           const c64* sf, c64* __restrict__ uvec, c64* wasm,
                                                           Groups G, int ldw, int TR) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    c64* ws = reinterpret_cast<c64*>(smem_raw);   // [k][GC]
    c64* wt = ws + GC * ldw;                      // [c][TR] boundary rows
    const int g = blockIdx.x % G.ngroup;
    const int f = (int)front_list[blockIdx.x / G.ngroup];
    const int* gs = G.gslot + G.gptr[g];
    const int gc = G.gptr[g + 1] - G.gptr[g];
    const int nown = (int)F.nown[f], nbnd = (int)F.nbnd[f], nf = nown + nbnd;
    const int64_t own0 = F.own_start[f];
    for (int q = threadIdx.x; q < GC * TR; q += blockDim.x) wt[q] = zero<double>();
    __syncthreads();
    fwd_gather<GC>(F, f, gs, gc, sf, uvec, ws, wt, TR, nown, nf);
    for (int q = threadIdx.x; q < gc * nown; q += blockDim.x) {
        const int c = q / nown, r = q - c * nown;
        wasm[(int64_t)gs[c] * F.nfac + own0 + r] = ws[r * GC + c];
    }
    for (int q = threadIdx.x; q < gc * nbnd; q += blockDim.x) {
        const int c = q / nbnd, j = q - c * nbnd;
        uvec[(int64_t)gs[c] * F.vec_total + F.vec_off[f] + j] = wt[c * TR + j];
    }
}

// pre: the front was assembled by fwd_assemble_kernel (own rows in wasm, boundary rows in uvec)
template <int GC>
__global__ void __launch_bounds__(SOLVE_THREADS, 2) fwd_gemv_kernel(Fronts F, const int64_t* __restrict__ front_list, int nblk,
                                                                 int rt, int kseg, const c64* __restrict__ panel,
                                                                 const c64* __restrict__ dinv, const c64* sf,
                                                                 c64* __restrict__ z, c64* __restrict__ uvec,
                                                                 const c64* wasm, Groups G, int ldw, int pre) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int TR = 32 * rt;
    c64* ws = reinterpret_cast<c64*>(smem_raw);   // [k][GC] own rows of w
    c64* wt = ws + GC * ldw;                      // [c][TR] the block's boundary rows of w
    c64* red = wt + GC * TR;                      // [seg][c][TR] partial sums
    const int b = blockIdx.x % nblk, rest = blockIdx.x / nblk;
    const int g = rest % G.ngroup;
    const int f = (int)front_list[rest / G.ngroup];
    const int nown = (int)F.nown[f], nf = nown + (int)F.nbnd[f];
    const int r0 = b * TR;
    if (r0 >= nf) return;
    const int r1 = min(nf, r0 + TR);
    const int* gs = G.gslot + G.gptr[g];
    const int gc = G.gptr[g + 1] - G.gptr[g], op = G.op[g];
    const int64_t own0 = F.own_start[f];
    const int tid = threadIdx.x, nth = blockDim.x;
    const c64* __restrict__ P = panel + (int64_t)op * F.panel_total + F.panel_off[f];
    const int lane = tid & 31, warp = tid >> 5;
    const int tile = warp % rt, seg = warp / rt;
    const int rl = tile * 32 + lane, r = r0 + rl;
    // the tile's rows need columns k < min(nown, last row + 1) (P is zero above its diagonal)
    const int kmax = min(nown, r0 + tile * 32 + 32);
    const int ks = (kmax + kseg - 1) / kseg;
    const int k0 = min(kmax, seg * ks), k1 = min(kmax, k0 + ks);
    const bool valid = r < r1;
    // lanes past the block's rows sweep its last row (results dropped)
    const c64* A = P + (int64_t)k0 * nf + min(r, r1 - 1);
    if (pre) {
        for (int q = tid; q < GC * nown; q += nth) {
            const int c = q / nown, r = q - c * nown;
            ws[r * GC + c] = c < gc ? wasm[(int64_t)gs[c] * F.nfac + own0 + r] : zero<double>();
        }
        for (int q = tid; q < GC * TR; q += nth) {
            const int c = q / TR, rr = q - c * TR, row = r0 + rr;
            wt[q] = (c < gc && row >= nown && row < r1)
                        ? uvec[(int64_t)gs[c] * F.vec_total + F.vec_off[f] + (row - nown)] : zero<double>();
        }
        __syncthreads();
    } else {
        for (int q = tid; q < GC * TR; q += nth) wt[q] = zero<double>();
        __syncthreads();
        fwd_gather<GC>(F, f, gs, gc, sf, uvec, ws, wt, TR, r0, r1);
    }
    c64 l0[LB];
    prefetch_run(A, nf, k1 - k0, l0);
    c64 acc[GC];
#pragma unroll
    for (int c = 0; c < GC; ++c) acc[c] = zero<double>();
    sweep<GC>(A, nf, ws + k0 * GC, GC, k1 - k0, l0, acc);
    if (kseg > 1) {
#pragma unroll
        for (int c = 0; c < GC; ++c)
            if (c < gc) red[(seg * GC + c) * TR + rl] = acc[c];
        __syncthreads();
        for (int q = tid; q < gc * TR; q += nth) {
            const int c = q / TR, rr = q - c * TR;
            if (r0 + rr >= r1) continue;
            c64 v = red[c * TR + rr];
            for (int sg = 1; sg < kseg; ++sg) v += red[(sg * GC + c) * TR + rr];
            const int row = r0 + rr;
            if (row < nown) z[(int64_t)gs[c] * F.nfac + own0 + row] = dinv[(int64_t)op * F.nfac + own0 + row] * v;
            else uvec[(int64_t)gs[c] * F.vec_total + F.vec_off[f] + (row - nown)] = wt[c * TR + rr] + v;
        }
    } else if (valid) {
        if (r < nown) {
            const c64 dv = dinv[(int64_t)op * F.nfac + own0 + r];
#pragma unroll
            for (int c = 0; c < GC; ++c)
                if (c < gc) z[(int64_t)gs[c] * F.nfac + own0 + r] = dv * acc[c];
        } else {
#pragma unroll
            for (int c = 0; c < GC; ++c)
                if (c < gc) uvec[(int64_t)gs[c] * F.vec_total + F.vec_off[f] + (r - nown)] = wt[c * TR + rl] + acc[c];
        }
    }
}

template <int GC>
__global__ void __launch_bounds__(SOLVE_THREADS, 2) bwd_gemv_kernel(Fronts F, const int64_t* __restrict__ front_list, int nblk,
                                                                 int ct, int iseg, int cw,
                                                                 const c64* __restrict__ panel_rm,
                                                                 const c64* __restrict__ z, c64* __restrict__ y,
                                                                 c64* __restrict__ sd, Groups G, int ldv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int TC = cw * ct;       // a tile: cw columns, its warp's 32 / cw lane groups take alternate rows
    c64* v = reinterpret_cast<c64*>(smem_raw);    // [i - kb0][GC]: rows kb0 .. nf of [z_own; y_bnd]
    c64* red = v + GC * ldv;                      // [seg][c][TC]
    const int b = blockIdx.x % nblk, rest = blockIdx.x / nblk;
    const int g = rest % G.ngroup;
    const int f = (int)front_list[rest / G.ngroup];
    const int nown = (int)F.nown[f], nf = nown + (int)F.nbnd[f];
    const int kb0 = b * TC;
    if (kb0 >= nown) return;
    const int kb1 = min(nown, kb0 + TC);
    const int* gs = G.gslot + G.gptr[g];
    const int gc = G.gptr[g + 1] - G.gptr[g], op = G.op[g];
    const int64_t own0 = F.own_start[f];
    const int64_t* bnd = F.bnd_idx + F.bnd_ptr[f];
    const int tid = threadIdx.x, nth = blockDim.x;
    const c64* __restrict__ P = panel_rm + (int64_t)op * F.panel_total + F.panel_off[f];   // (nf x nown) row-major
    const int lane = tid & 31, warp = tid >> 5;
    const int nph = 32 / cw, ph = lane / cw;
    const int tile = warp % ct, seg = warp / ct;
    const int kl = tile * cw + (lane - ph * cw), k = kb0 + kl;
    // the tile's columns need rows i >= its first column (P is zero above its diagonal)
    const int it0 = min(nf, kb0 + tile * cw);
    const int is = (nf - it0 + iseg - 1) / iseg;
    const int i0 = min(nf, it0 + seg * is), i1 = min(nf, i0 + is);
    const int cnt = max(0, (i1 - i0 - ph + nph - 1) / nph);
    const bool valid = k < kb1;
    // lanes past the block's columns sweep its last column (results dropped)
    const c64* A = P + (int64_t)(i0 + ph) * nown + min(k, kb1 - 1);
    c64 l0[LB];
    prefetch_run(A, nph * nown, cnt, l0);
    const int nv = nf - kb0, tot = gc * nv;
    for (int q = gc * nv + tid; q < GC * nv; q += nth) {
        const int c = q / nv;
        v[(q - c * nv) * GC + c] = zero<double>();
    }
    for (int q0 = tid; q0 < tot; q0 += 4 * nth) {
        int64_t src[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = min(q0 + u * nth, tot - 1), c = q / nv, i = kb0 + (q - c * nv);
            src[u] = (int64_t)gs[c] * F.nfac + (i < nown ? own0 + i : bnd[i - nown]);
        }
        c64 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = min(q0 + u * nth, tot - 1), c = q / nv, i = kb0 + (q - c * nv);
            x[u] = i < nown ? z[src[u]] : y[src[u]];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = q0 + u * nth;
            if (q < tot) v[(q % nv) * GC + q / nv] = x[u];
        }
    }
    __syncthreads();
    c64 acc[GC];
#pragma unroll
    for (int c = 0; c < GC; ++c) acc[c] = zero<double>();
    sweep<GC>(A, nph * nown, v + (i0 + ph - kb0) * GC, nph * GC, cnt, l0, acc);
    if (nph == 2) {
#pragma unroll
        for (int c = 0; c < GC; ++c) {
            acc[c].re += __shfl_xor_sync(0xffffffffu, acc[c].re, 16);
            acc[c].im += __shfl_xor_sync(0xffffffffu, acc[c].im, 16);
        }
    }
    if (iseg > 1) {
#pragma unroll
        for (int c = 0; c < GC; ++c)
            if (c < gc && ph == 0) red[(seg * GC + c) * TC + kl] = acc[c];
        __syncthreads();
        for (int q = tid; q < gc * TC; q += nth) {
            const int c = q / TC, kk = q - c * TC;
            if (kb0 + kk >= kb1) continue;
            c64 s = red[c * TC + kk];
            for (int sg = 1; sg < iseg; ++sg) s += red[(sg * GC + c) * TC + kk];
            y[(int64_t)gs[c] * F.nfac + own0 + kb0 + kk] = s;
            sd[(int64_t)gs[c] * F.nnode + F.iperm[own0 + kb0 + kk]] = s;
        }
    } else if (valid && ph == 0) {
        const int64_t node = F.iperm[own0 + k];
#pragma unroll
        for (int c = 0; c < GC; ++c)
            if (c < gc) {
                y[(int64_t)gs[c] * F.nfac + own0 + k] = acc[c];
                sd[(int64_t)gs[c] * F.nnode + node] = acc[c];
            }
    }
}

// Launch shape of a level, chosen from the level's fronts alone, never from the number of column groups in the
// solve: the split of the inner dimension sets the order in which partial sums meet, so a column's arithmetic
// (and rounding) must not depend on how many columns share the launch.  The choice assumes a nominal
// NOMINAL_GROUPS groups per front (the sweep batches 8 columns per group): with enough (front, group) tasks
// to fill the GPU a block takes a whole small front; otherwise a block takes one 32-row (32-column) tile and
// splits the inner dimension over warps.
constexpr int NOMINAL_GROUPS = 32;
static void solve_shape(int nfront_level, int ntile, int inner, int& per_blk, int& nseg) {
    const int fill = 8 * 152;
    const int64_t ntask = (int64_t)nfront_level * NOMINAL_GROUPS;
    if (ntask * ntile >= fill && ntile <= 4 && ntask >= fill / 2) {
        per_blk = ntile;
        nseg = 1;
    } else {
        per_blk = 1;
        nseg = std::max(1, std::min(SOLVE_THREADS / 32, (inner + 63) / 64));
    }
}

template <int GC>
static void fwd_level_gc(const Fronts& F, const int64_t* front_list, int nf_level, int max_nf, int max_nown,
                         const c64* panel, const c64* dinv, const c64* sf, c64* z, c64* uvec, c64* wasm,
                         const Groups& G, cudaStream_t st) {
    const int ntask = nf_level * G.ngroup;
    const int ntile = ceil_div(max_nf, 32);
    int rt, kseg;
    solve_shape(nf_level, ntile, max_nown, rt, kseg);
    const int nblk = ceil_div(ntile, rt), ldw = std::max(max_nown, 1);
    const int pre = nblk > 1;
    if (pre) {
        const int TRa = std::max(max_nf - 1, 1);
        const size_t sa = (size_t)GC * (ldw + TRa) * sizeof(c64);
        raise_smem((const void*)fwd_assemble_kernel<GC>, sa);
        fwd_assemble_kernel<GC><<<ntask, 256, sa, st>>>(F, front_list, sf, uvec, wasm, G, ldw, TRa);
        GT_LAUNCH_CHECK();
    }
    const size_t sm = (size_t)GC * (ldw + 32 * rt + (kseg > 1 ? kseg * 32 * rt : 0)) * sizeof(c64);
    raise_smem((const void*)fwd_gemv_kernel<GC>, sm);
    fwd_gemv_kernel<GC><<<ntask * nblk, 32 * rt * kseg, sm, st>>>(F, front_list, nblk, rt, kseg, panel, dinv, sf, z, uvec,
                                                                wasm, G, ldw, pre);
    GT_LAUNCH_CHECK();
}

template <int GC>
static void bwd_level_gc(const Fronts& F, const int64_t* front_list, int nf_level, int max_nf, int max_nown,
                         const c64* panel_rm, const c64* z, c64* y, c64* sd, const Groups& G, cudaStream_t st) {
    const int ntask = nf_level * G.ngroup;
    // tiles of 16 columns (two lane groups on alternate rows) where they waste fewer lanes than 32
    const int cw = ceil_div(max_nown, 16) * 16 - max_nown < ceil_div(max_nown, 32) * 32 - max_nown ? 16 : 32;
    const int ntile = ceil_div(max_nown, cw);
    int ct, iseg;
    solve_shape(nf_level, ntile, max_nf, ct, iseg);
    const int nblk = ceil_div(ntile, ct), ldv = std::max(max_nf, 1);
    const size_t sm = (size_t)GC * (ldv + (iseg > 1 ? iseg * cw * ct : 0)) * sizeof(c64);
    raise_smem((const void*)bwd_gemv_kernel<GC>, sm);
    bwd_gemv_kernel<GC><<<ntask * nblk, 32 * ct * iseg, sm, st>>>(F, front_list, nblk, ct, iseg, cw, panel_rm, z, y, sd,
                                                                 G, ldv);
    GT_LAUNCH_CHECK();
}

// the column-group widths the sweep kernels are built for: a front's rows for GC columns are staged in shared
// memory, so wide fronts take narrower groups (the panel is then read once per fewer columns)
void launch_fwd_level(const Fronts& F, const int64_t* front_list, int nf_level, int max_nf, int max_nown,
                      const c64* panel, const c64* dinv, const c64* sf, c64* z, c64* uvec, c64* wasm,
                      const Groups& G, int gmax, cudaStream_t st) {
    switch (gmax) {
        case 8: fwd_level_gc<8>(F, front_list, nf_level, max_nf, max_nown, panel, dinv, sf, z, uvec, wasm, G, st); return;
        case 4: fwd_level_gc<4>(F, front_list, nf_level, max_nf, max_nown, panel, dinv, sf, z, uvec, wasm, G, st); return;
        case 2: fwd_level_gc<2>(F, front_list, nf_level, max_nf, max_nown, panel, dinv, sf, z, uvec, wasm, G, st); return;
        case 1: fwd_level_gc<1>(F, front_list, nf_level, max_nf, max_nown, panel, dinv, sf, z, uvec, wasm, G, st); return;
        default: throw CudaError{cudaErrorInvalidValue, "column group width must be 8, 4, 2 or 1"};
    }
}

void launch_bwd_level(const Fronts& F, const int64_t* front_list, int nf_level, int max_nf, int max_nown,
                      const c64* panel_rm, const c64* z, c64* y, c64* sd, const Groups& G, int gmax,
                      cudaStream_t st) {
    switch (gmax) {
        case 8: bwd_level_gc<8>(F, front_list, nf_level, max_nf, max_nown, panel_rm, z, y, sd, G, st); return;
        case 4: bwd_level_gc<4>(F, front_list, nf_level, max_nf, max_nown, panel_rm, z, y, sd, G, st); return;
        case 2: bwd_level_gc<2>(F, front_list, nf_level, max_nf, max_nown, panel_rm, z, y, sd, G, st); return;
        case 1: bwd_level_gc<1>(F, front_list, nf_level, max_nf, max_nown, panel_rm, z, y, sd, G, st); return;
        default: throw CudaError{cudaErrorInvalidValue, "column group width must be 8, 4, 2 or 1"};
    }
}

}  // namespace gt
