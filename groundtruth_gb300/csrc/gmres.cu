// Krylov vector work of the restarted GMRES (GroundTruth: _gmres, peec.py:3093-3224; the device twin of
// gpu.TorchVectors, gpu.py:409-462), batched over slots (one basis per column being solved).
//
// Classical Gram-Schmidt with one conditional re-orthogonalisation (DGKS: a second pass when the norm fell
// below 0.7 of the product's, peec.py:3156-3159).  Dot products are reduced per warp by shuffles, per block
// through shared memory in FP64, and across blocks in FP64 by the slot's last block to finish, over per-block
// partials in a fixed order: results are reproducible.  The Hessenberg column, its Givens rotations and the
// least-squares right-hand side live on the device in FP64 (peec.py:3160-3184); so does the decision that a
// slot's cycle has converged.  A basis of the arithmetic's own type is stored unnormalised (vinv: 1 / norm).
#include <type_traits>
#include "kernels.h"
#include "solver.h"

namespace gt {

template <typename R> __device__ __forceinline__ R shfl_sum(R v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// basis entries: loads and stores of cx<R> or of FP16 pairs
template <typename R> __device__ __forceinline__ cx<R> bload(const cx<R>* p) { return *p; }
__device__ __forceinline__ c32 bload(const h16c* p) {
    const float2 f = __half22float2(p->v);
    return mk<float>(f.x, f.y);
}
template <typename R> __device__ __forceinline__ void bstore(cx<R>* p, cx<R> v) { *p = v; }
__device__ __forceinline__ void bstore(h16c* p, c32 v) { p->v = __floats2half2_rn(v.re, v.im); }

constexpr int DOT_THREADS = 256;
constexpr int DOT_EPT = 8;
constexpr int DOT_CHUNK = DOT_THREADS * DOT_EPT;
// the update keeps fewer elements per thread (more blocks resident, more basis vectors in flight); with 2 or 1 it is slower
// where it matters (128 columns of 100,000 unknowns: 243 and 412 ms of updates against 207) and 1 us faster on one small column
constexpr int UPD_EPT = 4;
constexpr int UPD_CHUNK = DOT_THREADS * UPD_EPT;

int update_chunks(int64_t n) { return (int)((n + UPD_CHUNK - 1) / UPD_CHUNK); }
constexpr int MAXV = 256;

// Whether the calling block is the last of the slot's nblk to get here (its partial results, and the others', are then
// visible to it); it leaves the slot's counter at zero for the next kernel.
__device__ __forceinline__ bool last_of_slot(int* done, int slot, int nblk) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(done + slot, 1) == nblk - 1;
        if (last) done[slot] = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// partial[(slot * nchunk + chunk) * (nv + 1) + i] = sum over the chunk of conj(V_i) w, i < nv; index nv: |w|^2.  The
// slot's last block adds the chunks in a fixed order to out[slot * ldo + i]: a reduction kernel of its own, one block per
// slot, was a launch more on a chain of short ones.
template <typename R, typename B>
__global__ void __launch_bounds__(DOT_THREADS) dots_kernel(const B* __restrict__ V, int64_t ldv, int64_t lds, int nv,
                                                           const cx<R>* __restrict__ w, int64_t ldw, int64_t n,
                                                           const int* __restrict__ active, c64* __restrict__ partial,
                                                           int nchunk, int vpb, R vs, const double* __restrict__ vinv, int ldi,
                                                           c64* __restrict__ out, int ldo, int* done) {
    pdl_enter();
    __shared__ c64 red[DOT_THREADS / 32][MAXV + 1];
    const int slot = blockIdx.y;
    if (active && !active[slot]) return;
    const int chunk = blockIdx.x;
    const int64_t base = (int64_t)chunk * DOT_CHUNK;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    cx<R> wv[DOT_EPT];
    R nrm = 0;
#pragma unroll
    for (int e = 0; e < DOT_EPT; ++e) {
        int64_t q = base + e * DOT_THREADS + tid;
        wv[e] = q < n ? w[(int64_t)slot * ldw + q] : zero<R>();
        nrm += norm2(wv[e]);
    }
    const B* Vs = V + (int64_t)slot * lds;
    // UN basis vectors' loads in flight together (FP32 arithmetic; FP64 keeps one)
    constexpr int UN = sizeof(R) == 4 ? 2 : 1;
    const int i0 = blockIdx.z * vpb, i1 = min(nv, i0 + vpb);
    for (int i = i0; i < i1; i += UN) {
        cx<R> v[UN][DOT_EPT];
#pragma unroll
        for (int u = 0; u < UN; ++u)
#pragma unroll
            for (int e = 0; e < DOT_EPT; ++e) {
                const int64_t q = base + e * DOT_THREADS + tid;
                v[u][e] = i + u < i1 && q < n ? bload(Vs + (int64_t)(i + u) * ldv + q) : zero<R>();
            }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            R ar = 0, ai = 0;
#pragma unroll
            for (int e = 0; e < DOT_EPT; ++e) {
                ar += v[u][e].re * wv[e].re + v[u][e].im * wv[e].im;
                ai += v[u][e].re * wv[e].im - v[u][e].im * wv[e].re;
            }
            ar = shfl_sum(ar);
            ai = shfl_sum(ai);
            if (lane == 0 && i + u < i1) red[warp][i + u] = mk<double>((double)ar * vs, (double)ai * vs);
        }
    }
    nrm = shfl_sum(nrm);
    if (lane == 0) red[warp][nv] = mk<double>(nrm, 0.0);
    __syncthreads();
    for (int i = i0 + tid; i < i1 + (i1 == nv); i += DOT_THREADS) {
        c64 acc = zero<double>();
        for (int q = 0; q < DOT_THREADS / 32; ++q) acc += red[q][i];
        partial[((int64_t)slot * nchunk + chunk) * (nv + 1) + i] = acc;
    }
    if (!last_of_slot(done, slot, nchunk * gridDim.z)) return;
    const c64* ps = partial + (int64_t)slot * nchunk * (nv + 1);
    constexpr int PER = 4;                               // threads per sum
    for (int b = 0; b <= nv; b += DOT_THREADS / PER) {
        const int i = b + tid / PER, sub = tid % PER;
        c64 acc = zero<double>();
        if (i <= nv)
            for (int c = sub; c < nchunk; c += PER) {
                const double2 v = __ldcg(reinterpret_cast<const double2*>(ps + (int64_t)c * (nv + 1) + i));
                acc += mk<double>(v.x, v.y);
            }
        for (int o = 1; o < PER; o <<= 1) {
            acc.re += __shfl_xor_sync(0xffffffffu, acc.re, o);
            acc.im += __shfl_xor_sync(0xffffffffu, acc.im, o);
        }
        if (i <= nv && sub == 0)
            out[(int64_t)slot * ldo + i] = vinv && i < nv ? vinv[(int64_t)slot * ldi + i] * acc : acc;
    }
}

template <typename R, typename B>
void launch_dots(const B* V, int64_t ldv, int64_t lds, int nv, const cx<R>* w, int64_t ldw, int64_t n, int nslot,
                 const int* active, c64* partial, int nchunk, c64* out, int ldo, int* done, cudaStream_t st, R vs,
                 const double* vinv, int ldi) {
    // few chunks of few slots: the vectors over blocks too, two at least to each (a block's loop over 50 vectors waits 25
    // times for memory: 14 us on average at 3,700 unknowns, 10 us so), up to three blocks for each of the 152 SMs.  A sum is
    // the same however the vectors are dealt out.
    const int groups = std::max(1, std::min((nv + 1) / 2, 456 / (nchunk * nslot)));
    const int vpb = std::max(2, (ceil_div(nv, groups) + 1) / 2 * 2);
    pdl_launch(dots_kernel<R, B>, dim3(nchunk, nslot, std::max(1, ceil_div(nv, vpb))), DOT_THREADS, 0, st, 
        V, ldv, lds, nv, w, ldw, n, active, partial, nchunk, vpb, vs, vinv, ldi, out, ldo, done);
    GT_LAUNCH_CHECK();
}

// The Hessenberg column j of a slot by one warp: rotate, new rotation, residual estimate, convergence.  An FP64 instruction
// holds its pipe for 64 cycles whatever the number of lanes that take part, so what can be done side by side is: the
// products cs_i h_{i+1} before the chain x_{i+1} = cs_i h_{i+1} - conj(sn_i) x_i, its real and its imaginary part on two
// lanes (a step is two multiply-adds), the rotated entries after it, and the new rotation's norms, quotients and roots one
// to a lane.  Everything it reads is in shared memory or registers before the chain begins.  With the last three done one
// after the other by a lane and the rotations read from memory, the second Gram-Schmidt pass of one column of 3,700
// unknowns took 24.6 us, 22.0 so, and its solve 9.6 and 9.3 ms.
// sm: 4 (MAXV + 1) complex values.
__device__ void givens_column(const GmresState& s, int j, int slot, bool re, double hn, c64* sm) {
    const int lane = threadIdx.x & 31, m = s.m;
    c64* hs = sm;                                        // h_0 .. h_j
    c64* ts = sm + MAXV + 1;                             // cs_i h_{i+1}
    c64* xs = sm + 2 * (MAXV + 1);                       // the chain
    c64* ss = sm + 3 * (MAXV + 1);                       // sn_i
    c64* H = s.H + (int64_t)slot * (m + 1) * m + (int64_t)j * (m + 1);
    const c64* h = s.hvec + (int64_t)slot * s.ldh;
    const c64* h2 = s.h2vec + (int64_t)slot * s.ldh;
    double* cs = s.cs + (int64_t)slot * m;
    c64* sn = s.sn + (int64_t)slot * m;
    c64* g = s.g + (int64_t)slot * (m + 1);
    const c64 gj = g[j];
    const int total = s.its_total[slot] + 1;
    const double eta = s.eta[slot];
    double hnorm2 = 0;
    for (int i = lane; i <= j; i += 32) {
        c64 v = h[i];
        if (re) v += h2[i];
        hs[i] = v;
        if (i < j) ss[i] = sn[i];
        hnorm2 += norm2(v);
    }
    hnorm2 = shfl_sum(hnorm2);
    __syncwarp();
    for (int i = lane; i < j; i += 32) ts[i] = cs[i] * hs[i + 1];
    __syncwarp();
    // lanes 0 and 1: the real and the imaginary part
    double x = lane & 1 ? hs[0].im : hs[0].re;
#pragma unroll 4
    for (int i = 0; i < j; ++i) {
        if (lane < 2) reinterpret_cast<double*>(xs + i)[lane] = x;
        const double o = __shfl_xor_sync(0xffffffffu, x, 1);
        const c64 sv = ss[i];
        const double t = lane & 1 ? ts[i].im : ts[i].re;
        x = __fma_rn(lane & 1 ? sv.im : -sv.im, o, __fma_rn(-sv.re, x, t));
    }
    __syncwarp();
    for (int i = lane; i < j; i += 32) H[i] = cs[i] * xs[i] + ss[i] * hs[i + 1];
    const c64 a = mk<double>(__shfl_sync(0xffffffffu, x, 0), __shfl_sync(0xffffffffu, x, 1));
    // lane 0: |a|, lane 1: |(a, hn)|
    const double nrm = norm3d(a.re, a.im, lane == 1 ? hn : 0.0);
    const double aa = __shfl_sync(0xffffffffu, nrm, 0), rho = __shfl_sync(0xffffffffu, nrm, 1);
    // lane 0: |a| / rho, 1: hn / rho, 2 and 3: a / |a|, 4: 1 / hn
    const double num = lane == 0 ? aa : lane == 1 ? hn : lane == 2 ? a.re : lane == 3 ? a.im : 1.0;
    const double den = lane < 2 ? rho : lane < 4 ? aa : hn;
    const double quo = num / (den != 0.0 ? den : 1.0);
    double c = __shfl_sync(0xffffffffu, quo, 0);
    const double sr = __shfl_sync(0xffffffffu, quo, 1), inv_hn = __shfl_sync(0xffffffffu, quo, 4);
    const c64 ph = mk<double>(__shfl_sync(0xffffffffu, quo, 2), __shfl_sync(0xffffffffu, quo, 3));
    c64 sj = sr * ph, hj = rho * ph;
    if (rho == 0.0) {
        c = 1.0;
        sj = zero<double>();
        hj = a;
    } else if (aa == 0.0) {
        c = 0.0;
        sj = mk<double>(1.0, 0.0);
        hj = mk<double>(hn, 0.0);
    }
    const c64 gn = mk<double>(-1.0, 0.0) * (conj(sj) * gj);
    // lane 0: the residual estimate, lane 1: the column's norm
    const double root = sqrt(lane == 1 ? hnorm2 : norm2(gn));
    const double res = root, hnorm = __shfl_sync(0xffffffffu, root, 1);
    if (lane) return;
    cs[j] = c;
    sn[j] = sj;
    H[j] = hj;
    H[j + 1] = zero<double>();
    g[j + 1] = gn;
    g[j] = c * gj;
    s.it[slot] = j + 1;
    s.its_total[slot] = total;
    const bool breakdown = hn <= 1e-14 * hnorm;
    const double inv = (hn > 0 && !breakdown) ? inv_hn : 0.0;
    s.inv_hn[slot] = inv;
    s.vinv[(int64_t)slot * (m + 1) + j + 1] = inv;
    const bool over = res <= eta || breakdown || j + 1 >= m || total >= s.max_its;
    if (over) s.active[slot] = s.reorth[slot] = 0;       // (no second pass on a later step either)
    if (!over) s.to_go[slot] = res / eta;
}

// w += sign * sum_i h_i V_i (sign -1: Gram-Schmidt; +1: the cycle's combination); partial |w|^2 per chunk of
// UPD_CHUNK elements (nchunk = update_chunks(n)).  The slot's last block finishes: tail 1: |w|^2 to out[slot]; 2: as that,
// for the first Gram-Schmidt pass: decide the second one (DGKS) and, without it, the Hessenberg column; 3: as that, for
// the second pass.
// Four blocks an SM (64 registers): 195.7 ms of updates in a solve of 32 columns of 460,000 unknowns, 207.9 with three.
template <typename R, typename B>
__global__ void __launch_bounds__(DOT_THREADS, 4) update_kernel(const B* __restrict__ V, int64_t ldv, int64_t lds,
                                                             int nv, const c64* __restrict__ h, int ldh,
                                                             cx<R>* __restrict__ w, int64_t ldw, int64_t n,
                                                             const int* __restrict__ active, c64* __restrict__ partial,
                                                             int nchunk, int sign, R vs, const double* __restrict__ vinv, int ldi,
                                                             int tail, c64* __restrict__ out, int* done, GmresState s, int j) {
    pdl_enter();
    __shared__ cx<R> hs[MAXV + 16];
    __shared__ double red[DOT_THREADS / 32];
    __shared__ c64 gv[4 * (MAXV + 1)];
    const int slot = blockIdx.y;
    if (active && !active[slot]) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // UN basis vectors' loads in flight together (FP32 arithmetic; FP64 keeps fewer); the coefficients' last group of UN is
    // filled up with zeros
    constexpr int UN = (sizeof(R) == 4 ? 16 : 4) / UPD_EPT;
    for (int i = tid; i < (nv + UN - 1) / UN * UN; i += DOT_THREADS) {
        c64 v = i < nv ? h[(int64_t)slot * ldh + i] : zero<double>();
        if (vinv && i < nv) v = vinv[(int64_t)slot * ldi + i] * v;
        hs[i] = mk<R>(R(sign * v.re * vs), R(sign * v.im * vs));
    }
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * UPD_CHUNK;
    cx<R> acc[UPD_EPT];
#pragma unroll
    for (int e = 0; e < UPD_EPT; ++e) {
        int64_t q = base + e * DOT_THREADS + tid;
        acc[e] = q < n ? w[(int64_t)slot * ldw + q] : zero<R>();
    }
    const B* Vs = V + (int64_t)slot * lds;
    for (int i = 0; i < nv; i += UN) {
        cx<R> v[UN][UPD_EPT];
#pragma unroll
        for (int u = 0; u < UN; ++u)
#pragma unroll
            for (int e = 0; e < UPD_EPT; ++e) {
                const int64_t q = base + e * DOT_THREADS + tid;
                v[u][e] = i + u < nv && q < n ? bload(Vs + (int64_t)(i + u) * ldv + q) : zero<R>();
            }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const cx<R> hi = hs[i + u];
#pragma unroll
            for (int e = 0; e < UPD_EPT; ++e) acc[e] += hi * v[u][e];
        }
    }
    R nrm = 0;
#pragma unroll
    for (int e = 0; e < UPD_EPT; ++e) {
        int64_t q = base + e * DOT_THREADS + tid;
        if (q < n) {
            w[(int64_t)slot * ldw + q] = acc[e];
            nrm += norm2(acc[e]);
        }
    }
    nrm = shfl_sum(nrm);
    if (lane == 0) red[warp] = nrm;
    __syncthreads();
    if (!tail) return;
    if (tid == 0) {
        double t = 0;
        for (int q = 0; q < DOT_THREADS / 32; ++q) t += red[q];
        partial[(int64_t)slot * nchunk + blockIdx.x] = mk<double>(t, 0.0);
    }
    if (!last_of_slot(done, slot, nchunk)) return;
    double t = 0;
    for (int c = tid; c < nchunk; c += DOT_THREADS) t += __ldcg(&partial[(int64_t)slot * nchunk + c].re);
    t = shfl_sum(t);
    if (lane == 0) red[warp] = t;
    __syncthreads();
    if (warp) return;
    t = 0;
    for (int q = 0; q < DOT_THREADS / 32; ++q) t += red[q];
    if (lane == 0) out[slot] = mk<double>(t, 0.0);
    if (tail == 1) return;
    bool re = tail == 3;
    if (tail == 2) {
        re = sqrt(t) < s.reorth_ratio * sqrt(s.hvec[(int64_t)slot * s.ldh + j + 1].re);
        if (lane == 0) s.reorth[slot] = re;
        if (re) return;
    }
    givens_column(s, j, slot, re, sqrt(t), gv);
}

template <typename R, typename B>
static void update_launch(const B* V, int64_t ldv, int64_t lds, int nv, const c64* h, int ldh, cx<R>* w, int64_t ldw, int64_t n,
                          int nslot, const int* active, c64* partial, int sign, R vs, const double* vinv, int ldi, int tail, c64* out, int* done,
                          const GmresState& s, int j, cudaStream_t st) {
    const int nchunk = update_chunks(n);
    pdl_launch(update_kernel<R, B>, dim3(nchunk, nslot), DOT_THREADS, 0, st, V, ldv, lds, nv, h, ldh, w, ldw, n, active,
                                                                      partial, nchunk, sign, vs, vinv, ldi, tail, out, done, s, j);
    GT_LAUNCH_CHECK();
}

template <typename R, typename B>
void launch_update(const B* V, int64_t ldv, int64_t lds, int nv, const c64* h, int ldh, cx<R>* w, int64_t ldw,
                   int64_t n, int nslot, const int* active, c64* partial, c64* nrm2, int* done, int sign, cudaStream_t st, R vs,
                   const double* vinv, int ldi) {
    update_launch<R, B>(V, ldv, lds, nv, h, ldh, w, ldw, n, nslot, active, partial, sign, vs, vinv, ldi, nrm2 ? 1 : 0, nrm2, done,
                        GmresState{}, 0, st);
}

template <typename R, typename B>
void launch_gram_schmidt(const B* V, int64_t ldv, int64_t lds, int pass, cx<R>* w, int64_t ldw, int64_t n, c64* partial, int* done,
                         const GmresState& s, int j, cudaStream_t st, R vs) {
    update_launch<R, B>(V, ldv, lds, j + 1, pass == 2 ? s.h2vec : s.hvec, s.ldh, w, ldw, n, s.nslot,
                        pass == 2 ? s.reorth : s.active, partial, -1, vs, std::is_same<B, cx<R>>::value ? s.vinv : nullptr, s.m + 1,
                        pass + 1, pass == 2 ? s.hn2b : s.hn2, done, s, j, st);
}

template void launch_dots<float, c32>(const c32*, int64_t, int64_t, int, const c32*, int64_t, int64_t, int, const int*, c64*, int, c64*, int, int*, cudaStream_t, float, const double*, int);
template void launch_dots<float, h16c>(const h16c*, int64_t, int64_t, int, const c32*, int64_t, int64_t, int, const int*, c64*, int, c64*, int, int*, cudaStream_t, float, const double*, int);
template void launch_dots<double, c64>(const c64*, int64_t, int64_t, int, const c64*, int64_t, int64_t, int, const int*, c64*, int, c64*, int, int*, cudaStream_t, double, const double*, int);
template void launch_update<float, c32>(const c32*, int64_t, int64_t, int, const c64*, int, c32*, int64_t, int64_t, int, const int*, c64*, c64*, int*, int, cudaStream_t, float, const double*, int);
template void launch_update<float, h16c>(const h16c*, int64_t, int64_t, int, const c64*, int, c32*, int64_t, int64_t, int, const int*, c64*, c64*, int*, int, cudaStream_t, float, const double*, int);
template void launch_update<double, c64>(const c64*, int64_t, int64_t, int, const c64*, int, c64*, int64_t, int64_t, int, const int*, c64*, c64*, int*, int, cudaStream_t, double, const double*, int);

template void launch_gram_schmidt<float, c32>(const c32*, int64_t, int64_t, int, c32*, int64_t, int64_t, c64*, int*, const GmresState&, int, cudaStream_t, float);
template void launch_gram_schmidt<float, h16c>(const h16c*, int64_t, int64_t, int, c32*, int64_t, int64_t, c64*, int*, const GmresState&, int, cudaStream_t, float);
template void launch_gram_schmidt<double, c64>(const c64*, int64_t, int64_t, int, c64*, int64_t, int64_t, c64*, int*, const GmresState&, int, cudaStream_t, double);

// ------------------------------------------------------------------------------------------ per-slot scalars
// store v (a basis vector, unscaled) at p[q]; with a narrower basis type also the stored value, unscaled,
// to vc[q] (the vector the next product is applied to)
template <typename R, typename B>
__device__ __forceinline__ void put_basis(const GmresStateT<R, B>& s, B* p, cx<R>* vc, int64_t q, cx<R> v) {
    if constexpr (std::is_same<B, cx<R>>::value) {
        p[q] = v;
    } else {
        bstore(p + q, s.scale * v);
        vc[q] = (R(1) / s.scale) * bload(p + q);
    }
}

// the next vector of a narrow basis: w normalised and rounded
template <typename R, typename B>
__global__ void scale_kernel(GmresStateT<R, B> s, int j, int64_t n) {
    pdl_enter();
    const int slot = blockIdx.y;
    if (!s.active[slot]) return;
    const R f = R(s.inv_hn[slot]);
    const cx<R>* w = s.w + (int64_t)slot * s.ldv;
    B* v = s.V + (int64_t)slot * s.lds + (int64_t)(j + 1) * s.ldv;
    cx<R>* vc = s.vcur ? s.vcur + (int64_t)slot * s.ldv : nullptr;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        put_basis(s, v, vc, q, f * w[q]);
}

// y = R^-1 g over the slot's k = it columns (back substitution, FP64), a warp per slot, column by column: the divisions
// are made beforehand, side by side, and each column is taken off the rest of g by all lanes.  By one thread, row by row,
// it took 0.1 ms at 50 steps, every load waited for.
__global__ void __launch_bounds__(32) hsolve_kernel(GmresState s) {
    __shared__ c64 gs[MAXV], di[MAXV];
    const int slot = blockIdx.x, lane = threadIdx.x, m = s.m, k = s.it[slot];
    const c64* H = s.H + (int64_t)slot * (m + 1) * m;
    const c64* g = s.g + (int64_t)slot * (m + 1);
    c64* y = s.y + (int64_t)slot * s.ldh;
    for (int i = lane; i < k; i += 32) {
        const c64 d = H[(int64_t)i * (m + 1) + i];
        di[i] = norm2(d) > 0 ? cdiv(mk<double>(1.0, 0.0), d) : zero<double>();
        gs[i] = g[i];
    }
    __syncwarp();
    for (int q = k - 1; q >= 0; --q) {
        const c64 v = gs[q] * di[q];
        if (lane == 0) y[q] = v;
        const c64* h = H + (int64_t)q * (m + 1);
        for (int i = lane; i < q; i += 32) gs[i] -= h[i] * v;
        __syncwarp();
    }
    for (int i = k + lane; i < m; i += 32) y[i] = zero<double>();
}

// a slot's cycle starts from r / rho: V_0 = r / rho, g = (1, 0, ...), rotations cleared
template <typename R, typename B>
__global__ void init_cycle_kernel(GmresStateT<R, B> s, const c64* __restrict__ r, int64_t ldr, const int* __restrict__ slot_col,
                                  const double* __restrict__ rho, int64_t n) {
    const int slot = blockIdx.y;
    const int col = slot_col[slot];
    const double inv = rho[col] > 0 ? 1.0 / rho[col] : 0.0;
    B* v = s.V + (int64_t)slot * s.lds;
    cx<R>* vc = s.vcur ? s.vcur + (int64_t)slot * s.ldv : nullptr;
    const c64* rc = r + (int64_t)col * ldr;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        put_basis(s, v, vc, q, cvt<R>(inv * rc[q]));
}

__global__ void init_state_kernel(GmresState s, const int* __restrict__ slot_col, const double* __restrict__ rho,
                                  const double* __restrict__ bnorm, double tol, double inner_tol) {
    int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= s.nslot) return;
    int col = slot_col[slot];
    c64* g = s.g + (int64_t)slot * (s.m + 1);
    g[0] = mk<double>(1.0, 0.0);
    for (int i = 1; i <= s.m; ++i) g[i] = zero<double>();
    s.it[slot] = 0;
    s.active[slot] = 1;
    // the cycle's first vector is stored normalised; no later one is weighted before it is made
    s.inv_hn[slot] = 1.0;
    for (int i = 0; i <= s.m; ++i) s.vinv[(int64_t)slot * (s.m + 1) + i] = i ? 0.0 : 1.0;
    // the cycle needs to reach the outer tolerance at most (half of it, as a margin), never below inner_tol
    double need = rho[col] > 0 ? 0.5 * tol * bnorm[col] / rho[col] : 1.0;
    s.eta[slot] = fmax(inner_tol, need);
}

__global__ void sqrt_norms_kernel(const c64* __restrict__ nrm2, int ld, int n, double* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = sqrt(nrm2[(int64_t)i * ld].re);
}

template <typename R>
__global__ void to64_kernel(c64* __restrict__ dst, int64_t ldd, const cx<R>* __restrict__ src, int64_t lds,
                            const int* __restrict__ slot_col, int64_t n) {
    const int s = blockIdx.y;
    c64* d = dst + (int64_t)slot_col[s] * ldd;
    const cx<R>* x = src + (int64_t)s * lds;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        d[q] = cvt<double>(x[q]);
}

// dst slot c = src slot c converted to D, for the listed slots (all nslot when list is null): the FP32 inner
// solve's vectors into and out of an FP64 preconditioner apply
template <typename D, typename S>
__global__ void recast_kernel(cx<D>* __restrict__ dst, int64_t ldd, const cx<S>* __restrict__ src, int64_t lds,
                              const int* __restrict__ list, int64_t n, const double* __restrict__ scale) {
    pdl_enter();
    const int c = list ? list[blockIdx.y] : (int)blockIdx.y;
    const double f = scale ? scale[c] : 1.0;
    cx<D>* d = dst + (int64_t)c * ldd;
    const cx<S>* x = src + (int64_t)c * lds;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        d[q] = cvt<D>(f * cvt<double>(x[q]));
}

__global__ void gcr_scale_kernel(c64* __restrict__ p, c64* __restrict__ q, int64_t ld, const c64* __restrict__ nu2,
                                 const int* __restrict__ active, int64_t n) {
    const int c = blockIdx.y;
    if (active && !active[c]) return;
    const double nu = sqrt(nu2[c].re);
    const double f = nu > 0 ? 1.0 / nu : 0.0;
    c64* pc = p + (int64_t)c * ld;
    c64* qc = q + (int64_t)c * ld;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        pc[i] = f * pc[i];
        qc[i] = f * qc[i];
    }
}

// ------------------------------------------------------------------------------------------ launchers
template <typename R>
void launch_to64(c64* dst, int64_t ldd, const cx<R>* src, int64_t lds, const int* slot_col, int64_t n, int nslot,
                 cudaStream_t st) {
    int blocks = (int)std::min<int64_t>((n + 255) / 256, 1024);
    to64_kernel<R><<<dim3(blocks, nslot), 256, 0, st>>>(dst, ldd, src, lds, slot_col, n);
    GT_LAUNCH_CHECK();
}
template void launch_to64<float>(c64*, int64_t, const c32*, int64_t, const int*, int64_t, int, cudaStream_t);
template void launch_to64<double>(c64*, int64_t, const c64*, int64_t, const int*, int64_t, int, cudaStream_t);

template <typename D, typename S>
void launch_recast(cx<D>* dst, int64_t ldd, const cx<S>* src, int64_t lds, const int* list, int64_t n, int nslot,
                   const double* scale, cudaStream_t st) {
    if (nslot <= 0) return;
    int blocks = (int)std::min<int64_t>((n + 255) / 256, 1024);
    pdl_launch(recast_kernel<D, S>, dim3(blocks, nslot), 256, 0, st, dst, ldd, src, lds, list, n, scale);
    GT_LAUNCH_CHECK();
}
template void launch_recast<double, float>(c64*, int64_t, const c32*, int64_t, const int*, int64_t, int, const double*, cudaStream_t);
template void launch_recast<float, double>(c32*, int64_t, const c64*, int64_t, const int*, int64_t, int, const double*, cudaStream_t);

void launch_gcr_scale(c64* p, c64* q, int64_t ld, const c64* nu2, const int* active, int64_t n, int ncol,
                      cudaStream_t st) {
    int blocks = (int)std::min<int64_t>((n + 255) / 256, 1024);
    gcr_scale_kernel<<<dim3(blocks, ncol), 256, 0, st>>>(p, q, ld, nu2, active, n);
    GT_LAUNCH_CHECK();
}

template <typename R, typename B>
void launch_scale(const GmresStateT<R, B>& s, int j, int64_t n, cudaStream_t st) {
    int blocks = (int)std::min<int64_t>((n + 255) / 256, 1024);
    pdl_launch(scale_kernel<R, B>, dim3(blocks, s.nslot), 256, 0, st, s, j, n);
    GT_LAUNCH_CHECK();
}
void launch_hsolve(const GmresState& s, cudaStream_t st) {
    hsolve_kernel<<<s.nslot, 32, 0, st>>>(s);
    GT_LAUNCH_CHECK();
}
template <typename R, typename B>
void launch_init_cycle(const GmresStateT<R, B>& s, const c64* r, int64_t ldr, const int* slot_col, const double* rho,
                       int64_t n, cudaStream_t st) {
    int blocks = (int)std::min<int64_t>((n + 255) / 256, 1024);
    init_cycle_kernel<R, B><<<dim3(blocks, s.nslot), 256, 0, st>>>(s, r, ldr, slot_col, rho, n);
    GT_LAUNCH_CHECK();
}
void launch_init_state(const GmresState& s, const int* slot_col, const double* rho, const double* bnorm, double tol,
                       double inner_tol, cudaStream_t st) {
    init_state_kernel<<<ceil_div(s.nslot, 64), 64, 0, st>>>(s, slot_col, rho, bnorm, tol, inner_tol);
    GT_LAUNCH_CHECK();
}
__global__ void sqrt_norms_active_kernel(const c64* __restrict__ nrm2, int ld, int n, const int* __restrict__ active,
                                         double* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && active[i]) out[i] = sqrt(nrm2[(int64_t)i * ld].re);
}

void launch_sqrt_norms_active(const c64* nrm2, int ld, int n, const int* active, double* out, cudaStream_t st) {
    sqrt_norms_active_kernel<<<ceil_div(n, 128), 128, 0, st>>>(nrm2, ld, n, active, out);
    GT_LAUNCH_CHECK();
}

void launch_sqrt_norms(const c64* nrm2, int ld, int n, double* out, cudaStream_t st) {
    sqrt_norms_kernel<<<ceil_div(n, 128), 128, 0, st>>>(nrm2, ld, n, out);
    GT_LAUNCH_CHECK();
}

template void launch_scale<float, h16c>(const GmresStateT<float, h16c>&, int, int64_t, cudaStream_t);
template void launch_init_cycle<float, c32>(const GmresStateT<float, c32>&, const c64*, int64_t, const int*, const double*, int64_t, cudaStream_t);
template void launch_init_cycle<float, h16c>(const GmresStateT<float, h16c>&, const c64*, int64_t, const int*, const double*, int64_t, cudaStream_t);
template void launch_init_cycle<double, c64>(const GmresStateT<double, c64>&, const c64*, int64_t, const int*, const double*, int64_t, cudaStream_t);

}  // namespace gt
