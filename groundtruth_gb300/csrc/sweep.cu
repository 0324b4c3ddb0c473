// The FP32 triangular sweeps of the preconditioner (the solves with the factorised Schur complement, peec.py:3071)
// as one kernel: every front of the elimination tree, forward and backward, and every column group in one launch.
//
// After the factorisation a front's panel is P = [Linv_own; -L_bnd Linv_own] (factor.cu), so its solves are two dense
// products without a sequential chain:
//     forward   out = P w_own: own rows z_own = dinv * out, boundary rows (children's updates + out) go up
//     backward  y_own = P^T [z_own; y_bnd]
// A task is one output tile of one front: up to 128 rows of the forward product or columns of the backward one, for a
// group of up to 8 columns that share the operator.  The FP32 panels are stored tile by tile in the order the tasks
// read them, [inner index][outputs], the zeros above the own block's diagonal left out at tile granularity, so that a
// task's panel is one contiguous run.
//
// Why one launch: a level at a time, the top of the tree (one to a few fronts per level) left the GPU idle between
// 26-40 dependent launches of ~20 us each; the slotted pair at 256 x 256 took 1.08 ms per application with 32 columns at four
// frequencies, where its panels are 0.15 ms of HBM time.  Here blocks draw tickets from a counter, and tickets are numbered so that
// a task's inputs always have smaller ones: leaves to root, then root to leaves.  A block waits (bounded) on a counter
// of its inputs' finished tiles; whoever holds the smallest unfinished ticket never waits, so the kernel finishes
// however many of its blocks are resident.  A block's fifth warp runs ahead of the other four: it takes the next
// ticket and brings its panel run into a ring of shared-memory stages by bulk copies while the present task waits
// for its inputs or computes, so the panel streams at HBM rate through the tree's dependent steps.
//
// The vectors between tasks (update vectors, z, y) are interleaved by column group, a row's columns side by side as
// pairs (re0 re1 im0 im1), which the gathers read as 16-byte pieces and the packed FP32 FMAs (two per instruction)
// take as they are.
//
// A column's arithmetic is set by the fronts alone (tile, stage and segment sizes), never by the other columns.
#include "kernels.h"

#include <algorithm>
#include <cstdlib>
#include <map>
#include <mutex>

namespace gt {

constexpr int SWT = 128;               // consumer threads
constexpr int SWW = SWT / 32;
constexpr int SW_BLOCK = SWT + 32;     // and the producer warp
constexpr int SW_STAGES = 2;
constexpr int SW_STAGE_ENT = 1792;     // panel entries per stage (14 KB)
constexpr int SW_XROWS = 256;          // inner rows staged at once (16 KB at 8 columns)
constexpr int SW_HMAX = 128;
constexpr long long SW_WAIT_CYCLES = 4000000000ll;       // two seconds
constexpr long long SW_TEST_WAIT_CYCLES = 2000000ll;     // a millisecond, where a test makes a wait run out
constexpr uint32_t SW_POLLS = 1u << 28;

struct SwDesc {                        // a task, written by the producer beside its first ring stage
    int f_dir;                         // 0 forward, 1 backward, -1 no more work
    int g;                             // column group
    int step;                          // inner indices per stage
    SwTask t;
};

struct alignas(16) SwShared {
    float2 ring[SW_STAGES][SW_STAGE_ENT];
    float4 x[SW_XROWS * 4];            // inner rows [row][pair]; then the partial sums [seg][output][pair]
    float4 ext[SW_HMAX * 4];           // per output entry, its thread's own: forward, the pivot's reciprocal of an own row or
                                       // the updates so far of a boundary row; backward, the dense node
    int xrow[2][SW_XROWS];             // staged rows' sources: forward, the first two children's update rows; backward [0]
    int hrow[2][SW_HMAX];              // forward: the outputs' sources
    SwDesc desc[SW_STAGES];
    uint64_t full[SW_STAGES], empty[SW_STAGES];
    int quit;                          // a consumer has not got the next task: the block leaves
};
static_assert(SW_XROWS * 4 >= 2 * SWT * 4, "the partial sums take the staged rows' place");

__device__ __forceinline__ uint32_t sw_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool sw_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Waits are bounded.  One that gives up is counted in the call's own word (gave_up), which ends the call's other waits, and
// the host reports GT_TIMEOUT.  What follows a wait that gave up stays in bounds and leads to the launch's end:
//   for another tile's results (sw_wait_count)   the tile is made from what is there
//   for a task's first stage (full)              its descriptor may not be there: sm.quit, which all of the block's consumers
//                                                look at behind the task's second barrier, and leave
//   for a further stage of a task (full)         the tile is made from what is there, the number of its stages being the
//                                                task's; the consumers leave as they do without the next descriptor, which is
//                                                not looked for: a thread that went on without a stage may be ahead by the
//                                                whole ring, where a barrier's parity takes an old stage for the one it wants
//   for a stage to be read (empty)               the producer stops, as it does before a stage whose last copy is not
//                                                complete, and waits once more for its copies in flight before it leaves
__device__ __noinline__ void sw_gave_up(unsigned int* gave_up) { atomicAdd(gave_up, 1u); }
__device__ __noinline__ bool sw_wait_slow(uint32_t bar, uint32_t parity, unsigned int* gave_up, long long limit) {
    const long long t0 = clock64();
    for (uint32_t it = 0; it < SW_POLLS; ++it) {
        if (sw_try(bar, parity)) return true;
        if ((it & 1023) == 1023 && *(volatile unsigned int*)gave_up) return false;
        if (clock64() - t0 > 2 * limit) break;
    }
    sw_gave_up(gave_up);
    return false;
}
__device__ __forceinline__ bool sw_wait_bar(uint64_t* b, uint32_t parity, unsigned int* gave_up, long long limit) {
    const uint32_t bar = sw_smem(b);
    return sw_try(bar, parity) || sw_wait_slow(bar, parity, gave_up, limit);
}
// a wait without a count and whatever the word says: the copies in flight of a block that leaves
__device__ __noinline__ void sw_drain(uint64_t* b, uint32_t parity, long long limit) {
    const uint32_t bar = sw_smem(b);
    const long long t0 = clock64();
    for (uint32_t it = 0; it < SW_POLLS; ++it)
        if (sw_try(bar, parity) || clock64() - t0 > limit) return;
}
__device__ __forceinline__ int sw_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void sw_wait_count(const int* p, int need, unsigned int* gave_up, long long limit) {
    if (sw_acquire(p) >= need) return;
    const long long t0 = clock64();
    for (uint32_t it = 0; it < SW_POLLS; ++it) {
        if (sw_acquire(p) >= need) return;
        if ((it & 63) == 63) {
            if (*(volatile unsigned int*)gave_up) return;        // someone of this call gave up already
            if (clock64() - t0 > limit) break;
        }
        __nanosleep(32);
    }
    sw_gave_up(gave_up);
}
__device__ __forceinline__ void sw_sync() { asm volatile("bar.sync 1, %0;" ::"n"(SWT) : "memory"); }

// two packed FP32 FMAs: each half of acc += a b
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t both(float a) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(a));
    return v;
}
__device__ __forceinline__ float4 halves(uint64_t re, uint64_t im) {
    float4 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(re));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.z), "=f"(v.w) : "l"(im));
    return v;
}
__device__ __forceinline__ void add4(float4& a, float4 b) {
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
}

// (re, im) of NP column pairs += (pr + j pi) x
template <int NP>
__device__ __forceinline__ void mac_row(uint64_t* re, uint64_t* im, float pr, float pi, const ulonglong2* X) {
    const uint64_t r2 = both(pr), i2 = both(pi), n2 = both(-pi);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const ulonglong2 x = X[p];                       // the pair's real parts, its imaginary parts
        fma2(re[p], r2, x.x);
        fma2(im[p], r2, x.y);
        fma2(re[p], n2, x.y);
        fma2(im[p], i2, x.x);
    }
}

struct SwArgs {
    const SwTask* tasks;               // nft forward tasks, then the backward ones
    int nft;
    int nsrc;
    int64_t src_rows;
    const int* src;                    // [nsrc][src_rows] update-vector rows added into a front's rows (-1: none)
    const int* bidx;                   // boundary rows' factor indices
    const int64_t* iperm;
    int64_t nfac, nvec, nnode, ptotal;
    const float2* pf;                  // [op][ptotal] forward tiles
    const float2* pb;                  // [op][ptotal] backward tiles
    const float2* dinv;                // [op][nfac]
    const float2* s;                   // [slot][nfac] right-hand sides, factor order
    float4* z;                         // interleaved [group][nfac][pairs]
    float4* y;
    float4* u;                         // interleaved [group][nvec][pairs]
    float2* sd;                        // [slot][nnode] solutions, node order
    Groups G;
    int* cnt;                          // [counter][ngroup] finished tiles
    int* ticket;                       // this launch's ticket counter
    int t0, t1;                        // tickets of this launch
    unsigned int* gave_up;             // the call's count of waits that ran out
    long long wait;                    // the limit of the waits for tiles, in clock cycles; those for stages have twice as long
    int surplus, missing;              // 0, except when a test makes waits run out: tiles that nobody finishes, bytes of a stage
                                       // that no copy brings
};

// where the partial sum of row pair row2, entry e = row * NP + pair, stands: the entries of a row pair permuted by the row
// pair, so that the warp that stores one entry of 32 row pairs, and the one that reads them in order, meet all banks
template <int NP>
__device__ __forceinline__ int sw_slot(int row2, int e) {
    return row2 * 2 * NP + (e ^ ((row2 / (4 / NP)) & (2 * NP - 1)));
}

// The update rows that the first two children have for the front's rows row0 .. row0 + n, into rows (a barrier follows).
__device__ __forceinline__ void sw_sources(const SwArgs& A, int nsrc, int64_t row0, int n, int (*rows)[SW_XROWS], int tid) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < SW_XROWS / SWT; ++i) {
            const int r = tid + i * SWT;
            if (r < n) rows[c][r] = c < nsrc ? A.src[c * A.src_rows + row0 + r] : -1;
        }
}

// out += the children's updates of n rows (from row `from` on), in the children's order: the thread's entries tid + i SWT, i < N, each a column
// pair p of row rt + i RS.  Two entries' values of two children are in flight together; four spill registers, which
// took an application with 128 columns 1.35 times as long.
template <int NP, int N>
__device__ __forceinline__ void sw_add_children(const SwArgs& A, int nsrc, int64_t row0, int n, int from, const int* rows0,
                                                const int* rows1, const float4* u, float4* out, int tid) {
    constexpr int RS = SWT / NP, B = N < 2 ? N : 2;
    const int p = tid % NP, rt = tid / NP;
#pragma unroll 1
    for (int i0 = 0; i0 < N; i0 += B) {
        if (rt + i0 * RS >= n) break;
        int e[2][B];
        float4 a[B], b[2][B];
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int r = rt + (i0 + i) * RS;
            e[0][i] = r < n ? rows0[r] : -1;
            e[1][i] = r < n ? rows1[r] : -1;
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < B; ++i)
                b[c][i] = e[c][i] >= 0 ? __ldcg(u + (int64_t)e[c][i] * NP + p) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int r = rt + (i0 + i) * RS;
            if (r >= n) continue;
            a[i] = out[tid + (i0 + i) * SWT];
            if (e[0][i] >= 0) add4(a[i], b[0][i]);
            if (e[1][i] >= 0) add4(a[i], b[1][i]);
#pragma unroll 1
            for (int c = 2; c < nsrc; ++c) {             // a front with more than two children
                const int f = r >= from ? A.src[c * A.src_rows + row0 + r] : -1;
                if (f >= 0) add4(a[i], __ldcg(u + (int64_t)f * NP + p));
            }
            out[tid + (i0 + i) * SWT] = a[i];
        }
    }
}

// the backward sweep's inner rows k .. k + n into sm.x: own rows from z, boundary rows from y, the row's index from rows
template <int NP, int N>
__device__ __forceinline__ void sw_stage_back(const float4* z, const float4* y, int n, int own, const int* rows, float4* x, int tid) {
    constexpr int RS = SWT / NP;
    const int p = tid % NP, rt = tid / NP;
    constexpr int B = N < 4 ? N : 4;
#pragma unroll 1
    for (int i0 = 0; i0 < N; i0 += B) {
        if (rt + i0 * RS >= n) break;
        float4 a[B];
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const int r = rt + (i0 + i) * RS;
            a[i] = r < n ? __ldcg((r < own ? z : y) + (int64_t)rows[r] * NP + p) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < B; ++i)
            if (rt + (i0 + i) * RS < n) x[tid + (i0 + i) * SWT] = a[i];
    }
}

// forward: the right-hand sides of n rows (s: the first one's in slot 0; c0, c1: the pair's slots or -1) into x
template <int NP, int N>
__device__ __forceinline__ void sw_stage_own(const float2* s, int64_t nfac, int c0, int c1, int n, float4* x, int tid) {
    constexpr int RS = SWT / NP;
    const int rt = tid / NP;
    const float2 none = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int i = 0; i < N; ++i) {
        const int r = rt + i * RS;
        if (r >= n) break;
        const float2 a0 = c0 >= 0 ? s[c0 * nfac + r] : none, a1 = c1 >= 0 ? s[c1 * nfac + r] : none;
        x[tid + i * SWT] = make_float4(a0.x, a1.x, a0.y, a1.y);
    }
}

// backward: where the inner rows k .. k + n stand, own rows in z, boundary rows in y
__device__ __forceinline__ void sw_back_rows(const int* bidx, int own0, int nown, int k, int n, int* rows, int tid) {
#pragma unroll
    for (int i = 0; i < SW_XROWS / SWT; ++i) {
        const int r = tid + i * SWT, row = k + r;
        if (r < n) rows[r] = row < nown ? own0 + row : bidx[row - nown];
    }
}

// false: one of the consumers did not get here with the task.  bad: this thread went on without a stage
template <int NP>
__device__ bool sw_task(const SwArgs& A, SwShared& sm, uint32_t& it, const SwDesc& d0, bool& bad) {
    const int tid = threadIdx.x;
    const SwTask t = d0.t;
    const int dir = d0.f_dir, g = d0.g, step = d0.step, ng = A.G.ngroup;
    const int* gs = A.G.gslot + A.G.gptr[g];
    const int gc = A.G.gptr[g + 1] - A.G.gptr[g];
    const int64_t gb = A.G.pair0[g];                     // column pairs before this group's
    float4* __restrict__ z = A.z + gb * A.nfac;
    float4* __restrict__ y = A.y + gb * A.nfac;
    float4* __restrict__ u = A.u + gb * A.nvec;
    const int h = t.h, hp = (h + 1) & ~1;
    const int np2 = hp >> 1;                             // pairs of outputs
    const int nseg = SWT / np2;
    const int seg = tid / np2, row2 = tid - seg * np2;
    const bool act = seg < nseg;
    // A thread's entries (of the staged rows and of the outputs) are one column pair of every RS-th row.  All that does not
    // depend on other tasks is fetched before their results are waited for: the rows' sources, the right-hand sides, what
    // the outputs need besides the product.  A tile's time is in these chains of loads (row index, then value), not in its
    // product: fetched one entry after the other, after the wait, they made an application 708 us with 32 columns (529
    // now), 2316 with 128 (1695), 393 with 6 on the stack (314), 77 and 56 with one column on small planes (49 and 38).
    constexpr int RS = SWT / NP, XE = SW_XROWS / RS, HE = SW_HMAX / RS;
    const int p = tid % NP, rt = tid / NP;
    const int c0 = 2 * p < gc ? gs[2 * p] : -1, c1 = 2 * p + 1 < gc ? gs[2 * p + 1] : -1;
    const int nsrc = t.need > 0 ? A.nsrc : 0;            // (forward: a front without children waits for nobody)
    const int lo = min(h, max(0, t.nown - t.r0));        // forward: the tile's first boundary row
    int xbeg = t.k0, xend = min(t.k1, t.k0 + SW_XROWS);
    if (dir == 0) {
        const int64_t op = A.G.op[g];
        if (nsrc) {
            sw_sources(A, nsrc, t.goff + t.k0, xend - xbeg, sm.xrow, tid);
#pragma unroll
            for (int c = 0; c < 2; ++c)
                if (tid < h) sm.hrow[c][tid] = tid >= lo && c < nsrc ? A.src[c * A.src_rows + t.goff + t.r0 + tid] : -1;
        }
        sw_stage_own<NP, XE>(A.s + t.own0 + t.k0, A.nfac, c0, c1, xend - xbeg, sm.x, tid);
#pragma unroll
        for (int i = 0; i < HE; ++i) {
            const int r = rt + i * RS;
            const float2 d = r < lo ? A.dinv[op * A.nfac + t.own0 + t.r0 + r] : make_float2(0.f, 0.f);
            sm.ext[tid + i * SWT] = make_float4(d.x, d.y, 0.f, 0.f);
        }
        if (nsrc) {
            if (tid == 0) sw_wait_count(A.cnt + (int64_t)t.dep * ng + g, t.need + A.surplus, A.gave_up, A.wait);
            sw_sync();
            sw_add_children<NP, HE>(A, nsrc, t.goff + t.r0, h, lo, sm.hrow[0], sm.hrow[1], u, sm.ext, tid);
            sw_add_children<NP, XE>(A, nsrc, t.goff + t.k0, xend - xbeg, 0, sm.xrow[0], sm.xrow[1], u, sm.x, tid);
        } else {
            sw_sync();
        }
    } else {
        sw_back_rows(A.bidx + t.goff, t.own0, t.nown, xbeg, xend - xbeg, sm.xrow[0], tid);
#pragma unroll
        for (int i = 0; i < HE; ++i)
            if (rt + i * RS < h) sm.ext[tid + i * SWT].x = __int_as_float((int)A.iperm[t.own0 + t.r0 + rt + i * RS]);
        if (tid == 0 && t.need > 0) sw_wait_count(A.cnt + (int64_t)t.dep * ng + g, t.need + A.surplus, A.gave_up, A.wait);
        sw_sync();
        sw_stage_back<NP, XE>(z, y, xend - xbeg, t.nown - xbeg, sm.xrow[0], sm.x, tid);
    }
    const int quit = *(const volatile int*)&sm.quit;     // (set before the first barrier, or not at all)
    sw_sync();
    if (quit) return false;
    uint64_t re[2][NP], im[2][NP];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int p = 0; p < NP; ++p) re[r][p] = im[r][p] = 0;
    int ka = t.k0;
    do {
        const int slot = it % SW_STAGES;
        bad |= !sw_wait_bar(&sm.full[slot], (it / SW_STAGES) & 1, A.gave_up, A.wait);
        const int kb = min(t.k1, ka + step);
        const float2* ring = sm.ring[slot];
        for (int k = ka; k < kb;) {
            if (k >= xend) {
                sw_sync();                               // the rows staged before have been read
                xbeg = k;
                xend = min(t.k1, k + SW_XROWS);
                if (dir == 0) {
                    if (nsrc) sw_sources(A, nsrc, t.goff + k, xend - k, sm.xrow, tid);
                    sw_stage_own<NP, XE>(A.s + t.own0 + k, A.nfac, c0, c1, xend - k, sm.x, tid);
                    if (nsrc) {
                        sw_sync();
                        sw_add_children<NP, XE>(A, nsrc, t.goff + k, xend - k, 0, sm.xrow[0], sm.xrow[1], u, sm.x, tid);
                    }
                } else {
                    sw_back_rows(A.bidx + t.goff, t.own0, t.nown, k, xend - k, sm.xrow[0], tid);
                    sw_sync();
                    sw_stage_back<NP, XE>(z, y, xend - k, t.nown - k, sm.xrow[0], sm.x, tid);
                }
                sw_sync();
            }
            const int e = min(kb, xend);
            if (act) {
                const float4* P = reinterpret_cast<const float4*>(ring) + (k - ka + seg) * np2 + row2;
                const ulonglong2* X = reinterpret_cast<const ulonglong2*>(sm.x) + (k - xbeg + seg) * NP;
#pragma unroll 1
                for (int q = k + seg; q < e; q += nseg, P += nseg * np2, X += nseg * NP) {
                    const float4 a = *P;                  // outputs 2 row2, 2 row2 + 1
                    mac_row<NP>(re[0], im[0], a.x, a.y, X);
                    mac_row<NP>(re[1], im[1], a.z, a.w, X);
                }
            }
            k = e;
        }
        ++it;
        ka = kb;
        __syncwarp();
        if ((tid & 31) == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sw_smem(&sm.empty[slot])) : "memory");
    } while (ka < t.k1);
    // the segments' partial sums meet in the staged rows' place
    sw_sync();
    if (act) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int p = 0; p < NP; ++p) sm.x[seg * hp * NP + sw_slot<NP>(row2, r * NP + p)] = halves(re[r][p], im[r][p]);
    }
    sw_sync();
#pragma unroll
    for (int i = 0; i < HE; ++i) {
        const int r = rt + i * RS, q = tid + i * SWT, row = t.r0 + r;
        if (r >= h) continue;
        const int at = sw_slot<NP>(q / (2 * NP), q % (2 * NP));
        float4 v = sm.x[at];
        for (int sg = 1; sg < nseg; ++sg) add4(v, sm.x[sg * hp * NP + at]);
        if (dir == 0) {
            const float4 b = sm.ext[tid + i * SWT];
            if (r < lo)
                z[(int64_t)(t.own0 + row) * NP + p] = make_float4(b.x * v.x - b.y * v.z, b.x * v.y - b.y * v.w,
                                                                  b.x * v.z + b.y * v.x, b.x * v.w + b.y * v.y);
            else
                u[(int64_t)(t.voff + row - t.nown) * NP + p] = make_float4(b.x + v.x, b.y + v.y, b.z + v.z, b.w + v.w);
        } else {
            y[(int64_t)(t.own0 + row) * NP + p] = v;
            const int node = __float_as_int(sm.ext[tid + i * SWT].x);
            if (c0 >= 0) A.sd[(int64_t)c0 * A.nnode + node] = make_float2(v.x, v.z);
            if (c1 >= 0) A.sd[(int64_t)c1 * A.nnode + node] = make_float2(v.y, v.w);
        }
    }
    sw_sync();                                           // every output of the tile is written
    // (the release carries the whole block's outputs, ordered before it by the barrier)
    if (tid == 0 && t.sig >= 0)
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(A.cnt + (int64_t)t.sig * ng + g) : "memory");
    return true;
}

__global__ void __launch_bounds__(SW_BLOCK, 4) sweep_kernel(SwArgs A) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SwShared& sm = *reinterpret_cast<SwShared*>(smem_raw);
    if (threadIdx.x == 0) {
        sm.quit = 0;
        for (int s = 0; s < SW_STAGES; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sw_smem(&sm.full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sw_smem(&sm.empty[s])), "r"(SWW) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x >= SWT) {
        if (threadIdx.x != SWT) return;
        // the producer: tickets in order, each task's panel run stage by stage
        uint32_t it = 0;
        for (bool go = true; go;) {
            const int tk = A.t0 + atomicAdd(A.ticket, 1);
            const bool done = tk >= A.t1;
            SwTask t{};
            int g = 0, dir = -1;
            const float2* src = nullptr;
            if (!done) {
                const int task = tk / A.G.ngroup;
                g = tk - task * A.G.ngroup;
                t = A.tasks[task];
                dir = task >= A.nft;
                src = (dir ? A.pb : A.pf) + (int64_t)A.G.op[g] * A.ptotal + t.off;
            }
            const int hp = (t.h + 1) & ~1;
            const int step = done ? 1 : SW_STAGE_ENT / hp;
            int k = t.k0;
            do {
                const int slot = it % SW_STAGES;
                if (it >= SW_STAGES) {
                    const uint32_t prev = (it / SW_STAGES - 1) & 1;
                    if (!sw_wait_bar(&sm.empty[slot], prev, A.gave_up, A.wait) || !sw_try(sw_smem(&sm.full[slot]), prev)) {
                        go = false;
                        break;
                    }
                }
                const int e = min(t.k1, k + step);
                if (k == t.k0) {
                    SwDesc& d = sm.desc[slot];
                    d.f_dir = dir;
                    d.g = g;
                    d.step = step;
                    d.t = t;
                }
                const uint32_t bytes = (uint32_t)(e - k) * hp * sizeof(float2), bar = sw_smem(&sm.full[slot]);
                if (bytes) {
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes + A.missing) : "memory");
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(sw_smem(sm.ring[slot])), "l"(src + (int64_t)(k - t.k0) * hp), "r"(bytes), "r"(bar)
                                 : "memory");
                } else {
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
                }
                ++it;
                k = e;
            } while (k < t.k1);
            if (done) go = false;
        }
        for (uint32_t q = it - min(it, (uint32_t)SW_STAGES); q < it; ++q)
            sw_drain(&sm.full[q % SW_STAGES], (q / SW_STAGES) & 1, A.wait);
        return;
    }
    uint32_t it = 0;
    bool bad = false;
    for (;;) {
        const int slot = it % SW_STAGES;
        const bool here = __all_sync(0xffffffffu, !bad && sw_wait_bar(&sm.full[slot], (it / SW_STAGES) & 1, A.gave_up, A.wait));
        const SwDesc& d = sm.desc[slot];
        if (!here) sm.quit = 1;
        if (!here || d.f_dir < 0) {                      // (the barriers of those that have a task)
            sw_sync();
            sw_sync();
            return;
        }
        bool go;
        switch (A.G.pair0[d.g + 1] - A.G.pair0[d.g]) {
            case 1: go = sw_task<1>(A, sm, it, d, bad); break;
            case 2: go = sw_task<2>(A, sm, it, d, bad); break;
            default: go = sw_task<4>(A, sm, it, d, bad); break;
        }
        if (!go) return;
    }
}

// blocks of the sweep kernel the current device holds at once
static int resident_blocks() {
    static std::mutex lock;
    static std::map<int, int> held;
    int dev = 0;
    GT_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(lock);
    int& n = held[dev];
    if (!n) {
        int sms = 0, per = 0;
        GT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        GT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sweep_kernel, SW_BLOCK, sizeof(SwShared)));
        n = std::max(1, sms * std::max(per, 1));
    }
    return n;
}

void launch_sweep(const SweepPlan& S, const Fronts& F, const c32* pf, const c32* pb, const c32* dinv, const c32* s, c32* z,
                  c32* y, c32* u, c32* sd, const Groups& G, int* cnt, unsigned int* gave_up, int t0, int t1, cudaStream_t st) {
    SwArgs A{};
    A.tasks = S.tasks;
    A.nft = S.nft;
    A.nsrc = S.nsrc;
    A.src_rows = S.src_rows;
    A.src = S.src;
    A.bidx = S.bidx;
    A.iperm = F.iperm;
    A.nfac = F.nfac;
    A.nvec = F.vec_total;
    A.nnode = F.nnode;
    A.ptotal = S.ptotal;
    A.pf = reinterpret_cast<const float2*>(pf);
    A.pb = reinterpret_cast<const float2*>(pb);
    A.dinv = reinterpret_cast<const float2*>(dinv);
    A.s = reinterpret_cast<const float2*>(s);
    A.z = reinterpret_cast<float4*>(z);
    A.y = reinterpret_cast<float4*>(y);
    A.u = reinterpret_cast<float4*>(u);
    A.sd = reinterpret_cast<float2*>(sd);
    A.G = G;
    A.cnt = cnt + 1;
    A.ticket = cnt;
    A.t0 = t0 * G.ngroup;
    A.t1 = t1 * G.ngroup;
    const char* test = std::getenv("GT_SWEEP_TEST_SHORTFALL");
    const bool shortfall = test && test[0] == '1', stages = test && test[0] == '2';
    A.gave_up = gave_up;
    A.wait = shortfall || stages ? SW_TEST_WAIT_CYCLES : SW_WAIT_CYCLES;
    A.surplus = shortfall ? 1 : 0;
    A.missing = stages ? 16 : 0;
    const int64_t tickets = (int64_t)(t1 - t0) * G.ngroup;
    if (tickets <= 0) return;
    raise_smem((const void*)sweep_kernel, sizeof(SwShared));
    pdl_launch(sweep_kernel, (int)std::min<int64_t>(tickets, resident_blocks()), SW_BLOCK, sizeof(SwShared), st, A);
    GT_LAUNCH_CHECK();
}

}  // namespace gt
