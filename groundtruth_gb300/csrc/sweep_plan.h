// The plan of the FP32 sweeps (sweep.cu): tiles, tasks and the counters they wait on, from the elimination tree alone.
// Host code without CUDA, so that the plan's order can be checked where there is no GPU.
#pragma once
#include <stdint.h>
#include <algorithm>
#include <vector>

namespace gt {

struct alignas(16) SwTask {
    int r0, h;             // outputs r0 .. r0 + h: rows of the front (forward) or own columns (backward)
    int k0, k1;            // inner indices: own columns (forward), front rows (backward)
    int dep, need;         // counter to wait on and the finished tiles it has to show
    int sig;               // counter to raise when done
    int nown, own0, voff;  // the front's own count, first factor index and place among the update vectors
    int64_t goff;          // forward: the front's first row in the source table; backward: its first boundary entry
    int64_t off;           // first panel entry
};
struct SweepPlanHost {
    std::vector<SwTask> tasks;          // forward, leaves to root, then backward, root to leaves
    int nft = 0, nbt = 0, nsrc = 0;
    int64_t src_rows = 0, ptotal = 0;
    std::vector<int> src, bidx;
    std::vector<int> hf, hb;            // outputs per tile of each front
    std::vector<int64_t> offf, offb;    // first entry of each front's tiles
    std::vector<int> level_f, level_b;  // tasks up to the end of each level, in the order they run
};

// Outputs per tile of a level: whole fronts while the level has tasks enough for the GPU by them, else 128, 64, 32 or 16,
// the widest that gives a column group 96 tasks (a wide tile gathers its inner rows once for more outputs; the top of the
// tree, one or a few fronts, takes narrow tiles to spread over the SMs).  6 columns of 131 x 203 x 4 solved in 159.4 ms; with
// 48 tasks 163.2, 32 169.3, 192 158.3, 384 159.8; 32 columns of 256 x 256 x 2 in 892, 893, 901, 892 and 901.
inline int sweep_tile_of(const int64_t* fronts, int64_t n, const std::vector<int>& ext) {
    for (int H : {128, 64, 32}) {
        int64_t tasks = 0;
        for (int64_t q = 0; q < n; ++q) tasks += (ext[fronts[q]] + H - 1) / H;
        if (tasks >= 96) return H;
    }
    return 16;
}

inline SweepPlanHost make_sweep_plan(int nfront, int nlev, const int64_t* level_ptr, const int64_t* order,
                                     const int64_t* own_start, const int64_t* nown, const int64_t* nbnd, const int64_t* bnd_ptr,
                                     const int64_t* bnd_idx, const int64_t* child_ptr, const int64_t* child_idx,
                                     const int64_t* cmap_ptr, const int64_t* cmap_idx, const int64_t* vec_off) {
    SweepPlanHost S;
    std::vector<int> nf(nfront), no(nfront), parent(nfront, -1);
    std::vector<int64_t> roff(nfront + 1, 0);
    for (int f = 0; f < nfront; ++f) {
        no[f] = (int)nown[f];
        nf[f] = (int)(nown[f] + nbnd[f]);
        roff[f + 1] = roff[f] + nf[f];
        // A front without a boundary passes nothing up and takes nothing down, wherever the tree has put it: it is a root
        // here.  Copper that falls apart along a dissection line makes them, under a front without a row; that one has no
        // tile, so that a wait on it would be a wait on nothing.
        for (int64_t c = child_ptr[f]; c < child_ptr[f + 1]; ++c)
            if (nbnd[child_idx[c]] > 0) parent[child_idx[c]] = f;
    }
    // each front row's sources among the update vectors, in the children's order
    S.src_rows = std::max<int64_t>(roff[nfront], 1);
    std::vector<std::vector<int>> lists;
    std::vector<int> held(S.src_rows, 0);
    for (int f = 0; f < nfront; ++f)
        for (int64_t ci = child_ptr[f]; ci < child_ptr[f + 1]; ++ci) {
            const int64_t c = child_idx[ci];
            for (int64_t i = 0; i < nbnd[c]; ++i) {
                const int64_t row = roff[f] + cmap_idx[cmap_ptr[ci] + i];
                const int k = held[row]++;
                if (k >= (int)lists.size()) lists.emplace_back(S.src_rows, -1);
                lists[k][row] = (int)(vec_off[c] + i);
            }
        }
    S.nsrc = (int)lists.size();
    for (auto& l : lists) S.src.insert(S.src.end(), l.begin(), l.end());
    S.bidx.assign(bnd_idx, bnd_idx + bnd_ptr[nfront]);
    // tile widths per front and the tiles' places in the panel copies
    S.hf.assign(nfront, 16);
    S.hb.assign(nfront, 16);
    for (int h = 0; h < nlev; ++h) {
        const int64_t* fr = order + level_ptr[h];
        const int64_t n = level_ptr[h + 1] - level_ptr[h];
        const int tf = sweep_tile_of(fr, n, nf), tb = sweep_tile_of(fr, n, no);
        for (int64_t q = 0; q < n; ++q) S.hf[fr[q]] = tf, S.hb[fr[q]] = tb;
    }
    S.offf.resize(nfront);
    S.offb.resize(nfront);
    std::vector<int> ntf(nfront, 0), ntb(nfront, 0);
    int64_t pf = 0, pb = 0;
    for (int f = 0; f < nfront; ++f) {
        S.offf[f] = pf;
        S.offb[f] = pb;
        for (int r = 0; r < nf[f]; r += S.hf[f]) {
            const int h = std::min(S.hf[f], nf[f] - r);
            pf += (int64_t)((h + 1) & ~1) * std::min(no[f], r + S.hf[f]);
            ++ntf[f];
        }
        for (int k = 0; k < no[f]; k += S.hb[f]) {
            const int h = std::min(S.hb[f], no[f] - k);
            pb += (int64_t)((h + 1) & ~1) * (nf[f] - k);
            ++ntb[f];
        }
    }
    S.ptotal = std::max<int64_t>({pf, pb, 2});
    S.ptotal += S.ptotal & 1;
    // counters: f: tiles of f's children done going up; nfront + f: f's own tiles done coming down; 2 nfront + f: a
    // root's own tiles done going up
    std::vector<int> need(nfront, 0);
    for (int f = 0; f < nfront; ++f)
        if (parent[f] >= 0) need[parent[f]] += ntf[f];
    for (int h = 0; h < nlev; ++h) {
        for (int64_t q = level_ptr[h]; q < level_ptr[h + 1]; ++q) {
            const int f = (int)order[q];
            int64_t off = S.offf[f];
            for (int r = 0; r < nf[f]; r += S.hf[f]) {
                SwTask t{};
                t.r0 = r;
                t.h = std::min(S.hf[f], nf[f] - r);
                t.k0 = 0;
                t.k1 = std::min(no[f], r + S.hf[f]);
                t.dep = f;
                t.need = need[f];
                t.sig = parent[f] >= 0 ? parent[f] : 2 * nfront + f;
                t.nown = no[f];
                t.own0 = (int)own_start[f];
                t.voff = (int)vec_off[f];
                t.goff = roff[f];
                t.off = off;
                off += (int64_t)((t.h + 1) & ~1) * t.k1;
                S.tasks.push_back(t);
            }
        }
        S.level_f.push_back((int)S.tasks.size());
    }
    S.nft = (int)S.tasks.size();
    for (int h = nlev - 1; h >= 0; --h) {
        for (int64_t q = level_ptr[h]; q < level_ptr[h + 1]; ++q) {
            const int f = (int)order[q];
            int a = parent[f];
            while (a >= 0 && !ntb[a]) a = parent[a];
            int root = f;
            while (parent[root] >= 0) root = parent[root];
            int64_t off = S.offb[f];
            for (int k = 0; k < no[f]; k += S.hb[f]) {
                SwTask t{};
                t.r0 = k;
                t.h = std::min(S.hb[f], no[f] - k);
                t.k0 = k;
                t.k1 = nf[f];
                t.dep = a >= 0 ? nfront + a : 2 * nfront + root;
                t.need = a >= 0 ? ntb[a] : ntf[root];
                t.sig = nfront + f;
                t.nown = no[f];
                t.own0 = (int)own_start[f];
                t.voff = (int)vec_off[f];
                t.goff = bnd_ptr[f];
                t.off = off;
                off += (int64_t)((t.h + 1) & ~1) * (t.k1 - t.k0);
                S.tasks.push_back(t);
            }
        }
        S.level_b.push_back((int)S.tasks.size());
    }
    S.nbt = (int)S.tasks.size() - S.nft;
    return S;
}

}  // namespace gt
