// link.cu -- frame-to-frame linking on the device.
//
// Restates the reference linker (gpu-tracking/src/linking.rs:197-492):
// candidate pairs closer than search_range (strict, squared distance),
// connected components of the bipartite source/destination graph discovered
// from each destination in index order, 1-1 components linked directly, and
// every other component resolved by the reference's exhaustive
// branch-and-bound (recurse2, linking.rs:390-452) with the same f32 score
// arithmetic, option order (sources ascending, null last) and tie rule.
//
// Parallel structure.  Frame t's assignment depends only on the positions of
// frames t-1 and t and on the memory entries M(t) (unlinked particles of the
// previous `memory` frames, deduplicated by trajectory).  All frames are
// linked at once with M = {}; M is then evaluated from the result, and links
// and M are updated in turn until no M changes in reach of a destination.
// M(t) depends on frames < t only, so iteration k settles frame k at the
// latest and the fixed point is the sequential result.
//
// What bounds it: latency.  A pass changes little (the benchmark movie of
// 1000 x 400 particles: 178k of its destinations in pass 1, a few hundred from
// pass 6 on), so a pass touches what changed and nothing else:
//   - membership in M is a bit per (particle, frame distance), and a
//     component whose memory entries did not change keeps its links: adding
//     or removing entries alters exactly the components that hold a
//     destination in reach of one (every piece that a removed entry leaves
//     behind was next to it), so those destinations are the pass's seeds;
//   - a warp (in the first linking a thread) explores one seed's component
//     through the frames' cell grids and resolves it; of the seeds of a
//     component the smallest does it.
//     There is no per-frame state, so the work spreads over the whole grid
//     whatever the frames' sizes.
// Relinking whole frames instead, a block per changed frame with the graph in
// shared memory, took 0.99 ms for that movie, 64 ms for 200 frames of 15k
// particles with memory 3 and 9.2 ms for a table of 500 frames of 760.
#include <cooperative_groups.h>

#include <climits>
#include <type_traits>

#include "gt_device.cuh"

namespace cg = cooperative_groups;

namespace gt {

namespace {
constexpr int NTL = 256;  // threads of a linker block
constexpr int NEAR = 2;   // candidates loaded at once by a thread


__device__ __forceinline__ bool within_r(float qy, float qx, float iy, float ix, float r, float* dist) {
    // kd-tree box pre-filter + linking.rs:91-100 distance (dest - source)
    if (iy < qy - r || iy > qy + r) return false;
    if (ix < qx - r || ix > qx + r) return false;
    const float dy = iy - qy, dx = ix - qx;
    float dd = 0.f;
    dd = dd + dy * dy;
    dd = dd + dx * dx;
    *dist = dd;
    return dd < r * r;
}

// The frame of compact particle index g, in [lo, hi).
__device__ __forceinline__ int frame_of(const LinkBufs& L, int g, int lo, int hi) {
    --hi;
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (__ldg(L.off + m) <= g) lo = m;
        else hi = m - 1;
    }
    return lo;
}

// fn(index, y, x) for the particles of frame f in the 3 x 3 cells around
// (qy, qx): a row of cells is one range of the cell-ordered positions.  The
// cells are at least search_range + 1 wide, so rounding of the cell number
// cannot lose a pair.  Stops when fn returns false.
template <class F>
__device__ __forceinline__ bool near(const LinkBufs& L, int f, float qy, float qx, F&& fn) {
    const float ig = L.inv_g;
    const int cy = clampi((int)floorf(qy * ig), 0, L.ncy - 1), cx = clampi((int)floorf(qx * ig), 0, L.ncx - 1);
    const int x0 = max(cx - 1, 0), x1 = min(cx + 1, L.ncx - 1) + 1;
    const int* gs = L.gstart + (size_t)f * ((size_t)L.ncx * L.ncy + 1);
    int a[3], n[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const int yy = cy + q - 1;
        const bool in = yy >= 0 && yy < L.ncy;
        a[q] = in ? __ldg(gs + yy * L.ncx + x0) : 0;
        n[q] = in ? __ldg(gs + yy * L.ncx + x1) - a[q] : 0;
    }
    const size_t base = (size_t)f * L.cap_p;
    const int n01 = n[0] + n[1], total = n01 + n[2];
    // a few candidates' loads in flight at once
    for (int s = 0; s < total; s += NEAR) {
        float2 p[NEAR];
        int id[NEAR];
#pragma unroll
        for (int u = 0; u < NEAR; ++u) {
            const int q = min(s + u, total - 1);
            const size_t at = base + (q < n[0] ? a[0] + q : q < n01 ? a[1] + (q - n[0]) : a[2] + (q - n01));
            p[u] = __ldg(L.gpos + at);
            id[u] = __ldg(L.gidx + at);
        }
#pragma unroll
        for (int u = 0; u < NEAR; ++u)
            if (s + u < total && !fn(id[u], p[u].x, p[u].y)) return false;
    }
    return true;
}

// *ctr += 1: one atomic for the lanes that call together with the same
// counter (lanes of a warp may be at different movies of a batch).
__device__ __forceinline__ int push_slot(int* ctr) {
    const unsigned same = __match_any_sync(__activemask(), (unsigned long long)ctr);
    const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(ctr, __popc(same));
    return __shfl_sync(same, base, leader) + __popc(same & ((1u << lane) - 1u));
}

// One component: destinations (index in frame t), sources (keys that order
// them as linking.rs:244-259 does: frame t-1 by index, then the memory
// entries by (frame, index): cap_p + slab handle) and their edges.  By size:
//   8 destinations, 8 sources, 24 edges   a thread's local arrays (SmallComp),
//                                         in the first linking;
//   32, 32, 112                           a warp's registers (WarpComp), in the
//                                         first linking and the passes;
//   256, 256, 1024                        a warp with the block's arrays (MemComp);
//   beyond                                a warp with a slot of LinkBufs::big.
// A thread that goes on to 32 takes far longer than a warp: tables of 300 chains
// of 31 particles 1.22 ms a call, 0.28 with the warps; and one thread of 64
// blocks at a time for all that is larger 0.78 ms and more (4000 chains of 40:
// 217 ms, 1.4 with the block's arrays; 300 of 400: 2.7).
constexpr int CAP_T = 8, CAP_TE = 24, CAP_N = 32, CAP_E = 112;

// Set of at most 32 sources or destinations.
struct BitSet {
    unsigned m = 0;
    __device__ bool has(int i) const { return (m >> i) & 1u; }
    __device__ void add(int i) { m |= 1u << i; }
    __device__ void del(int i) { m &= ~(1u << i); }
    __device__ void clear(int) { m = 0; }
};

template <class I>
struct ArraySet {
    I* p;
    __device__ bool has(int i) const { return p[i] != 0; }
    __device__ void add(int i) { p[i] = 1; }
    __device__ void del(int i) { p[i] = 0; }
    __device__ void clear(int n) {
        for (int i = 0; i < n; ++i) p[i] = 0;
    }
};

struct SmallComp {
    int D[CAP_T];
    unsigned S[CAP_T];
    float ew[CAP_TE], dw[CAP_TE];
    unsigned char ed[CAP_TE], es[CAP_TE], dsrc[CAP_TE];
    unsigned char doff[CAP_T + 1], path[CAP_T], oi[CAP_T], stk[2 * CAP_T];
    signed char cur[CAP_T], best[CAP_T];
    __device__ BitSet sset() { return BitSet(); }
};

// Arrays for cd destinations, cs sources and ce edges (comp_bytes), in shared
// memory (I: 16 bits) or in a slot of LinkBufs::big (I: int).
template <class I>
struct MemComp {
    int cd, cs, ce;
    float* dw;               // edges, grouped by destination in the order found
    int* D;
    unsigned* S;
    I *dsrc, *list, *doff;   // source per edge; the sources' lists
    int* soff;               // ends of the sources' lists
    I *path, *oi, *stk, *used, *vis;
    typename std::make_signed<I>::type *cur, *best;
    char* hash;              // during the exploration, in the place of soff and the others
    __device__ ArraySet<I> sset() const { return ArraySet<I>{used}; }

    __device__ MemComp(void* mem, int cd_, int cs_, int ce_) : cd(cd_), cs(cs_), ce(ce_) {
        dw = (float*)mem;
        D = (int*)(dw + ce);
        S = (unsigned*)(D + cd);
        dsrc = (I*)(S + cs);
        list = dsrc + ce;
        doff = list + ce;
        hash = (char*)mem + comp_lists(cd, cs, ce, sizeof(I));
        soff = (int*)hash;
        I* q = (I*)(soff + cs);
        auto take = [&](int n) { I* r = q; q += n; return r; };
        path = take(cd); oi = take(cd); stk = take(cd + cs); used = take(cs); vis = take(cd);
        cur = (decltype(cur))take(cd); best = (decltype(best))take(cd);
    }
};

// Keys and their numbers in the order of arrival: a warp's lanes put theirs in
// side by side (a search among the arrived ones: 300 chains of 255 2.03 ms a
// call instead of 1.27).
constexpr unsigned NO_KEY = 0xffffffffu;
template <class I>
struct KeyTable {
    unsigned* key;
    I* val;
    int size;  // a power of two
    __device__ void clear() {
        for (int i = threadIdx.x & 31; i < size; i += 32) key[i] = NO_KEY;
    }
    // The number of each key that is wanted: new ones from *n on, if cap holds
    // them (else false).  Every lane calls it.
    __device__ bool put(unsigned k, bool want, int cap, int* n, int* idx, bool* fresh) {
        const unsigned full = 0xffffffffu;
        unsigned h = (k * 2654435761u) >> (__clz(size) + 1);
        bool is_new = false;
        if (want)
            while (true) {
                const unsigned old = atomicCAS(key + h, NO_KEY, k);
                is_new = old == NO_KEY;
                if (is_new || old == k) break;
                h = (h + 1) & (size - 1);
            }
        const unsigned news = __ballot_sync(full, is_new);
        *fresh = is_new;
        *idx = *n + __popc(news & ((1u << (threadIdx.x & 31)) - 1u));
        if (*n + __popc(news) > cap) return false;
        if (is_new) val[h] = (I)*idx;
        __syncwarp();
        if (want && !is_new) *idx = val[h];
        *n += __popc(news);
        return true;
    }
};

// A component of the block's own arrays.
constexpr int MID_N = 256, MID_E = 1024;
constexpr int MID_BYTES = (int)comp_bytes(MID_N, MID_N, MID_E, 2);

// DFS preorder of the destinations from `first` (linking.rs:316-342) over
// the per-destination lists: neighbours in ascending order, so the next node
// is the smallest one not yet visited.
__device__ void dfs_order(SmallComp& c, int first, int nd, int ne) {
    BitSet vis, used;
    int top = 1, np = 0;
    c.stk[0] = first;
    vis.add(first);
    c.path[np++] = first;
    while (top > 0) {
        const int node = c.stk[top - 1];
        int next = -1;
        if (node < nd) {
            for (int z = c.doff[node]; z < c.doff[node + 1]; ++z)
                if (!used.has(c.dsrc[z])) { next = c.dsrc[z]; break; }
            if (next >= 0) {
                used.add(next);
                next += nd;
            }
        } else {
            const int s = node - nd;
            for (int e = 0; e < ne; ++e)
                if (c.es[e] == s && !vis.has(c.ed[e]) && (next < 0 || c.D[c.ed[e]] < c.D[next])) next = c.ed[e];
            if (next >= 0) {
                vis.add(next);
                c.path[np++] = next;
            }
        }
        if (next < 0) --top;
        else c.stk[top++] = next;
    }
}

// The same over the lists of both sides.
template <class I>
__device__ void dfs_order(const MemComp<I>& c, int first, int nd) {
    int top = 1, np = 0;
    c.stk[0] = (I)first;
    c.vis[first] = 1;
    c.path[np++] = (I)first;
    while (top > 0) {
        const int node = c.stk[top - 1];
        int next = -1;
        if (node < nd) {
            const int z1 = c.doff[node + 1];
            for (int z = c.doff[node]; z < z1 && next < 0; ++z)
                if (!c.used[c.dsrc[z]]) next = c.dsrc[z];
            if (next >= 0) {
                c.used[next] = 1;
                next += nd;
            }
        } else {
            const int s = node - nd, z1 = c.soff[s];
            int dn = 0;
            for (int z = s > 0 ? c.soff[s - 1] : 0; z < z1; ++z) {
                const int q = c.list[z];
                if (c.vis[q]) continue;
                const int dq = c.D[q];
                if (next < 0 || dq < dn) { next = q; dn = dq; }
            }
            if (next >= 0) {
                c.vis[next] = 1;
                c.path[np++] = (I)next;
            }
        }
        if (next < 0) --top;
        else c.stk[top++] = (I)next;
    }
}

// Exhaustive search of one subnet (linking.rs:390-452): destinations in DFS
// order (path); sources are chosen through the per-destination lists
// (ascending source order), null costs r^2.  Returns false when the
// option-trial budget is exhausted.
template <class C>
__device__ bool solve_subnet(C& c, int nd, int ns, long long budget, float null_cost) {
    auto used = c.sset();
    used.clear(ns);
    float score = 0.f, best = CUDART_INF_F;
    long long trials = 0;
    int l = 0, o = 0, d0 = 0, nreal = 0;  // level, its option, its list
    auto level = [&](int q) {
        const int d = c.path[q];
        d0 = c.doff[d];
        nreal = c.doff[d + 1] - d0;
    };
    level(0);
    while (true) {
        if (o > nreal || score > best) {  // options exhausted, or early return
            if (l == 0) break;
            level(--l);
            // child returned: undo this level's option and advance
            o = c.oi[l];
            float w = null_cost;
            if (o < nreal) {
                w = c.dw[d0 + o];
                used.del(c.dsrc[d0 + o]);
            }
            score -= w;
            ++o;
            continue;
        }
        if (++trials > budget) return false;
        float w = null_cost;
        int s = -1;
        if (o < nreal) {
            w = c.dw[d0 + o];
            s = c.dsrc[d0 + o];
        }
        score += w;
        if (s >= 0) {
            if (used.has(s)) { score -= w; ++o; continue; }
            used.add(s);
        }
        c.cur[l] = s;
        if (l == nd - 1) {
            if (score < best) {
                best = score;
                for (int q = 0; q < nd; ++q) c.best[q] = c.cur[q];
            }
            if (s >= 0) used.del(s);
            score -= w;
            ++o;
        } else {
            c.oi[l] = o;
            level(++l);
            o = 0;
        }
    }
    return true;
}

enum CompResult { COMP_DONE = 0, COMP_SKIP = 1, COMP_BIG = 2 };

__device__ __forceinline__ bool in_memory(const LinkBufs& L, int g, int dist) {
    return (__ldcg(L.mm + (size_t)((dist - 1) >> 5) * L.np + g) >> ((dist - 1) & 31)) & 1u;
}

// Writes the link of destination g (frame t): pred, the linked bits of the
// old and the new source, and (pass > 0) both sources for the next pass's
// membership check.  Bit j of L.lnk: linked by the frame j + 1 later.
__device__ __forceinline__ void mark_linked(const LinkBufs& L, int src, int fs, int t, int k, bool set) {
    const int j = t - fs - 1;
    if (j < 2) {
        if (set) atomicOr(L.lnk + src, 1u << j);
        else atomicAnd(L.lnk + src, ~(1u << j));
        if (k > 0 && L.memory <= 2 && atomicExch(L.rstamp + src, k) != k)
            L.recq[push_slot(L.ctr + (k & 3) * NCTR + C_CHECKS)] = src;
    }
}

// The compact index of source `key` (-1: none) of frame t and its frame.
__device__ __forceinline__ int source_of(const LinkBufs& L, long long key, int t, int* fs) {
    *fs = t - 1;
    if (key < 0) return -1;
    unsigned h = (unsigned)key;
    if (h >= (unsigned)L.cap_p) {
        h -= (unsigned)L.cap_p;
        *fs = (int)(h / (unsigned)L.cap_p);
        h -= (unsigned)(*fs * L.cap_p);
    }
    return __ldg(L.off + *fs) + (int)h;
}

// Destination g (frame t) gets source `key`: give_up releases its former
// source if that is another, take_up writes the link.
__device__ __forceinline__ void give_up(const LinkBufs& L, long long key, int g, int t, int k) {
    int fs;
    const int src = source_of(L, key, t, &fs);
    const int old = __ldcg(L.pred + g);
    if (old < 0 || old == src) return;
    int fo = t - 1;
    while (__ldg(L.off + fo) > old) --fo;
    mark_linked(L, old, fo, t, k, false);
}

__device__ __forceinline__ void take_up(const LinkBufs& L, long long key, int g, int t, int k) {
    int fs;
    const int src = source_of(L, key, t, &fs);
    if (k > 0 && __ldcg(L.pred + g) == src) return;
    L.pred[g] = src;
    if (k > 0 && L.memory > 2) {  // the trajectories that the change touches
        L.cstamp[__ldcg(L.root + g)] = k + 1;
        if (src >= 0) L.cstamp[__ldcg(L.root + src)] = k + 1;
    }
    if (src >= 0 && L.memory > 0) mark_linked(L, src, fs, t, k, true);
}

// Explores the component of destination d of frame t and resolves it, in the
// first linking: every destination is a seed and there are no memory entries.
// COMP_SKIP: a smaller seed of the same component does it; COMP_BIG: it does
// not fit c (nothing is written).
__device__ int link_component(const LinkBufs& L, SmallComp& c, int t, int d) {
    const float r = L.r;
    const int offt = __ldg(L.off + t);
    const size_t bt = (size_t)t * L.cap_p;
    int nd = 1, ns = 0, ne = 0, qd = 0, qs = 0, res = COMP_DONE;
    c.D[0] = d;
    while (true) {
        if (qd < nd) {
            const int di = qd++;
            const float y = __ldg(L.py + bt + c.D[di]), x = __ldg(L.px + bt + c.D[di]);
            if (t > 0)
                near(L, t - 1, y, x, [&](int i, float sy, float sx) {
                    float w;
                    if (!within_r(sy, sx, y, x, r, &w)) return true;
                    int s = 0;
                    while (s < ns && c.S[s] != (unsigned)i) ++s;
                    if (ne == CAP_TE || s == CAP_T) { res = COMP_BIG; return false; }
                    if (s == ns) c.S[ns++] = (unsigned)i;
                    c.ed[ne] = di;
                    c.es[ne] = s;
                    c.ew[ne++] = w;
                    return true;
                });
        } else if (qs < ns) {
            const size_t h = (size_t)(t - 1) * L.cap_p + c.S[qs++];
            const float sy = __ldg(L.py + h), sx = __ldg(L.px + h);
            near(L, t, sy, sx, [&](int i, float y, float x) {
                float w;
                if (!within_r(sy, sx, y, x, r, &w)) return true;
                int q = 0;
                while (q < nd && c.D[q] != i) ++q;
                if (q < nd) return true;
                if (i < d) { res = COMP_SKIP; return false; }
                if (nd == CAP_T) { res = COMP_BIG; return false; }
                c.D[nd++] = i;
                return true;
            });
        } else {
            break;
        }
        if (res != COMP_DONE) return res;
    }
    if (nd == 1 && ns <= 1) {
        c.path[0] = 0;
        c.best[0] = ns - 1;  // the only source, or none
    } else {
        // per-destination lists, ascending source order (linking.rs:310-315)
        for (int q = 0; q <= nd; ++q) c.doff[q] = 0;
        for (int e = 0; e < ne; ++e) ++c.doff[c.ed[e] + 1];
        for (int q = 0; q < nd; ++q) c.doff[q + 1] = c.doff[q + 1] + c.doff[q];
        for (int q = 0; q < nd; ++q) c.path[q] = 0;  // entries so far
        for (int e = 0; e < ne; ++e) {
            const int q = c.ed[e];
            const int s = c.es[e];
            const float w = c.ew[e];
            int z = c.doff[q] + c.path[q];
            c.path[q] = c.path[q] + 1;
            while (z > c.doff[q] && c.S[c.dsrc[z - 1]] > c.S[s]) {
                c.dsrc[z] = c.dsrc[z - 1];
                c.dw[z] = c.dw[z - 1];
                --z;
            }
            c.dsrc[z] = s;
            c.dw[z] = w;
        }
        int first = 0;
        for (int q = 1; q < nd; ++q)
            if (c.D[q] < c.D[first]) first = q;
        dfs_order(c, first, nd, ne);
        for (int q = 0; q < nd; ++q) c.best[q] = -1;
        if (!solve_subnet(c, nd, ns, L.budget, r * r)) atomicOr(L.err, ERR_SUBNET_BUDGET);
    }
    for (int q = 0; q < nd; ++q) take_up(L, c.best[q] < 0 ? -1 : (long long)c.S[c.best[q]], offt + c.D[c.path[q]], t, 0);
    return COMP_DONE;
}

// A seed's component by a warp: what a thread does one
// dependent load after the other (up to 100k cycles for a component of 3
// destinations and 5 sources with memory 3) the lanes do side by side.  The
// nodes of a search level are expanded together: their cell ranges in all
// frames, then the ranges' particles, then the membership bits.  Lane i holds
// destination i and source i; edges go through shared memory.
struct WarpComp {
    float ew[CAP_E], w[CAP_E];  // edges as found, then by search level
    unsigned char ed[CAP_E], es[CAP_E], s[CAP_E];
};

// Row q of the 3 x 3 cells around (y, x) in frame f: its first slab index and
// particle count (0 for rows outside the grid).
__device__ __forceinline__ void cell_row(const LinkBufs& L, int f, int q, float y, float x, unsigned* a, int* n) {
    const int cy = clampi((int)floorf(y * L.inv_g), 0, L.ncy - 1) + q - 1;
    const int cx = clampi((int)floorf(x * L.inv_g), 0, L.ncx - 1);
    *a = 0;
    *n = 0;
    if (cy < 0 || cy >= L.ncy) return;
    const int* gs = L.gstart + (size_t)f * ((size_t)L.ncx * L.ncy + 1) + (size_t)cy * L.ncx;
    const int a0 = __ldg(gs + max(cx - 1, 0)), a1 = __ldg(gs + min(cx + 1, L.ncx - 1) + 1);
    *a = (unsigned)(f * L.cap_p + a0);
    *n = a1 - a0;
}

// fn(row, slab index in cell order) for the particles of the rows held by
// lanes [0, nrows) (first index a, count n), 32 particles at a time; row is -1
// on lanes without one.  Stops when fn (uniform) returns false.
template <class F>
__device__ __forceinline__ bool each_in_rows(unsigned a, int n, int nrows, F&& fn) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int incl = lane < nrows ? n : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(full, incl, d);
        if (lane >= d) incl += v;
    }
    const int total = __shfl_sync(full, incl, 31);
    for (int base = 0; base < total; base += 32) {
        // the row of particle idx: the first whose inclusive sum exceeds it
        // (binary search over the lanes)
        const int idx = base + lane;
        int row = 0;
#pragma unroll
        for (int b = 16; b > 0; b >>= 1)
            if (__shfl_sync(full, incl, row + b - 1) <= idx) row += b;
        row = min(row, nrows - 1);
        const unsigned first = __shfl_sync(full, a, row);
        const int before = __shfl_sync(full, incl - n, row);
        if (!fn(idx < total ? row : -1, first + (unsigned)(idx - before))) return false;
    }
    return true;
}

// The component of seed d of frame t (t >= 1) in pass k, as link_component (k =
// 0: the first linking).
__device__ int link_component_warp(const LinkBufs& L, WarpComp& c, int t, int d, int k) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const float r = L.r;
    const int offt = __ldg(L.off + t);
    int myD = d;  // lane i: destination i, its position, source i, its position
    float dy = __ldg(L.py + (size_t)t * L.cap_p + d), dx = __ldg(L.px + (size_t)t * L.cap_p + d);
    unsigned myS = 0;
    float sy = 0.f, sx = 0.f;
    int nd = 1, ns = 0, ne = 0, qd = 0, qs = 0, res = COMP_DONE;
    const int ngr = k == 0 ? 1 : min(L.memory, t - 1) + 1;  // source frames t-1, t-2, ...
    while (true) {
        if (qd < nd) {
            // 3 rows of cells in each source frame; several destinations at
            // once while their rows fit the warp
            const int nb = 3 * ngr <= 16 ? min(nd - qd, 32 / (3 * ngr)) : 1;
            for (int j0 = 0; j0 < ngr; j0 += 10) {
                const int per = 3 * min(10, ngr - j0);
                const int mine = qd + min(lane / per, nb - 1);
                const float y = __shfl_sync(full, dy, mine), x = __shfl_sync(full, dx, mine);
                const int q = lane - (mine - qd) * per;
                unsigned a = 0;
                int n = 0;
                if (lane < nb * per) cell_row(L, t - 1 - j0 - q / 3, q % 3, y, x, &a, &n);
                const bool go = each_in_rows(a, n, nb * per, [&](int row, unsigned at) {
                    const int node = max(row, 0) / per;
                    const float y = __shfl_sync(full, dy, qd + node), x = __shfl_sync(full, dx, qd + node);
                    unsigned key = 0;
                    float w = 0.f;
                    float2 p = make_float2(0.f, 0.f);
                    bool hit = false;
                    if (row >= 0) {
                        const int j = j0 + (row - node * per) / 3, f = t - 1 - j;
                        p = __ldg(L.gpos + at);
                        const int i = __ldg(L.gidx + at);
                        hit = within_r(p.x, p.y, y, x, r, &w);
                        if (hit && j > 0) hit = in_memory(L, __ldg(L.off + f) + i, j);
                        key = j == 0 ? (unsigned)i : (unsigned)L.cap_p + (unsigned)(f * L.cap_p + i);
                    }
                    for (unsigned m = __ballot_sync(full, hit); m; m &= m - 1) {
                        const int b = __ffs(m) - 1;
                        const unsigned kb = __shfl_sync(full, key, b);
                        const float yb = __shfl_sync(full, p.x, b), xb = __shfl_sync(full, p.y, b);
                        const unsigned same = __ballot_sync(full, lane < ns && myS == kb);
                        int s = __ffs(same) - 1;
                        if (!same) {
                            if (ns == CAP_N) { res = COMP_BIG; return false; }
                            s = ns++;
                            if (lane == s) { myS = kb; sy = yb; sx = xb; }
                        }
                        if (ne == CAP_E) { res = COMP_BIG; return false; }
                        if (lane == b) {
                            c.ed[ne] = (unsigned char)(qd + node);
                            c.es[ne] = (unsigned char)s;
                            c.ew[ne] = w;
                        }
                        ++ne;
                    }
                    return true;
                });
                if (!go) return res;
            }
            qd += nb;
        } else if (qs < ns) {
            const int nb = min(ns - qs, 10);
            const int mine = qs + min(lane / 3, nb - 1);
            const float y = __shfl_sync(full, sy, mine), x = __shfl_sync(full, sx, mine);
            unsigned a = 0;
            int n = 0;
            if (lane < 3 * nb) cell_row(L, t, lane % 3, y, x, &a, &n);
            const bool go = each_in_rows(a, n, 3 * nb, [&](int row, unsigned at) {
                const int node = qs + max(row, 0) / 3;
                const float y = __shfl_sync(full, sy, node), x = __shfl_sync(full, sx, node);
                int i = -1;
                bool hit = false, smaller = false;
                float2 p = make_float2(0.f, 0.f);
                if (row >= 0) {
                    p = __ldg(L.gpos + at);
                    i = __ldg(L.gidx + at);
                    float w;
                    hit = within_r(y, x, p.x, p.y, r, &w);
                    smaller = hit && i < d && (k == 0 || __ldcg(L.stamp + offt + i) == k);
                }
                if (__any_sync(full, smaller)) { res = COMP_SKIP; return false; }
                for (unsigned m = __ballot_sync(full, hit); m; m &= m - 1) {
                    const int b = __ffs(m) - 1;
                    const int ib = __shfl_sync(full, i, b);
                    const float yb = __shfl_sync(full, p.x, b), xb = __shfl_sync(full, p.y, b);
                    if (__any_sync(full, lane < nd && myD == ib)) continue;
                    if (nd == CAP_N) { res = COMP_BIG; return false; }
                    if (lane == nd) { myD = ib; dy = yb; dx = xb; }
                    ++nd;
                }
                return true;
            });
            if (!go) return res;
            qs += nb;
        } else {
            break;
        }
    }
    long long key = -1;  // lane i < nd: the source that destination mine gets
    int mine = myD;
    if (nd == 1 && ns <= 1) {
        if (ns == 1) key = __shfl_sync(full, myS, 0);
    } else {
        // ranks: destinations by index, sources by key, so that the search's
        // "ascending" is the order of bits
        int rd = 0, rs = 0;
        for (int q = 0; q < nd; ++q) rd += __shfl_sync(full, myD, q) < myD;
        for (int q = 0; q < ns; ++q) rs += __shfl_sync(full, myS, q) < myS;
        unsigned srcs = 0, dsts = 0;  // lane i: neighbours of destination i, of source i (ranks)
        int sortD = 0, sortS = 0;     // the destination and the source of rank i
        for (int q = 0; q < nd; ++q)
            if (__shfl_sync(full, rd, q) == lane) sortD = q;
        for (int q = 0; q < ns; ++q)
            if (__shfl_sync(full, rs, q) == lane) sortS = q;
        mine = __shfl_sync(full, myD, sortD);
        const unsigned keyS = __shfl_sync(full, myS, sortS);
        __syncwarp();
        for (int e0 = 0; e0 < ne; e0 += 32) {
            const int e = e0 + lane;
            const int q = __shfl_sync(full, rd, e < ne ? c.ed[e] : 0), s = __shfl_sync(full, rs, e < ne ? c.es[e] : 0);
            const int cnt = min(32, ne - e0);
            for (int b = 0; b < cnt; ++b) {
                const int qb = __shfl_sync(full, q, b), sb = __shfl_sync(full, s, b);
                if (lane == qb) srcs |= 1u << sb;
                if (lane == sb) dsts |= 1u << qb;
            }
        }
        // DFS preorder from the smallest destination (linking.rs:316-342)
        unsigned vd = 1u, vs = 0u;
        int level = lane == 0 ? 0 : -1;  // lane i: level of destination i in the order
        int np = 1, node = 0, top = 0;   // node < 32: destination, else source + 32
        int stk = 0;                     // lane q: entry q of the stack (entries 32.. in stk2)
        int stk2 = 0;
        while (true) {
            const bool isd = node < 32;
            const unsigned nb = __shfl_sync(full, isd ? srcs : dsts, node & 31) & ~(isd ? vs : vd);
            if (nb) {
                const int x = __ffs(nb) - 1;
                if (lane == (top & 31)) {
                    if (top < 32) stk = node;
                    else stk2 = node;
                }
                ++top;
                if (isd) {
                    vs |= 1u << x;
                    node = x + 32;
                } else {
                    vd |= 1u << x;
                    if (lane == x) level = np;
                    ++np;
                    node = x;
                }
            } else {
                if (top == 0) break;
                --top;
                node = __shfl_sync(full, top < 32 ? stk : stk2, top & 31);
            }
        }
        // the search's option lists: lane l holds level l's destination, the
        // start of its list and its length
        int dest = 0;
        for (int q = 0; q < nd; ++q)
            if (__shfl_sync(full, level, q) == lane) dest = q;
        const unsigned lsrcs = __shfl_sync(full, srcs, dest);
        const int deg = lane < nd ? __popc(lsrcs) : 0;
        int start = deg;
#pragma unroll
        for (int q = 1; q < 32; q <<= 1) {
            const int v = __shfl_up_sync(full, start, q);
            if (lane >= q) start += v;
        }
        start -= deg;
        for (int e0 = 0; e0 < ne; e0 += 32) {
            const int e = e0 + lane;
            const bool in = e < ne;
            const int q = __shfl_sync(full, rd, in ? c.ed[e] : 0), s = __shfl_sync(full, rs, in ? c.es[e] : 0);
            const int at = __shfl_sync(full, start, __shfl_sync(full, level, q));
            const unsigned before = __shfl_sync(full, srcs, q) & ((1u << s) - 1u);
            if (in) {
                c.w[at + __popc(before)] = c.ew[e];
                c.s[at + __popc(before)] = (unsigned char)s;
            }
        }
        __syncwarp();
        // exhaustive search (solve_subnet), every lane in step; lane l keeps
        // level l's option
        const float null_cost = r * r;
        float score = 0.f, best = CUDART_INF_F;
        unsigned used = 0;
        int l = 0, o = 0, opt = -1, bopt = -1;
        int l0 = __shfl_sync(full, start, 0), nreal = __shfl_sync(full, deg, 0);
        long long trials = 0;
        while (true) {
            if (o > nreal || score > best) {
                if (l == 0) break;
                --l;
                l0 = __shfl_sync(full, start, l);
                nreal = __shfl_sync(full, deg, l);
                o = __shfl_sync(full, opt, l);
                float w = null_cost;
                if (o < nreal) {
                    w = c.w[l0 + o];
                    used &= ~(1u << c.s[l0 + o]);
                }
                score -= w;
                ++o;
                continue;
            }
            if (++trials > L.budget) {
                if (lane == 0) atomicOr(L.err, ERR_SUBNET_BUDGET);
                break;
            }
            float w = null_cost;
            unsigned bit = 0;
            if (o < nreal) {
                w = c.w[l0 + o];
                bit = 1u << c.s[l0 + o];
            }
            score += w;
            if (used & bit) { score -= w; ++o; continue; }
            if (lane == l) opt = o;
            if (l == nd - 1) {
                if (score < best) {
                    best = score;
                    bopt = opt;
                }
                score -= w;
                ++o;
            } else {
                used |= bit;
                ++l;
                l0 = __shfl_sync(full, start, l);
                nreal = __shfl_sync(full, deg, l);
                o = 0;
            }
        }
        const bool real = lane < nd && bopt >= 0 && bopt < deg;
        const unsigned got = __shfl_sync(full, keyS, real ? c.s[start + bopt] : 0);
        if (real) key = got;
        mine = __shfl_sync(full, mine, dest);
    }
    // every source given up before any is taken
    if (k > 0 && lane < nd) give_up(L, key, offt + mine, t, k);
    __syncwarp();
    if (lane < nd) take_up(L, key, offt + mine, t, k);
    __syncwarp();
    return COMP_DONE;
}

// The component of seed d of frame t (t >= 1) in pass k by a warp, with arrays
// in memory: explored as in link_component_warp, then lanes sort the
// destinations' lists and make the sources', and lane 0 orders and searches.
// What bounds it: latency, of the exploration's steps and of the search's loads.
template <class I>
__device__ int link_component_mem(const LinkBufs& L, MemComp<I> c, int t, int d, int k) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const float r = L.r;
    const int offt = __ldg(L.off + t);
    const size_t bt = (size_t)t * L.cap_p;
    int nd = 0, ns = 0, ne = 0, qd = 0, qs = 0, res = COMP_DONE;
    const int ngr = k == 0 ? 1 : min(L.memory, t - 1) + 1;  // source frames t-1, t-2, ...
    const int hd = hash_size(c.cd), hs = hash_size(c.cs);
    unsigned* keys = (unsigned*)c.hash;
    KeyTable<I> dt{keys, (I*)(keys + hd + hs), hd}, stab{keys + hd, (I*)(keys + hd + hs) + hd, hs};
    dt.clear();
    stab.clear();
    if (lane == 0) c.D[0] = d;
    __syncwarp();
    int idx;
    bool fresh;
    dt.put((unsigned)d, lane == 0, c.cd, &nd, &idx, &fresh);
    while (true) {
        if (qd < nd) {
            const int nb = 3 * ngr <= 16 ? min(nd - qd, 32 / (3 * ngr)) : 1;
            for (int j0 = 0; j0 < ngr; j0 += 10) {
                const int per = 3 * min(10, ngr - j0);
                const int mine = qd + min(lane / per, nb - 1);
                const float y = __ldg(L.py + bt + c.D[mine]), x = __ldg(L.px + bt + c.D[mine]);
                const int q = lane - (mine - qd) * per;
                unsigned a = 0;
                int n = 0;
                if (lane < nb * per) cell_row(L, t - 1 - j0 - q / 3, q % 3, y, x, &a, &n);
                const bool go = each_in_rows(a, n, nb * per, [&](int row, unsigned at) {
                    const int node = max(row, 0) / per;
                    const float y1 = __shfl_sync(full, y, node * per), x1 = __shfl_sync(full, x, node * per);
                    unsigned key = 0;
                    float w = 0.f;
                    bool hit = false;
                    if (row >= 0) {
                        const int j = j0 + (row - node * per) / 3, f = t - 1 - j;
                        const float2 p = __ldg(L.gpos + at);
                        const int i = __ldg(L.gidx + at);
                        hit = within_r(p.x, p.y, y1, x1, r, &w);
                        if (hit && j > 0) hit = in_memory(L, __ldg(L.off + f) + i, j);
                        key = j == 0 ? (unsigned)i : (unsigned)L.cap_p + (unsigned)(f * L.cap_p + i);
                    }
                    const unsigned hits = __ballot_sync(full, hit);
                    int s;
                    bool first;
                    if (ne + __popc(hits) > c.ce || !stab.put(key, hit, c.cs, &ns, &s, &first)) {
                        res = COMP_BIG;
                        return false;
                    }
                    // a destination's edges follow one another: rows are in its order
                    const int e = ne + __popc(hits & ((1u << lane) - 1u));
                    if (first) c.S[s] = key;
                    if (hit) {
                        c.dsrc[e] = (I)s;
                        c.dw[e] = w;
                        c.list[e] = (I)(qd + node);  // the edge's destination, for now
                    }
                    ne += __popc(hits);
                    __syncwarp();
                    return true;
                });
                if (!go) return res;
            }
            qd += nb;
        } else if (qs < ns) {
            const int nb = min(ns - qs, 10);
            const unsigned key = c.S[qs + min(lane / 3, nb - 1)];
            const size_t h = key < (unsigned)L.cap_p ? (size_t)(t - 1) * L.cap_p + key : (size_t)(key - (unsigned)L.cap_p);
            const float y = __ldg(L.py + h), x = __ldg(L.px + h);
            unsigned a = 0;
            int n = 0;
            if (lane < 3 * nb) cell_row(L, t, lane % 3, y, x, &a, &n);
            const bool go = each_in_rows(a, n, 3 * nb, [&](int row, unsigned at) {
                const int from = max(row, 0) / 3 * 3;
                const float y1 = __shfl_sync(full, y, from), x1 = __shfl_sync(full, x, from);
                int i = 0;
                bool hit = false, smaller = false;
                if (row >= 0) {
                    const float2 p = __ldg(L.gpos + at);
                    float w;
                    i = __ldg(L.gidx + at);
                    hit = within_r(y1, x1, p.x, p.y, r, &w);
                    smaller = hit && i < d && (k == 0 || __ldcg(L.stamp + offt + i) == k);
                }
                if (__any_sync(full, smaller)) { res = COMP_SKIP; return false; }
                int q;
                bool first;
                if (!dt.put((unsigned)i, hit, c.cd, &nd, &q, &first)) { res = COMP_BIG; return false; }
                if (first) c.D[q] = i;
                __syncwarp();
                return true;
            });
            if (!go) return res;
            qs += nb;
        } else {
            break;
        }
    }
    __syncwarp();  // the tables' place is free
    // the destinations' lists (every destination has an edge, or it is alone)
    for (int e = lane; e < ne; e += 32)
        if (e == 0 || c.list[e - 1] != c.list[e]) c.doff[c.list[e]] = (I)e;
    if (lane == 0) {
        c.doff[0] = 0;
        c.doff[nd] = (I)ne;
    }
    for (int q = lane; q < nd; q += 32) c.vis[q] = 0;
    for (int s = lane; s < ns; s += 32) {
        c.used[s] = 0;
        c.soff[s] = 0;
    }
    __syncwarp();
    for (int e = lane; e < ne; e += 32) atomicAdd(c.soff + c.dsrc[e], 1);
    __syncwarp();
    // in ascending source order (linking.rs:310-315)
    for (int q = lane; q < nd; q += 32) {
        const int z0 = c.doff[q], z1 = c.doff[q + 1];
        for (int e = z0 + 1; e < z1; ++e) {
            const int s = c.dsrc[e];
            const float w = c.dw[e];
            const unsigned key = c.S[s];
            int z = e;
            for (; z > z0 && c.S[c.dsrc[z - 1]] > key; --z) {
                c.dsrc[z] = c.dsrc[z - 1];
                c.dw[z] = c.dw[z - 1];
            }
            c.dsrc[z] = (I)s;
            c.dw[z] = w;
        }
    }
    __syncwarp();
    // the sources' lists: starts, which the entries move on to the ends
    for (int s0 = 0, before = 0; s0 < ns; s0 += 32) {
        const int n = s0 + lane < ns ? c.soff[s0 + lane] : 0;
        int incl = n;
#pragma unroll
        for (int b = 1; b < 32; b <<= 1) {
            const int v = __shfl_up_sync(full, incl, b);
            if (lane >= b) incl += v;
        }
        if (s0 + lane < ns) c.soff[s0 + lane] = before + incl - n;
        before += __shfl_sync(full, incl, 31);
    }
    __syncwarp();
    for (int q = lane; q < nd; q += 32)
        for (int z = c.doff[q]; z < c.doff[q + 1]; ++z) c.list[atomicAdd(c.soff + c.dsrc[z], 1)] = (I)q;
    int low = INT_MAX;
    for (int q = lane; q < nd; q += 32) low = min(low, c.D[q]);
    low = __reduce_min_sync(full, low);
    int first = INT_MAX;
    for (int q = lane; q < nd; q += 32)
        if (c.D[q] == low) first = q;
    first = __reduce_min_sync(full, first);
    for (int q = lane; q < nd; q += 32) c.best[q] = -1;
    __syncwarp();
    if (lane == 0) {
        dfs_order(c, first, nd);
        if (!solve_subnet(c, nd, ns, L.budget, r * r)) atomicOr(L.err, ERR_SUBNET_BUDGET);
    }
    __syncwarp();
    // every source given up before any is taken
    auto source = [&](int q) { return c.best[q] < 0 ? -1 : (long long)c.S[c.best[q]]; };
    if (k > 0)
        for (int q = lane; q < nd; q += 32) give_up(L, source(q), offt + c.D[c.path[q]], t, k);
    __syncwarp();
    for (int q = lane; q < nd; q += 32) take_up(L, source(q), offt + c.D[c.path[q]], t, k);
    __syncwarp();
    return COMP_DONE;
}

// Links every destination of the window with M = {}.
__device__ void link_all(const LinkBufs& L, int tid, int nthr) {
    const int g1 = __ldg(L.off + L.te);
    for (int g = __ldg(L.off + L.tb) + tid; g < g1; g += nthr) {
        const int t = frame_of(L, g, L.tb, L.te);
        const int d = g - __ldg(L.off + t);
        SmallComp c;
        if (link_component(L, c, t, d) == COMP_BIG) L.seedq[push_slot(L.ctr + C_SEEDS)] = t * L.cap_p + d;
    }
}

// Resolves the components of pass k's seeds (k = 0: of those that link_all left),
// starting with a warp per block.
__device__ void link_seeds(const LinkBufs& L, WarpComp* wc, int k, int vw, int nwarp) {
    int* ctr = L.ctr + (k & 3) * NCTR;
    const int n = __ldcg(ctr + C_SEEDS);
    for (int q = vw; q < n; q += nwarp) {
        const int h = __ldcg(L.seedq + q);
        const int t = h / L.cap_p;
        if (link_component_warp(L, wc[threadIdx.x >> 5], t, h - t * L.cap_p, k) == COMP_BIG && (threadIdx.x & 31) == 0)
            L.deferq[push_slot(ctr + C_MEM)] = h;
        __syncwarp();
    }
}

// The components that do not fit a warp's registers: a warp per block with the
// block's arrays (`mem`).  Those that do not fit these are marked in the queue,
// for link_slots.  Movies begin at block *r.
__device__ void link_deferred(const LinkBufs& L, void* mem, int k, int* r) {
    int* ctr = L.ctr + (k & 3) * NCTR;
    const int n = __ldcg(ctr + C_MEM);
    const int b = (int)blockIdx.x - *r;
    *r = (*r + n) % (int)gridDim.x;
    if (threadIdx.x >= 32) return;
    const MemComp<unsigned short> c(mem, MID_N, MID_N, MID_E);
    for (int q = b < 0 ? b + (int)gridDim.x : b; q < n; q += gridDim.x) {
        const int h = __ldcg(L.deferq + q);
        const int t = h / L.cap_p;
        if (link_component_mem(L, c, t, h - t * L.cap_p, k) == COMP_BIG && threadIdx.x == 0) {
            L.deferq[q] = ~h;
            atomicAdd(ctr + C_SLOT, 1);
        }
        __syncwarp();
    }
}

// A warp per block and scratch slot.
__device__ void link_slots(const LinkBufs& L, int k) {
    int* ctr = L.ctr + (k & 3) * NCTR;
    const int n = __ldcg(ctr + C_MEM);
    if (threadIdx.x >= 32 || (int)blockIdx.x >= L.nslot) return;
    const MemComp<int> c(L.big + (size_t)blockIdx.x * L.big_ints, L.big_d, L.big_s, L.big_e);
    for (int q = blockIdx.x; q < n; q += min((int)gridDim.x, L.nslot)) {
        const int h = ~__ldcg(L.deferq + q);
        if (h < 0) continue;
        const int t = h / L.cap_p;
        if (link_component_mem(L, c, t, h - t * L.cap_p, k) == COMP_BIG) {
            // the host retries with larger slots; until the launch ends every
            // link of the frame must be a valid index
            if (threadIdx.x == 0) atomicOr(L.err, ERR_EDGE_OVERFLOW);
            if (k == 0)
                for (int g = __ldg(L.off + t) + threadIdx.x; g < __ldg(L.off + t + 1); g += 32) L.pred[g] = -1;
        }
        __syncwarp();
        if (threadIdx.x == 0) atomicAdd(ctr + C_DONE, 1);
    }
}

// Until the slots are done, asleep: the grid barrier's polling keeps emptying
// the L1 that a busy block on the same SM works from (lattices of 10 x 10 in
// slots 174 ms a call beside it, 52 beside sleepers).  The limit only ends the
// sleep: the barrier follows.
__device__ void wait_slots(const LinkBufs& L, int k) {
    const int* ctr = L.ctr + (k & 3) * NCTR;
    const int n = __ldcg(ctr + C_SLOT);
    const volatile int* done = ctr + C_DONE;
    if (threadIdx.x == 0)
        for (int i = 0; i < (1 << 24) && *done < n; ++i) __nanosleep(1000);
}

// A block's seeds on their way to the queue: one global atomic per block
// instead of one per few lanes (a million pushes to one counter took 0.6 ms).
constexpr int SEED_BUF = 1024;
struct SeedBuf {
    int n;
    int h[SEED_BUF];
};

// Empties the block's buffer into the movie's queue; every thread calls it.
__device__ __forceinline__ void flush_seeds(const LinkBufs& L, SeedBuf& sb, int k) {
    __shared__ int s_base;
    __syncthreads();
    const int n = min(sb.n, SEED_BUF);
    if (threadIdx.x == 0 && n > 0) s_base = atomicAdd(L.ctr + (k & 3) * NCTR + C_SEEDS, n);
    // every thread has read the count: the next movie's seeds may come in
    __syncthreads();
    if (n == 0) return;
    for (int i = threadIdx.x; i < n; i += NTL) L.seedq[s_base + i] = sb.h[i];
    if (threadIdx.x == 0) sb.n = 0;
    __syncthreads();
}

// Sets the bits `wm` of word w of the lanes' particles' membership (particle
// g of frame f; wm 0: none) to `bits`, and makes every destination in reach of
// a particle whose bits changed, in the frames where they did, a seed of pass
// k.  The warp takes one changed particle after the other, its cell rows in up
// to ten frames at once: neighbour searches and the stamps' atomics by single
// lanes left the others waiting (1.0 ms of the dense movie's pass 1).  Every
// lane calls it.
__device__ __forceinline__ void set_members(const LinkBufs& L, SeedBuf& sb, int g, int f, int w, unsigned wm,
                                            unsigned bits, int k) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned diff = 0;
    float gy = 0.f, gx = 0.f;
    if (wm) {
        unsigned* m = L.mm + (size_t)w * L.np + g;
        const unsigned old = __ldcg(m);
        diff = (old ^ bits) & wm;
        if (diff) {
            *m = old ^ diff;
            const size_t h = (size_t)f * L.cap_p + (g - __ldg(L.off + f));
            gy = __ldg(L.py + h);
            gx = __ldg(L.px + h);
        }
    }
    for (unsigned todo = __ballot_sync(full, diff != 0); todo; todo &= todo - 1) {
        const int b = __ffs(todo) - 1;
        const float y = __shfl_sync(full, gy, b), x = __shfl_sync(full, gx, b);
        const int t0 = __shfl_sync(full, f, b) + 2 + 32 * w;
        for (unsigned d = __shfl_sync(full, diff, b); d;) {
            // lanes 3 i .. 3 i + 2: the rows of the i-th changed frame
            const int nf = min(__popc(d), 10);
            unsigned rest = d;
            for (int q = 0; q < lane / 3 && rest; ++q) rest &= rest - 1;
            const int t = t0 + __ffs(rest) - 1;
            unsigned a = 0;
            int n = 0;
            if (lane < 3 * nf) cell_row(L, t, lane % 3, y, x, &a, &n);
            each_in_rows(a, n, 3 * nf, [&](int row, unsigned at) {
                const int tt = __shfl_sync(full, t, max(row, 0));
                if (row >= 0) {
                    const float2 p = __ldg(L.gpos + at);
                    float dist;
                    if (within_r(y, x, p.x, p.y, L.r, &dist)) {
                        const int i = __ldg(L.gidx + at), h = tt * L.cap_p + i;
                        if (atomicExch(L.stamp + __ldg(L.off + tt) + i, k) != k) {
                            const int slot = atomicAdd(&sb.n, 1);
                            if (slot < SEED_BUF) sb.h[slot] = h;
                            else L.seedq[push_slot(L.ctr + (k & 3) * NCTR + C_SEEDS)] = h;
                            if (__ldcg(L.fstamp + tt) != k && atomicExch(L.fstamp + tt, k) != k)
                                atomicAdd(L.ctr + (k & 3) * NCTR + C_FRAMES, 1);
                        }
                    }
                }
                __syncwarp();
                return true;
            });
            for (int q = 0; q < nf; ++q) d &= d - 1;
        }
    }
}

// Frames whose particles can be memory entries of the window start here.
__device__ __forceinline__ int first_member(const LinkBufs& L) { return max(0, L.tb - 1 - L.memory); }

// Membership for memory 1 or 2, without trajectory roots.
//
// With at most two memory lists no trajectory branches: a particle left
// unused by the next frame is a memory candidate for the next two frames
// only, and once it is linked as a memory entry its trajectory id is
// present in the following frame, which excludes it there.  So, with ids
// unique within a frame (every source links at most one destination):
//   - a frame t-2 particle unused by frame t-1 never shares its id with a
//     frame t-1 particle (memory links into t-1 come from frames t-4 and
//     t-3) nor with a frame t-3 candidate (neither descends from the
//     other, and a common ancestor would be a branch);
//   - a frame t-3 particle unused by frame t-2 shares its id with a frame
//     t-1 particle exactly when that particle's pred is it (it was linked
//     into t-1 as a memory entry): it has no descendant in t-2.
// linking.rs:244-259 (unused lists oldest first, index order within a
// list, dedupe by id against prev and among the entries) thus makes a
// particle an entry of the frame 2 later when the next frame does not link
// it, and of the frame 3 later when the one between does not either.
// Pass 1 checks every particle, later passes those whose linked bits the
// pass before changed.
__device__ void members_short(const LinkBufs& L, SeedBuf& sb, int k, int tid, int nthr) {
    const int fb = first_member(L);
    const int g0 = __ldg(L.off + fb);
    // pass 1: all, in order; later: spread over the grid's warps
    const int n = k == 1 ? __ldg(L.off + L.te) - g0 : __ldcg(L.ctr + ((k - 1) & 3) * NCTR + C_CHECKS);
    for (int i = tid; __any_sync(0xffffffffu, i < n); i += nthr) {
        int g = 0, f = 0;
        unsigned wm = 0, bits = 0;
        if (i < n) {
            g = k == 1 ? g0 + i : __ldcg(L.recq + i);
            f = frame_of(L, g, fb, L.te);
            const unsigned l = __ldcg(L.lnk + g);
            if (f + 2 >= L.tb && f + 2 < L.te) {
                wm |= 1u;
                if (!(l & 1u)) bits |= 1u;
            }
            if (L.memory == 2 && f + 3 >= L.tb && f + 3 < L.te) {
                wm |= 2u;
                if (!(l & 3u)) bits |= 2u;
            }
        }
        set_members(L, sb, g, f, 0, wm, bits, k);
    }
}

// Membership for memory >= 3.  Trajectories can branch (a particle relinked
// from an older memory entry), so ids are compared by trajectory root.  A
// particle unused by the next frame is an entry of frame t unless its id is
// present in frame t-1 or an older frame of the window holds an unused
// particle of the same id (linking.rs:244-259).  Pass 1 evaluates all
// particles.  Later passes take those of the trajectories that the pass
// before changed (the former root of every relinked destination and of its new
// source): a root, a membership or a list can only change within them, and
// they are complete, since every particle of a new trajectory comes from one
// of them.  In steps, a grid barrier between them:
//   members_find     the particles of those trajectories (from pass 2 on);
//   roots_local, roots_global  their roots;
//   members_chain    the unused particles in lists hashed by (root, block of
//                    2^fshift >= memory frames), so that a lookup meets only
//                    its own stretch of a trajectory (lists by root alone grow
//                    with the trajectories: 480 us a pass instead of 130 for
//                    200 frames of 15k particles);
//   members_present  every particle marks, in the list entries of its id at
//                    most `memory` frames before it, that the id is present
//                    in its frame;
//   members_long     the membership bits of every particle;
//   members_clear    the lists emptied for the next pass.
__device__ __forceinline__ int list_mask(const LinkBufs& L) {
    const int n = __ldg(L.off + L.te) - __ldg(L.off + first_member(L));
    return n <= 1 ? 0 : (1 << (32 - __clz(n - 1))) - 1;
}

__device__ __forceinline__ unsigned list_of(int root, int block) {
    return ((unsigned)root * 2654435761u + (unsigned)block * 0x9E3779B1u) >> 3;
}

// fn(frame, index) for the unused particles of id `root` in frames [f0, f1].
template <class F>
__device__ __forceinline__ void each_unused(const LinkBufs& L, int mask, int root, int f0, int f1, F&& fn) {
    for (int b = max(f0, 0) >> L.fshift; b <= f1 >> L.fshift; ++b)
        for (int c = __ldcg(L.head + (list_of(root, b) & mask)); c >= 0;) {
            const int4 e = __ldcg(L.ent + c);  // root, frame, next
            if (e.x == root && e.y >= f0 && e.y <= f1) fn(e.y, c);
            c = e.z;
        }
}

// The particles that pass k evaluates: number, and the i-th.
__device__ __forceinline__ int find_count(const LinkBufs& L, int k) {
    return k == 1 ? __ldg(L.off + L.te) - __ldg(L.off + first_member(L)) : __ldcg(L.ctr + (k & 3) * NCTR + C_CHECKS);
}

__device__ __forceinline__ int find_item(const LinkBufs& L, int k, int i) {
    return k == 1 ? __ldg(L.off + first_member(L)) + i : __ldcg(L.recq + i);
}

__device__ void members_find(const LinkBufs& L, int k, int tid, int nthr) {
    const int g1 = __ldg(L.off + L.te);
    for (int g = __ldg(L.off + first_member(L)) + tid; g < g1; g += nthr)
        if (__ldcg(L.cstamp + __ldcg(L.root + g)) == k) L.recq[push_slot(L.ctr + (k & 3) * NCTR + C_CHECKS)] = g;
}

__device__ void members_chain(const LinkBufs& L, int k, int tid, int nthr) {
    const int n = find_count(L, k), nw = (L.memory + 31) >> 5, mask = list_mask(L);
    for (int i = tid; i < n; i += nthr) {
        const int g = find_item(L, k, i), f = __ldcg(L.gframe + g);
        if (f > L.te - 3 || (__ldcg(L.lnk + g) & 1u)) continue;
        for (int w = 0; w < nw; ++w) L.pres[(size_t)w * L.np + g] = 0u;
        const int root = __ldcg(L.root + g);
        const int next = atomicExch(L.head + (list_of(root, f >> L.fshift) & mask), g);
        L.ent[g] = make_int4(root, f, next, 0);
    }
}

__device__ void members_present(const LinkBufs& L, int k, int tid, int nthr) {
    const int n = find_count(L, k), mask = list_mask(L);
    for (int i = tid; i < n; i += nthr) {
        const int g = find_item(L, k, i), f = __ldcg(L.gframe + g);
        if (f > L.te - 2) continue;
        each_unused(L, mask, __ldcg(L.root + g), f - L.memory, f - 1, [&](int fc, int c) {
            const int b = f - fc - 1;
            atomicOr(L.pres + (size_t)(b >> 5) * L.np + c, 1u << (b & 31));
        });
    }
}

__device__ void members_long(const LinkBufs& L, SeedBuf& sb, int k, int tid, int nthr) {
    const int n = find_count(L, k), nw = (L.memory + 31) >> 5, mask = list_mask(L);
    for (int i = tid; __any_sync(0xffffffffu, i < n); i += nthr) {
        const int g = i < n ? find_item(L, k, i) : 0;
        const int f = i < n ? __ldcg(L.gframe + g) : L.te;
        const bool cand = f <= L.te - 3 && !(__ldcg(L.lnk + g) & 1u);
        // distances j (frame f + 1 + j) inside the window
        const int j0 = max(1, L.tb - 1 - f);
        const int j1 = min(L.memory, L.te - 2 - f);
        // frame f + 1 + j's entries reach back to frame f + j - memory: an
        // older unused particle of the same id in them goes first
        int jmin = 0;
        if (cand)
            each_unused(L, mask, __ldcg(L.root + g), f + 1 - L.memory, f - 1,
                        [&](int fc, int) { jmin = max(jmin, fc - f + L.memory + 1); });
        for (int w = 0; w < nw; ++w) {
            // bits of the distances lo .. hi of this word
            const int lo = max(j0 - 32 * w - 1, 0), hi = min(j1 - 32 * w - 1, 31);
            const unsigned wm = lo <= hi ? (0xffffffffu >> (31 - hi)) & (0xffffffffu << lo) : 0u;
            const int lom = max(jmin - 32 * w - 1, 0);
            unsigned bits = cand && lom < 32 ? wm & (0xffffffffu << lom) : 0u;
            if (bits) bits &= ~__ldcg(L.pres + (size_t)w * L.np + g);
            set_members(L, sb, g, f, w, wm, bits, k);
        }
    }
}

__device__ void members_clear(const LinkBufs& L, int k, int tid, int nthr) {
    const int n = find_count(L, k), mask = list_mask(L);
    for (int i = tid; i < n; i += nthr) {
        const int g = find_item(L, k, i);
        L.head[list_of(__ldcg(L.root + g), __ldcg(L.gframe + g) >> L.fshift) & mask] = -1;
    }
}

// State of the window's particles before the first pass (earlier windows'
// is kept; their rstamp may hold a pass number of their own).
__device__ void window_begin(const LinkBufs& L, int tid, int nthr) {
    const int nw = (L.memory + 31) >> 5;
    const int fb = first_member(L);
    const int gb = __ldg(L.off + L.tb), g1 = __ldg(L.off + L.te);
    for (int g = __ldg(L.off + fb) + tid; g < g1; g += nthr) {
        L.rstamp[g] = 0;
        if (L.memory > 2) L.cstamp[g < gb ? __ldcg(L.root + g) : g] = 0;  // earlier windows' roots are final
        if (g < gb) continue;
        L.lnk[g] = 0u;
        L.stamp[g] = 0;
        for (int w = 0; w < nw; ++w) L.mm[(size_t)w * L.np + g] = 0u;
        if (L.memory > 2) L.gframe[g] = frame_of(L, g, L.tb, L.te);
    }
    if (L.memory > 2)
        for (int h = tid; h <= list_mask(L); h += nthr) L.head[h] = -1;
    for (int t = L.tb + tid; t < L.te; t += nthr) L.fstamp[t] = 0;
}

// Trajectory roots (the first particle of each trajectory, compact index),
// in two levels.  Compact indices run in frame order and a pred always
// points to an earlier particle, so a chain only ever steps to smaller
// indices.  The window's particles are cut into about sqrt(frames) chunks
// of consecutive indices:
//   roots_local:  every particle walks its pred chain while it stays inside
//                 its own chunk (at most the chunk's frame count of hops)
//                 and records where the chain enters the chunk (lroot);
//                 root[] is cleared meanwhile;
//   roots_global: every particle steps from chunk to chunk through
//                 lroot(pred(entry)) until a trajectory start, a particle of
//                 an earlier (final) window, or a root another thread has
//                 written -- at most the chunk count of hops.
// root[] only ever receives final values, so no barrier is needed between
// hops; a chain costs O(sqrt(frames)) dependent loads instead of O(frames).
__device__ __forceinline__ int root_chunk(const LinkBufs& L) {
    const int n = L.off[L.te] - L.off[L.tb];
    int nc = 1;
    while (nc * nc < L.te - L.tb) ++nc;
    return max(1, (n + nc - 1) / nc);
}

// fn(i) gives the i-th of n particles to resolve (those before the window
// are skipped); a particle's whole chain inside the window must be among them.
template <class F>
__device__ __forceinline__ void roots_local(const LinkBufs& L, int n, int tid, int nthr, F&& item) {
    const int g0 = __ldg(L.off + L.tb);
    const int cs = root_chunk(L);
    for (int i = tid; i < n; i += nthr) {
        const int g = item(i);
        if (g < g0) continue;
        const int cbeg = g0 + (g - g0) / cs * cs;
        int r = g;
        while (true) {
            const int p = __ldcg(L.pred + r);
            if (p < cbeg) break;
            r = p;
        }
        L.lroot[g] = r;
        L.root[g] = -1;
    }
}

template <class F>
__device__ __forceinline__ void roots_global(const LinkBufs& L, int n, int tid, int nthr, F&& item) {
    const int g0 = __ldg(L.off + L.tb);
    volatile int* root = L.root;
    for (int i = tid; i < n; i += nthr) {
        const int g = item(i);
        if (g < g0) continue;
        int r = __ldcg(L.lroot + g);
        while (true) {
            const int known = root[r];
            if (known >= 0) { r = known; break; }
            const int p = __ldcg(L.pred + r);
            if (p < 0) break;
            if (p < g0) { r = root[p]; break; }  // earlier window: final
            r = __ldcg(L.lroot + p);
        }
        root[g] = r;
    }
}

// rank of each new particle within its frame (linking.rs:470), a block per
// frame
__device__ void new_ranks(const LinkBufs& L) {
    __shared__ int warp_tot[NTL / 32];
    __shared__ int s_total;
    for (int t = L.tb + blockIdx.x; t < L.te; t += gridDim.x) {
        const int o = __ldg(L.off + t), n = __ldg(L.off + t + 1) - o;
        int base = 0;
        for (int i0 = 0; i0 < n; i0 += NTL) {
            const int i = i0 + threadIdx.x;
            const bool fresh = i < n && __ldcg(L.pred + o + i) < 0;
            const int pos = block_excl_scan<NTL>(fresh ? 1 : 0, warp_tot, &s_total);
            if (i < n) L.newrank[o + i] = fresh ? base + pos : -1;
            base += s_total;
            __syncthreads();
        }
        if (threadIdx.x == 0) L.newcount[t] = base;
    }
}

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// The linker over movies 0 .. nm - 1 (movie(m) gives the buffers): one grid
// barrier per phase serves them all.  A movie without seeds in a pass is at
// its fixed point (movies are independent) and later passes skip it.
// stat: [0..3] nanoseconds of the first linking, roots, memory entries and
// relinking (summed over passes, stamped by block 0 after each barrier);
// [4 + k - 1] frames with seeds in pass k <= 8.
template <class M>
__device__ __forceinline__ void link_fixpoint(const M& movie, int nm, int max_passes, int* passes,
                                              unsigned long long* stat) {
    __shared__ SeedBuf sb;
    // the warps' edges, then (a grid barrier between) a deferred component
    constexpr int WARP_BYTES = (int)sizeof(WarpComp) * (NTL / 32);
    __shared__ __align__(16) unsigned char buf[WARP_BYTES > MID_BYTES ? WARP_BYTES : MID_BYTES];
    if (threadIdx.x == 0) sb.n = 0;
    cg::grid_group grid = cg::this_grid();
    const int nthr = gridDim.x * NTL;
    const int tid0 = blockIdx.x * NTL + threadIdx.x;
    // few items: lane 0 of a warp in every block first
    const int vt0 = ((threadIdx.x & 31) * (NTL / 32) + (threadIdx.x >> 5)) * gridDim.x + blockIdx.x;
    const int vw0 = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;  // the same for warps
    const bool stamp = blockIdx.x == 0 && threadIdx.x == 0;
    unsigned long long t0 = stamp ? gtimer() : 0, acc[4] = {0, 0, 0, 0};
    auto tick = [&](int i) {
        if (stamp) { const unsigned long long t = gtimer(); acc[i] += t - t0; t0 = t; }
    };
    // a movie's items start on the threads after the previous movie's
    auto rot = [&](int id, int& r, const LinkBufs& L) {
        const int v = id - r < 0 ? id - r + nthr : id - r;
        r = (int)(((long long)r + __ldg(L.off + L.te) - __ldg(L.off + L.tb)) % nthr);
        return v;
    };
    bool any_mem = false, any_long = false;
    for (int m = 0; m < nm; ++m) {
        const int mem = movie(m).memory;
        any_mem |= mem > 0;
        any_long |= mem > 2;
    }
    if (any_mem) {
        int r = 0;
        for (int m = 0; m < nm; ++m) {
            const LinkBufs L = movie(m);
            const int id = rot(tid0, r, L);
            if (L.memory > 0) window_begin(L, id, nthr);
        }
        grid.sync();
    }
    {
        int r = 0;
        for (int m = 0; m < nm; ++m) {
            const LinkBufs L = movie(m);
            link_all(L, rot(tid0, r, L), nthr);
        }
    }
    grid.sync();
    auto any = [&](int k, int what) {
        bool b = false;
        for (int m = 0; m < nm; ++m) b |= __ldcg(movie(m).ctr + (k & 3) * NCTR + what) > 0;
        return b;
    };
    auto deferred = [&](int k) {
        if (!any(k, C_MEM)) return;
        int r = 0;
        for (int m = 0; m < nm; ++m) link_deferred(movie(m), buf, k, &r);
        grid.sync();
        if (!any(k, C_SLOT)) return;
        for (int m = 0; m < nm; ++m) link_slots(movie(m), k);
        for (int m = 0; m < nm; ++m) wait_slots(movie(m), k);
        grid.sync();
    };
    if (any(0, C_SEEDS)) {
        int r = 0;
        for (int m = 0; m < nm; ++m) {
            const LinkBufs L = movie(m);
            const int id = rot(vw0 * 32, r, L) >> 5;
            link_seeds(L, (WarpComp*)buf, 0, id, nthr >> 5);
        }
        grid.sync();
        deferred(0);
    }
    tick(0);
    int k = 0;
    if (any_mem) {
        auto active = [&](const LinkBufs& L, int kk) {
            return L.memory > 0 && L.te > 2 && (kk == 1 || __ldcg(L.ctr + ((kk - 1) & 3) * NCTR + C_SEEDS) > 0);
        };
        for (k = 1; k <= max_passes; ++k) {
            bool longs = false;
            if (any_long)
                for (int m = 0; m < nm; ++m) {
                    const LinkBufs L = movie(m);
                    longs |= L.memory > 2 && active(L, k);
                }
            if (longs) {
                auto each = [&](auto&& fn) {
                    for (int m = 0; m < nm; ++m) {
                        const LinkBufs L = movie(m);
                        if (L.memory > 2 && active(L, k)) fn(L);
                    }
                    grid.sync();
                };
                // many items in order (neighbours share cache lines), few spread
                auto order = [&](const LinkBufs& L) { return find_count(L, k) > nthr / 8 ? tid0 : vt0; };
                if (k > 1) each([&](const LinkBufs& L) { members_find(L, k, tid0, nthr); });
                each([&](const LinkBufs& L) {
                    roots_local(L, find_count(L, k), order(L), nthr, [&](int i) { return find_item(L, k, i); });
                });
                each([&](const LinkBufs& L) {
                    roots_global(L, find_count(L, k), order(L), nthr, [&](int i) { return find_item(L, k, i); });
                });
                tick(1);
                each([&](const LinkBufs& L) { members_chain(L, k, order(L), nthr); });
                each([&](const LinkBufs& L) { members_present(L, k, order(L), nthr); });
            }
            int r = 0;
            for (int m = 0; m < nm; ++m) {
                const LinkBufs L = movie(m);
                const int id = rot(vt0, r, L);
                // the counters of pass k + 1 were last read in pass k - 2
                if (stamp)
                    for (int q = 0; q < NCTR; ++q) L.ctr[((k + 1) & 3) * NCTR + q] = 0;
                if (!active(L, k)) continue;
                if (L.memory <= 2) members_short(L, sb, k, k == 1 ? tid0 : id, nthr);
                else members_long(L, sb, k, find_count(L, k) > nthr / 8 ? tid0 : id, nthr);
                flush_seeds(L, sb, k);
            }
            grid.sync();
            int total = 0;
            for (int m = 0; m < nm; ++m) total += __ldcg(movie(m).ctr + (k & 3) * NCTR + C_SEEDS);
            tick(2);
            if (stamp && k <= 8) {
                unsigned long long nf = 0;
                for (int m = 0; m < nm; ++m) nf += (unsigned)__ldcg(movie(m).ctr + (k & 3) * NCTR + C_FRAMES);
                stat[4 + k - 1] += nf;
            }
            if (total == 0) break;
            r = 0;
            for (int m = 0; m < nm; ++m) {
                const LinkBufs L = movie(m);
                const int id = rot(vw0 * 32, r, L) >> 5;
                if (!active(L, k)) continue;
                if (L.memory > 2) members_clear(L, k, tid0, nthr);
                link_seeds(L, (WarpComp*)buf, k, id, nthr >> 5);
            }
            grid.sync();
            deferred(k);
            tick(3);
        }
    }
    for (int m = 0; m < nm; ++m) {
        const LinkBufs L = movie(m);
        const int g0 = __ldg(L.off + L.tb);
        roots_local(L, __ldg(L.off + L.te) - g0, tid0, nthr, [&](int i) { return g0 + i; });
        new_ranks(L);
    }
    grid.sync();
    for (int m = 0; m < nm; ++m) {
        const LinkBufs L = movie(m);
        const int g0 = __ldg(L.off + L.tb);
        roots_global(L, __ldg(L.off + L.te) - g0, tid0, nthr, [&](int i) { return g0 + i; });
    }
    if (stamp) {
        acc[1] += gtimer() - t0;
        *passes = max(*passes, k);  // several launches (frame windows) add up
        for (int i = 0; i < 4; ++i) stat[i] += acc[i];
    }
}
}  // namespace

// One movie (or one frame window of it) in one cooperative launch.
__global__ void __launch_bounds__(NTL, 4) link_fixpoint_kernel(const __grid_constant__ LinkBufs L, int max_passes,
                                                               int* passes, unsigned long long* stat) {
    link_fixpoint([&](int) -> const LinkBufs& { return L; }, 1, max_passes, passes, stat);
}

// Several movies in one cooperative launch (the batched path).
__global__ void __launch_bounds__(NTL, 4) link_fixpoint_multi_kernel(const LinkBufs* Ls, int nm, int max_passes,
                                                                     int* passes, unsigned long long* stat) {
    link_fixpoint([&](int m) { return Ls[m]; }, nm, max_passes, passes, stat);
}

cudaError_t link_blocks_per_sm(bool multi, int* per_sm) {
    const void* fn = multi ? (const void*)link_fixpoint_multi_kernel : (const void*)link_fixpoint_kernel;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, fn, NTL, 0);
}

cudaError_t launch_link(const LinkBufs& L, int max_passes, int* passes, unsigned long long* stat, int grid,
                        cudaStream_t st) {
    LinkBufs a = L;
    void* args[] = {&a, &max_passes, &passes, &stat};
    return cudaLaunchCooperativeKernel((const void*)link_fixpoint_kernel, dim3(grid), dim3(NTL), args, 0, st);
}

cudaError_t launch_link_multi(const LinkBufs* d_L, int nm, int max_passes, int* passes, unsigned long long* stat,
                              int grid, cudaStream_t st) {
    void* args[] = {&d_L, &nm, &max_passes, &passes, &stat};
    return cudaLaunchCooperativeKernel((const void*)link_fixpoint_multi_kernel, dim3(grid), dim3(NTL), args, 0, st);
}

}  // namespace gt
