// bvh_build.cu -- device binned-SAH build, collapsed to 8-wide quantised nodes.
//
// Replaces BVH8::Create / SplitSAH (src/s3d_bvh8.cpp:254-342,401-479), which splits a
// range three binary levels deep with a 16-bucket SAH on the longest centroid axis and
// recurses on the CPU.  Here:
//   1. a binary tree: 32 bins on each of the three centroid axes, cost = ntrav*SA(node) +
//      nL*SA(L) + nR*SA(R) against count*SA(node) for a leaf (the reference's cost form,
//      src/s3d_bvh8.cpp:300-317; ntrav is 0.3 by default instead of its 1, since small
//      leaves trace fastest here), leaves of at most 3 triangles.  Ranges of more than
//      kSub primitives are split breadth first by all blocks (k_top_bin, k_top_split,
//      k_top_partition); a smaller range's whole subtree, with its costs for the collapse,
//      is built by one block in shared memory (k_subtree).  Measured (GB300, 1M-triangle soup,
//      rebuild + 262,144 rays): 25.5 ms with every level as passes over all primitives and a
//      host round trip, 2.5 ms so; bound by latency in the subtrees (0.88 ms) and by the 12
//      top levels' passes (0.61 ms), which read and write the 32 MB of records from L2;
//   2. the binary tree is collapsed into 8-wide nodes: dynamic programming over the binary
//      tree picks the SAH-cheapest choice of wide nodes, leaves (subtrees of up to three
//      triangles) and opened nodes; the wide nodes are then written top down;
//   3. child boxes are quantised to 8 bits per plane against a per-node power-of-two
//      grid, rounding outward, so every quantised box contains the exact one.
#include <cfloat>
#include <cmath>

#include <algorithm>
#include <atomic>
#include <cstring>

#include "internal.h"

namespace salty {
namespace {

constexpr int kBins = 32;
// SAH weights of the collapse: one 8-wide node visit against one triangle test.  Measured
// on the traversal microbenchmark and the 1080p heightfield (GB300): any triangle weight
// from 1 to 2.6 node visits gives the same speed within noise, lighter ones put more
// triangles in each leaf and lose 3-10 %.
constexpr float kCollapseNodeCost = 1.0f;
constexpr float kCollapseTriCost = 2.0f;
constexpr size_t kKeepBuildBytes = 512ull << 20;
constexpr int kSub = 512;        // primitives of a subtree built by one block
constexpr int kChunk = 2048;     // primitives of a work item of the top levels
constexpr int kTopThreads = 256;
constexpr int kMaxLevels = 4096;
constexpr int kBinWords = 3 * kBins * 7;  // count + lo[3] + hi[3] per bin per axis

__device__ __forceinline__ int f2o(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// Primitives move as 32-byte records, (box lo, primitive index) (box hi, unused), so that
// every pass over a range reads and writes it in order.  The centroid is recomputed from
// the box (BoundingBox::center, include/s3d_math.h:2178-2183).
struct Rec {
    float lo[3], hi[3];
    int id;
    __device__ __forceinline__ float cen(int a) const { return (lo[a] + hi[a]) * 0.5f; }
};
__device__ __forceinline__ Rec load_rec(const float4* __restrict__ r, int p) {
    const float4 a = r[2 * p], b = r[2 * p + 1];
    return Rec{{a.x, a.y, a.z}, {b.x, b.y, b.z}, __float_as_int(a.w)};
}
__device__ __forceinline__ void store_rec(float4* __restrict__ r, int p, const Rec& q) {
    r[2 * p] = make_float4(q.lo[0], q.lo[1], q.lo[2], __int_as_float(q.id));
    r[2 * p + 1] = make_float4(q.hi[0], q.hi[1], q.hi[2], 0.0f);
}

// A range of more than kSub primitives, split by all blocks.
struct Top {
    int node, first, count;
    int cmin[3], cmax[3];         // ordered-int centroid bounds
    int axis, split, nleft;       // axis -1: median split by position
    int child[2];                 // the children's tasks of the next level, -1: a subtree
    int cursor[2];
};

// A range of at most kSub primitives: x = first position, y = binary node, z = count |
// record buffer << 15, w = level.
using SubTask = int4;

struct Counters {
    int ntop[2];      // tasks of the even / odd levels
    int nitem[2];     // their work items (task, chunk)
    int nsub;         // subtrees
    int ticket;       // subtrees taken
    int splits;       // binary splits (inner nodes)
    int depth;        // binary levels
    int ntris;        // leaf triangles written
    int error;        // set when a partition slot falls outside its range
    double sah;       // accumulated SAH numerator
    int rootbox[6];   // ordered-int bounds of all primitive boxes
    int rootcen[6];   // ordered-int bounds of all centroids
};

// Binary node numbering: a split at primitive position s (the right child's first) gives its
// node the children 2s - 1 and 2s.  Split positions are unique, so no node is allocated and
// the numbers do not depend on scheduling; the root is node 0.
__device__ __forceinline__ int child_pair(int split_pos) { return 2 * split_pos - 1; }

__device__ __forceinline__ void store_bnode(BNode* nodes, int id, const float* lo, const float* hi, int a, int count) {
    float4* d = reinterpret_cast<float4*>(nodes + id);
    d[0] = make_float4(lo[0], lo[1], lo[2], __int_as_float(a));
    d[1] = make_float4(hi[0], hi[1], hi[2], __int_as_float(count));
}

__device__ __forceinline__ int bin_of(float c, float cmin, float cmax, int B) {
    float ext = cmax - cmin;
    if (!(ext > 0.0f)) return 0;
    float k = (float)B / ext;
    int b = (int)((c - cmin) * k);
    return min(max(b, 0), B - 1);
}

__device__ __forceinline__ float area(float dx, float dy, float dz) {
    dx = fmaxf(dx, 0.0f); dy = fmaxf(dy, 0.0f); dz = fmaxf(dz, 0.0f);
    return 2.0f * (dx * dy + dx * dz + dy * dz);
}
__device__ __forceinline__ float box_area(const float* lo, const float* hi) {
    return area(hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]);
}

__device__ __forceinline__ int empty_bin_word(int i) {
    const int w = i % 7;
    return w == 0 ? 0 : (w <= 3 ? f2o(FLT_MAX) : f2o(-FLT_MAX));
}

// ---------------------------------------------------------------- setup
// Records of all primitives and the bounds of their boxes and centroids: reduced per block,
// one set of atomics per block (one per warp serialised on the same twelve words).
__global__ void __launch_bounds__(256) k_prim_setup(const float* __restrict__ pos, int n, float4* __restrict__ rec,
                                                    Counters* ctr) {
    __shared__ int sb[12];
    if (threadIdx.x < 12) sb[threadIdx.x] = (threadIdx.x % 6) < 3 ? f2o(FLT_MAX) : f2o(-FLT_MAX);
    __syncthreads();
    float v[12];
    for (int a = 0; a < 3; ++a) { v[a] = v[6 + a] = FLT_MAX; v[3 + a] = v[9 + a] = -FLT_MAX; }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* p = pos + (size_t)i * 9;
        Rec r;
        r.id = i;
        for (int a = 0; a < 3; ++a) {
            r.lo[a] = fminf(p[a], fminf(p[3 + a], p[6 + a]));
            r.hi[a] = fmaxf(p[a], fmaxf(p[3 + a], p[6 + a]));
            const float c = r.cen(a);
            v[a] = fminf(v[a], r.lo[a]);
            v[3 + a] = fmaxf(v[3 + a], r.hi[a]);
            v[6 + a] = fminf(v[6 + a], c);
            v[9 + a] = fmaxf(v[9 + a], c);
        }
        store_rec(rec, i, r);
    }
    for (int k = 0; k < 12; ++k) {
        const bool mn = k % 6 < 3;
        const int w = mn ? __reduce_min_sync(0xffffffffu, f2o(v[k])) : __reduce_max_sync(0xffffffffu, f2o(v[k]));
        if ((threadIdx.x & 31) == 0) {
            if (mn) atomicMin(&sb[k], w);
            else atomicMax(&sb[k], w);
        }
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        int* g = threadIdx.x < 6 ? &ctr->rootbox[threadIdx.x] : &ctr->rootcen[threadIdx.x - 6];
        if (threadIdx.x % 6 < 3) atomicMin(g, sb[threadIdx.x]);
        else atomicMax(g, sb[threadIdx.x]);
    }
}

// The root, as a task of level 0 or as the only subtree.
__global__ void k_root_init(Counters* ctr, Top* tops, int2* items, int* bins, SubTask* subs, int* lvl_off, BNode* nodes,
                            int n) {
    const int nitem = (n + kChunk - 1) / kChunk;
    for (int i = threadIdx.x; i < nitem; i += blockDim.x) items[i] = make_int2(0, i);
    for (int i = threadIdx.x; i < kBinWords; i += blockDim.x) bins[i] = empty_bin_word(i);
    if (threadIdx.x != 0) return;
    float lo[3], hi[3];
    for (int a = 0; a < 3; ++a) { lo[a] = o2f(ctr->rootbox[a]); hi[a] = o2f(ctr->rootbox[3 + a]); }
    store_bnode(nodes, 0, lo, hi, 0, 0);
    lvl_off[0] = 0;
    if (n <= kSub) {
        subs[0] = make_int4(0, 0, n, 0);
        ctr->nsub = 1;
        lvl_off[1] = 0;
        return;
    }
    Top t;
    t.node = 0; t.first = 0; t.count = n;
    for (int a = 0; a < 3; ++a) { t.cmin[a] = ctr->rootcen[a]; t.cmax[a] = ctr->rootcen[3 + a]; }
    t.axis = t.split = t.nleft = 0;
    t.child[0] = t.child[1] = -1;
    t.cursor[0] = t.cursor[1] = 0;
    tops[0] = t;
    ctr->ntop[0] = 1;
    ctr->nitem[0] = nitem;
}

// ---------------------------------------------------------------- top levels
// Bins a chunk of one task in shared memory and adds it to the task's bins.
__global__ void __launch_bounds__(kTopThreads)
k_top_bin(int level, const float4* __restrict__ rec, const Top* __restrict__ tops, const int2* __restrict__ items,
          int* __restrict__ bins, int B, Counters* ctr) {
    __shared__ int sb[kBinWords];
    const int par = level & 1, nitem = ctr->nitem[par];
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr->ntop[par ^ 1] = ctr->nitem[par ^ 1] = 0;  // the next level's lists
    for (int it = blockIdx.x; it < nitem; it += gridDim.x) {
        const int2 item = items[it];
        const Top& tk = tops[item.x];
        float cmin[3], cmax[3];
        for (int a = 0; a < 3; ++a) { cmin[a] = o2f(tk.cmin[a]); cmax[a] = o2f(tk.cmax[a]); }
        const int p0 = tk.first + item.y * kChunk, p1 = min(tk.first + tk.count, p0 + kChunk);
        for (int i = threadIdx.x; i < kBinWords; i += kTopThreads) sb[i] = empty_bin_word(i);
        __syncthreads();
        for (int p = p0 + threadIdx.x; p < p1; p += kTopThreads) {
            const Rec r = load_rec(rec, p);
            for (int a = 0; a < 3; ++a) {
                int* s = sb + (a * kBins + bin_of(r.cen(a), cmin[a], cmax[a], B)) * 7;
                atomicAdd(s, 1);
                for (int k = 0; k < 3; ++k) {
                    atomicMin(s + 1 + k, f2o(r.lo[k]));
                    atomicMax(s + 4 + k, f2o(r.hi[k]));
                }
            }
        }
        __syncthreads();
        int* g = bins + (size_t)item.x * kBinWords;
        for (int i = threadIdx.x; i < kBinWords; i += kTopThreads) {
            const int w = i % 7;
            if (sb[i - w] == 0) continue;
            if (w == 0) atomicAdd(g + i, sb[i]);
            else if (w <= 3) atomicMin(g + i, sb[i]);
            else atomicMax(g + i, sb[i]);
        }
        __syncthreads();
    }
}

struct BuildParams {
    int B;
    int max_leaf;
    float trav_cost;
};

// The cheapest split of a range from its bins (one warp; bin `lane` of each axis): axis -1
// when no bin boundary separates the range.  Ties go to the lower axis, then the lower bin.
struct Split {
    float cost;
    int axis, bin, nl;
    float llo[3], lhi[3], rlo[3], rhi[3];
};
__device__ __forceinline__ Split best_split(const int* g, int B, int lane) {
    constexpr unsigned m = 0xffffffffu;
    Split s;
    s.cost = INFINITY;
    s.axis = s.bin = -1;
    s.nl = 0;
    for (int a = 0; a < 3; ++a) {
        int cnt = 0;
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        if (lane < B) {
            const int* e = g + (a * kBins + lane) * 7;
            cnt = e[0];
            for (int k = 0; k < 3; ++k) { lo[k] = o2f(e[1 + k]); hi[k] = o2f(e[4 + k]); }
        }
        // inclusive prefix (left) and suffix (right)
        int lc = cnt, rc = cnt;
        float llo[3], lhi[3], rlo[3], rhi[3];
        for (int k = 0; k < 3; ++k) { llo[k] = rlo[k] = lo[k]; lhi[k] = rhi[k] = hi[k]; }
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(m, lc, off), w = __shfl_down_sync(m, rc, off);
            if (lane >= off) lc += v;
            if (lane + off < 32) rc += w;
            for (int k = 0; k < 3; ++k) {
                const float a1 = __shfl_up_sync(m, llo[k], off), a2 = __shfl_up_sync(m, lhi[k], off);
                const float b1 = __shfl_down_sync(m, rlo[k], off), b2 = __shfl_down_sync(m, rhi[k], off);
                if (lane >= off) { llo[k] = fminf(llo[k], a1); lhi[k] = fmaxf(lhi[k], a2); }
                if (lane + off < 32) { rlo[k] = fminf(rlo[k], b1); rhi[k] = fmaxf(rhi[k], b2); }
            }
        }
        // split after bin `lane`: left = prefix[lane], right = suffix[lane + 1]
        const int nr = __shfl_down_sync(m, rc, 1);
        float srlo[3], srhi[3];
        for (int k = 0; k < 3; ++k) {
            srlo[k] = __shfl_down_sync(m, rlo[k], 1);
            srhi[k] = __shfl_down_sync(m, rhi[k], 1);
        }
        const bool ok = (lane < B - 1) && lc > 0 && nr > 0;
        float mc = ok ? (float)lc * box_area(llo, lhi) + (float)nr * box_area(srlo, srhi) : INFINITY;
        int ml = lane;
        for (int off = 16; off > 0; off >>= 1) {
            const float oc = __shfl_xor_sync(m, mc, off);
            const int ol = __shfl_xor_sync(m, ml, off);
            if (oc < mc || (oc == mc && ol < ml)) { mc = oc; ml = ol; }
        }
        if (mc < s.cost) {
            s.cost = mc;
            s.axis = a;
            s.bin = ml;
            s.nl = __shfl_sync(m, lc, ml);
            for (int k = 0; k < 3; ++k) {
                s.llo[k] = __shfl_sync(m, llo[k], ml);
                s.lhi[k] = __shfl_sync(m, lhi[k], ml);
                s.rlo[k] = __shfl_sync(m, srlo[k], ml);
                s.rhi[k] = __shfl_sync(m, srhi[k], ml);
            }
        }
    }
    return s;
}

// Splits the tasks of one level (one warp each) and hands their children on: to the next
// level's tasks, with work items and empty bins, or to the subtrees.
constexpr int kSplitWarps = 4;
__global__ void __launch_bounds__(kSplitWarps * 32)
k_top_split(int level, Top* __restrict__ tops, Top* __restrict__ tops_next, const int* __restrict__ bins,
            int* __restrict__ bins_next, int2* __restrict__ items_next, SubTask* __restrict__ subs, BNode* nodes,
            int* __restrict__ hist, int* __restrict__ lvl_off, int B, Counters* ctr) {
    const int par = level & 1, ntop = ctr->ntop[par], off = lvl_off[level];
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        lvl_off[level + 1] = off + ntop;
        if (ntop > 0) atomicAdd(&ctr->splits, ntop);
    }
    for (int t = blockIdx.x * kSplitWarps + (threadIdx.x >> 5); t < ntop; t += gridDim.x * kSplitWarps) {
        Top& tk = tops[t];
        const int node = tk.node, first = tk.first, count = tk.count;
        Split s = best_split(bins + (size_t)t * kBinWords, B, lane);
        if (s.axis < 0) {  // all centroids in one bin: halves by position, each with the whole box
            s.nl = count / 2;
            for (int k = 0; k < 3; ++k) {
                s.llo[k] = s.rlo[k] = nodes[node].lo[k];
                s.lhi[k] = s.rhi[k] = nodes[node].hi[k];
            }
        }
        const int pair = child_pair(first + s.nl);
        int child[2] = {-1, -1};
        for (int c = 0; c < 2; ++c) {
            const int cf = c ? first + s.nl : first, cc = c ? count - s.nl : s.nl;
            if (cc <= kSub) {
                if (lane == 0) subs[atomicAdd(&ctr->nsub, 1)] = make_int4(cf, pair + c, cc | ((par ^ 1) << 15), level + 1);
                continue;
            }
            const int ni = (cc + kChunk - 1) / kChunk;
            int slot = 0, i0 = 0;
            if (lane == 0) {
                slot = atomicAdd(&ctr->ntop[par ^ 1], 1);
                i0 = atomicAdd(&ctr->nitem[par ^ 1], ni);
                Top n;
                n.node = pair + c; n.first = cf; n.count = cc;
                for (int k = 0; k < 3; ++k) { n.cmin[k] = f2o(FLT_MAX); n.cmax[k] = f2o(-FLT_MAX); }
                n.axis = n.split = n.nleft = 0;
                n.child[0] = n.child[1] = -1;
                n.cursor[0] = n.cursor[1] = 0;
                tops_next[slot] = n;
            }
            slot = __shfl_sync(0xffffffffu, slot, 0);
            i0 = __shfl_sync(0xffffffffu, i0, 0);
            child[c] = slot;
            for (int i = lane; i < ni; i += 32) items_next[i0 + i] = make_int2(slot, i);
            for (int i = lane; i < kBinWords; i += 32) bins_next[(size_t)slot * kBinWords + i] = empty_bin_word(i);
        }
        if (lane == 0) {
            tk.axis = s.axis;
            tk.split = s.bin;
            tk.nleft = s.nl;
            tk.child[0] = child[0];
            tk.child[1] = child[1];
            nodes[node].a = pair;
            nodes[node].count = 0;
            store_bnode(nodes, pair, s.llo, s.lhi, 0, 0);
            store_bnode(nodes, pair + 1, s.rlo, s.rhi, 0, 0);
            hist[off + t] = node;
        }
    }
}

// Moves a chunk's records to their children's ranges in the other buffer: ranks from ballots,
// one cursor atomic per side and block; the centroid bounds of children that are split further
// are reduced per block (per-lane atomics on the two children's bounds made this pass 15.7 of
// a 23.6 ms build of 1M triangles).
__global__ void __launch_bounds__(kTopThreads)
k_top_partition(int level, const float4* __restrict__ rec, float4* __restrict__ rec_next, Top* __restrict__ tops,
                Top* __restrict__ tops_next, const int2* __restrict__ items, int B, Counters* ctr) {
    constexpr int K = kChunk / kTopThreads, W = kTopThreads / 32;
    __shared__ int wl[W], wr[W], base[2], sb[12];
    const int par = level & 1, nitem = ctr->nitem[par];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int it = blockIdx.x; it < nitem; it += gridDim.x) {
        const int2 item = items[it];
        Top& tk = tops[item.x];
        const int first = tk.first, count = tk.count, nleft = tk.nleft, axis = tk.axis, split = tk.split;
        const int ch[2] = {tk.child[0], tk.child[1]};
        float cmin = 0.0f, cmax = 0.0f;
        if (axis >= 0) { cmin = o2f(tk.cmin[axis]); cmax = o2f(tk.cmax[axis]); }
        const int p0 = first + item.y * kChunk, p1 = min(first + count, p0 + kChunk);
        if (threadIdx.x < 12) sb[threadIdx.x] = (threadIdx.x % 6) < 3 ? f2o(FLT_MAX) : f2o(-FLT_MAX);
        Rec r[K];
        unsigned side = 0;  // bit k: record k goes right
        int nl = 0, nr = 0;
        float b[2][6];
        for (int c = 0; c < 2; ++c)
            for (int a = 0; a < 3; ++a) { b[c][a] = FLT_MAX; b[c][3 + a] = -FLT_MAX; }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int p = p0 + k * kTopThreads + threadIdx.x;
            const bool in = p < p1;
            bool right = false;
            if (in) {
                r[k] = load_rec(rec, p);
                right = axis < 0 ? p - first >= nleft
                                 : bin_of((axis == 0 ? r[k].cen(0) : (axis == 1 ? r[k].cen(1) : r[k].cen(2))), cmin, cmax, B) > split;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float c = r[k].cen(a);
                    if (right) { b[1][a] = fminf(b[1][a], c); b[1][3 + a] = fmaxf(b[1][3 + a], c); }
                    else { b[0][a] = fminf(b[0][a], c); b[0][3 + a] = fmaxf(b[0][3 + a], c); }
                }
            }
            if (right) side |= 1u << k;
            nl += __popc(__ballot_sync(0xffffffffu, in && !right));
            nr += __popc(__ballot_sync(0xffffffffu, in && right));
        }
        if (lane == 0) { wl[warp] = nl; wr[warp] = nr; }
        __syncthreads();
        if (threadIdx.x < 2) {
            int t = 0;
            for (int w = 0; w < W; ++w) t += threadIdx.x ? wr[w] : wl[w];
            base[threadIdx.x] = (threadIdx.x ? first + nleft : first) + atomicAdd(&tk.cursor[threadIdx.x], t);
        }
        for (int c = 0; c < 2; ++c)
            if (ch[c] >= 0)
                for (int a = 0; a < 6; ++a) {
                    const int v = a < 3 ? __reduce_min_sync(0xffffffffu, f2o(b[c][a]))
                                        : __reduce_max_sync(0xffffffffu, f2o(b[c][a]));
                    if (lane == 0) {
                        if (a < 3) atomicMin(&sb[c * 6 + a], v);
                        else atomicMax(&sb[c * 6 + a], v);
                    }
                }
        __syncthreads();
        if (threadIdx.x < 12 && ch[threadIdx.x / 6] >= 0) {
            Top& cn = tops_next[ch[threadIdx.x / 6]];
            const int a = threadIdx.x % 6;
            if (a < 3) atomicMin(&cn.cmin[a], sb[threadIdx.x]);
            else atomicMax(&cn.cmax[a - 3], sb[threadIdx.x]);
        }
        int ol = base[0], orr = base[1];
        for (int w = 0; w < warp; ++w) { ol += wl[w]; orr += wr[w]; }
        const int lim = first + nleft, end = first + count;
        bool bad = false;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const bool in = p0 + k * kTopThreads + (int)threadIdx.x < p1, right = (side >> k) & 1u;
            const unsigned ml = __ballot_sync(0xffffffffu, in && !right), mr = __ballot_sync(0xffffffffu, in && right);
            const unsigned lt = (1u << lane) - 1u;
            if (in) {
                const int np = right ? orr + __popc(mr & lt) : ol + __popc(ml & lt);
                // binning and partition disagree: report, never write out of range
                if (np < (right ? lim : first) || np >= (right ? end : lim)) bad = true;
                else store_rec(rec_next, np, r[k]);
            }
            ol += __popc(ml);
            orr += __popc(mr);
        }
        if (bad) atomicOr(&ctr->error, 1);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- collapse + quantise
__device__ __forceinline__ float bnode_area(const BNode& b) { return box_area(b.lo, b.hi); }

// Per-axis power-of-two grid: the smallest e >= -126 with 255 * 2^e >= hi - lo.  255 * 2^e is
// a float, so the exact difference can be replaced by its rounding up.
__device__ int quant_exponent(float lo, float hi) {
    float x = __fsub_ru(hi, lo);
    if (!(x > 0.0f)) return -126;
    int up = 0;
    if (isinf(x)) { x = __fsub_ru(0.5f * hi, 0.5f * lo); up = 1; }
    const int bits = __float_as_int(x), k = (bits >> 23) - 127 + up;  // x = m 2^k, 1 <= m < 2 (k = -127: denormal)
    const int e = (bits & 0x7fffff) <= 0x7f0000 ? k - 7 : k - 6;     // m <= 255/128
    return e < -126 ? -126 : e;
}

// ---------------------------------------------------------------- SAH-optimal collapse
// Which binary nodes become 8-wide nodes, which become leaves of the wide tree, and which
// are opened into their parent's child slots is decided by dynamic programming over the
// binary tree (Ylitie, Karras, Laine, "Efficient Incoherent Ray Traversal on GPUs Through
// Compressed Wide BVHs", HPG 2017, section 3.1): for every binary node n and every
// i = 1..7, C(n, i) is the least SAH cost of covering n's subtree with at most i roots, each
// an 8-wide node or a leaf of at most kMaxLeafTris triangles:
//   C(n, 1)  = min(leaf: A(n) p(n) c_tri  if p(n) <= kMaxLeafTris,
//                  node: A(n) c_node + D(n, 8))
//   C(n, i)  = min(C(n, i - 1), D(n, i))                           i = 2..7
//   D(n, j)  = min over k = 1..j-1 of C(left, k) + C(right, j - k)
// with A the surface area and p the triangle count.  Binary leaves can only be leaves.
// The nodes of one binary level are solved together, deepest level first.
struct CollapseDP {
    float c[7];          // C(n, 1..7)
    int first, count;    // the subtree's triangles: prim positions [first, first + count)
    unsigned dec;        // bit 0: C(n, 1) is a leaf; bits 1..6: C(n, i) takes D(n, i), i = 2..7;
                         // bits 8 + 3 (j - 2): the k of D(n, j), j = 2..8
};

__device__ __forceinline__ CollapseDP dp_leaf(float A, int first, int count, float c_tri) {
    CollapseDP r;
    r.first = first;
    r.count = count;
    const float leaf = A * (float)count * c_tri;
    for (int k = 0; k < 7; ++k) r.c[k] = leaf;
    r.dec = 1u;
    return r;
}

__device__ __forceinline__ CollapseDP dp_inner(float A, const CollapseDP& L, const CollapseDP& R, float c_node,
                                               float c_tri) {
    CollapseDP r;
    r.first = min(L.first, R.first);
    r.count = L.count + R.count;
    float D[9];
    unsigned dec = 0;
#pragma unroll
    for (int j = 2; j <= 8; ++j) {
        float best = INFINITY;
        int bk = 1;
#pragma unroll
        for (int k = 1; k < j; ++k) {
            const int kr = j - k;
            if (k > 7 || kr > 7) continue;
            const float v = L.c[k - 1] + R.c[kr - 1];
            if (v < best) { best = v; bk = k; }
        }
        D[j] = best;
        dec |= (unsigned)bk << (8 + 3 * (j - 2));
    }
    const float node = A * c_node + D[8];
    const float leaf = r.count <= kMaxLeafTris ? A * (float)r.count * c_tri : INFINITY;
    if (leaf <= node) { r.c[0] = leaf; dec |= 1u; }
    else r.c[0] = node;
#pragma unroll
    for (int k = 2; k <= 7; ++k) {
        if (D[k] < r.c[k - 2]) { r.c[k - 1] = D[k]; dec |= 1u << (k - 1); }
        else r.c[k - 1] = r.c[k - 2];
    }
    r.dec = dec;
    return r;
}

// The top levels' nodes, deepest level first (one block; the subtrees' roots are solved).
__global__ void __launch_bounds__(1024) k_top_dp(const BNode* __restrict__ bn, CollapseDP* dp, const int* __restrict__ hist,
                                                 const int* __restrict__ lvl_off, int levels, float c_node, float c_tri) {
    for (int l = levels - 1; l >= 0; --l) {
        for (int i = lvl_off[l] + threadIdx.x; i < lvl_off[l + 1]; i += blockDim.x) {
            const int id = hist[i];
            const BNode b = bn[id];
            dp[id] = dp_inner(bnode_area(b), dp[b.a], dp[b.a + 1], c_node, c_tri);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- subtrees
// The whole binary subtree of a range of at most kSub primitives, by one block: the records
// stay in shared memory, index lists are split level by level.  A range of more than 16
// primitives takes a warp and its 32 bins per axis; smaller ones take 16 or 8 lanes, one per
// primitive: lane i tries the split after its own bin (the only bins where the two sides
// change), which finds the same split as the bins do.  Then the costs of the collapse, deepest
// level first.  Building every level of 1M triangles with passes over all primitives took
// 23.1 ms of kernels; the levels below this size are one launch of 0.87 ms here.  Bound: the
// latency of shared-memory chains (issue 52 % at 16 warps per SM; 64 or 96 threads, five or six
// blocks per SM, and all warps on a level's one or two large ranges are no faster).
constexpr int kSubThreads = 128;
constexpr int kSubWarps = kSubThreads / 32;
constexpr unsigned short kNoLevel = 0xffff;

struct SubShared {
    float lo[3][kSub], hi[3][kSub];
    int id[kSub];
    int self[kSub];                     // node split at local position s (its right child's first)
    int qid[2][3][kSub / 2];            // nodes to split, by level parity and size class
    unsigned qfc[2][3][kSub / 2];       // first | count << 16
    unsigned short idx[2][kSub];        // index lists, by level parity
    unsigned short lev[kSub];           // level of self[s], kNoLevel: no split there
    int bins[kSubWarps][kBinWords];
    int nq[2][3];
    int ticket, splits, depth;
};

struct SubArgs {
    const float4* rec[2];
    const SubTask* subs;
    BNode* nodes;
    CollapseDP* dp;
    int* prim;      // primitive index by position
    Counters* ctr;
    BuildParams prm;
    float c_node, c_tri;
};

__device__ __forceinline__ int size_class(int count) { return count <= 8 ? 0 : (count <= 16 ? 1 : 2); }

// A range that is not split further: its primitives in their final positions.
__device__ __forceinline__ void sub_leaf(const SubArgs& A, int id, int pos, int count, float sa) {
    A.nodes[id].a = pos;
    A.nodes[id].count = count;
    A.dp[id] = dp_leaf(sa, pos, count, A.c_tri);
}

// Records a split found for node `id` = local range [f, f + c) and hands the children on (one
// lane): single primitives become leaves, the rest joins the next level's lists.
__device__ __forceinline__ void sub_split(const SubArgs& A, SubShared& S, int id, int first, int f, int c, int level,
                                          const float* llo, const float* lhi, const float* rlo, const float* rhi,
                                          int nl) {
    const int s = f + nl, pair = child_pair(first + s), par = (level & 1) ^ 1;
    A.nodes[id].a = pair;
    A.nodes[id].count = 0;
    S.self[s] = id;
    S.lev[s] = (unsigned short)level;
    atomicAdd(&S.splits, 1);
    atomicMax(&S.depth, level + 2);
    for (int k = 0; k < 2; ++k) {
        const int cf = k ? s : f, cc = k ? c - nl : nl;
        const float *lo = k ? rlo : llo, *hi = k ? rhi : lhi;
        if (cc == 1) {
            store_bnode(A.nodes, pair + k, lo, hi, first + cf, 1);
            A.dp[pair + k] = dp_leaf(box_area(lo, hi), first + cf, 1, A.c_tri);
        } else {
            store_bnode(A.nodes, pair + k, lo, hi, 0, 0);
            const int cls = size_class(cc), q = atomicAdd(&S.nq[par][cls], 1);
            S.qid[par][cls][q] = pair + k;
            S.qfc[par][cls][q] = (unsigned)cf | ((unsigned)cc << 16);
        }
    }
}

// Ranges of up to G primitives, one lane each.
template <int G>
__device__ __forceinline__ void sub_small(const SubArgs& A, SubShared& S, int cls, int first, int level) {
    const int par = level & 1, nq = S.nq[par][cls];
    const int lane = threadIdx.x & 31, gl = lane % G, g0 = lane - gl;
    const unsigned gm = (G == 32 ? 0xffffffffu : (1u << G) - 1u) << g0;
    const int B = A.prm.B;
    for (int k = threadIdx.x / G; k < nq; k += kSubThreads / G) {
        const int id = S.qid[par][cls][k];
        const unsigned fc = S.qfc[par][cls][k];
        const int f = (int)(fc & 0xffffu), c = (int)(fc >> 16);
        const bool act = gl < c;
        const int q = S.idx[par][f + (act ? gl : 0)];
        float lo[3], hi[3], cn[3];
        int b[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = S.lo[a][q];
            hi[a] = S.hi[a][q];
            cn[a] = (lo[a] + hi[a]) * 0.5f;
            float mn = cn[a], mx = cn[a];
            for (int o = G / 2; o > 0; o >>= 1) {
                mn = fminf(mn, __shfl_xor_sync(gm, mn, o));
                mx = fmaxf(mx, __shfl_xor_sync(gm, mx, o));
            }
            b[a] = bin_of(cn[a], mn, mx, B);
        }
        float blo[3], bhi[3];  // the node's box, for the leaf's cost
        for (int a = 0; a < 3; ++a) { blo[a] = FLT_MAX; bhi[a] = -FLT_MAX; }
        float L[3][6], R[3][6];
        int lc[3] = {0, 0, 0};
        for (int a = 0; a < 3; ++a)
            for (int e = 0; e < 3; ++e) {
                L[a][e] = R[a][e] = FLT_MAX;
                L[a][3 + e] = R[a][3 + e] = -FLT_MAX;
            }
        for (int j = 0; j < c; ++j) {
            const int bj[3] = {__shfl_sync(gm, b[0], g0 + j), __shfl_sync(gm, b[1], g0 + j), __shfl_sync(gm, b[2], g0 + j)};
            float l[3], h[3];
            for (int e = 0; e < 3; ++e) {
                l[e] = __shfl_sync(gm, lo[e], g0 + j);
                h[e] = __shfl_sync(gm, hi[e], g0 + j);
                blo[e] = fminf(blo[e], l[e]);
                bhi[e] = fmaxf(bhi[e], h[e]);
            }
            for (int a = 0; a < 3; ++a) {
                const bool left = bj[a] <= b[a];
                lc[a] += left ? 1 : 0;
                for (int e = 0; e < 3; ++e) {
                    L[a][e] = fminf(L[a][e], left ? l[e] : FLT_MAX);
                    L[a][3 + e] = fmaxf(L[a][3 + e], left ? h[e] : -FLT_MAX);
                    R[a][e] = fminf(R[a][e], left ? FLT_MAX : l[e]);
                    R[a][3 + e] = fmaxf(R[a][3 + e], left ? -FLT_MAX : h[e]);
                }
            }
        }
        float cost = INFINITY;
        int key = 1 << 20;  // axis * 32 + bin; ties go to the lowest
        for (int a = 0; a < 3; ++a) {
            const int rc = c - lc[a];
            const float v = act && rc > 0 ? (float)lc[a] * box_area(L[a], L[a] + 3) + (float)rc * box_area(R[a], R[a] + 3)
                                          : INFINITY;
            if (v < cost) { cost = v; key = a * 32 + b[a]; }
        }
        const int own = key;
        for (int o = G / 2; o > 0; o >>= 1) {
            const float oc = __shfl_xor_sync(gm, cost, o);
            const int ok = __shfl_xor_sync(gm, key, o);
            if (oc < cost || (oc == cost && ok < key)) { cost = oc; key = ok; }
        }
        const float sa = box_area(blo, bhi);
        const float leaf_cost = (float)c * sa, split_cost = A.prm.trav_cost * sa + cost;
        const bool can = cost < INFINITY;
        const bool leaf = c <= A.prm.max_leaf && (leaf_cost <= split_cost || !can);
        if (leaf) {
            if (gl == 0) sub_leaf(A, id, first + f, c, sa);
            if (act) A.prim[first + f + gl] = S.id[q];
            continue;
        }
        int nl = c / 2;
        bool right = gl >= nl;
        if (can) {
            const int ax = key >> 5, bin = key & 31;
            right = (ax == 0 ? b[0] : (ax == 1 ? b[1] : b[2])) > bin;
        }
        const unsigned mr = __ballot_sync(gm, act && right) & gm, ml = __ballot_sync(gm, act && !right) & gm;
        if (can) nl = __popc(ml);
        if (act) {
            const unsigned lt = (1u << lane) - 1u;
            const int np = right ? f + nl + __popc(mr & lt) : f + __popc(ml & lt);
            S.idx[par ^ 1][np] = (unsigned short)q;
            if (right ? c - nl == 1 : nl == 1) A.prim[first + np] = S.id[q];
        }
        if (!can) {
            if (gl == 0) sub_split(A, S, id, first, f, c, level, blo, bhi, blo, bhi, nl);
        } else {
            // the lowest lane whose own best is the winner holds the children's boxes
            const unsigned win = __ballot_sync(gm, act && own == key) & gm;
            if (lane == __ffs(win) - 1) {
                const int ax = key >> 5;
                float llo[3], lhi[3], rlo[3], rhi[3];
                for (int e = 0; e < 3; ++e) {
                    llo[e] = ax == 0 ? L[0][e] : (ax == 1 ? L[1][e] : L[2][e]);
                    lhi[e] = ax == 0 ? L[0][3 + e] : (ax == 1 ? L[1][3 + e] : L[2][3 + e]);
                    rlo[e] = ax == 0 ? R[0][e] : (ax == 1 ? R[1][e] : R[2][e]);
                    rhi[e] = ax == 0 ? R[0][3 + e] : (ax == 1 ? R[1][3 + e] : R[2][3 + e]);
                }
                sub_split(A, S, id, first, f, c, level, llo, lhi, rlo, rhi, nl);
            }
        }
    }
}

// Ranges of more than 16 primitives (above max_leaf, so always split), one warp each.
__device__ __forceinline__ void sub_large(const SubArgs& A, SubShared& S, int first, int level) {
    constexpr unsigned m = 0xffffffffu;
    const int par = level & 1, nq = S.nq[par][2], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int B = A.prm.B;
    int* bins = S.bins[warp];
    for (int k = warp; k < nq; k += kSubWarps) {
        const int id = S.qid[par][2][k];
        const unsigned fc = S.qfc[par][2][k];
        const int f = (int)(fc & 0xffffu), c = (int)(fc >> 16);
        float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (int i = lane; i < c; i += 32) {
            const int q = S.idx[par][f + i];
            for (int a = 0; a < 3; ++a) {
                const float cn = (S.lo[a][q] + S.hi[a][q]) * 0.5f;
                mn[a] = fminf(mn[a], cn);
                mx[a] = fmaxf(mx[a], cn);
            }
        }
        for (int a = 0; a < 3; ++a) {
            mn[a] = o2f(__reduce_min_sync(m, f2o(mn[a])));
            mx[a] = o2f(__reduce_max_sync(m, f2o(mx[a])));
        }
        __syncwarp();
        for (int i = lane; i < kBinWords; i += 32) bins[i] = empty_bin_word(i);
        __syncwarp();
        for (int i = lane; i < c; i += 32) {
            const int q = S.idx[par][f + i];
            const float lo[3] = {S.lo[0][q], S.lo[1][q], S.lo[2][q]}, hi[3] = {S.hi[0][q], S.hi[1][q], S.hi[2][q]};
            for (int a = 0; a < 3; ++a) {
                int* e = bins + (a * kBins + bin_of((lo[a] + hi[a]) * 0.5f, mn[a], mx[a], B)) * 7;
                atomicAdd(e, 1);
                for (int j = 0; j < 3; ++j) {
                    atomicMin(e + 1 + j, f2o(lo[j]));
                    atomicMax(e + 4 + j, f2o(hi[j]));
                }
            }
        }
        __syncwarp();
        Split s = best_split(bins, B, lane);
        if (s.axis < 0) {  // all centroids in one bin: halves by position, each with the whole box
            s.nl = c / 2;
            for (int a = 0; a < 3; ++a) {
                float l = FLT_MAX, h = -FLT_MAX;
                for (int i = lane; i < c; i += 32) {
                    const int q = S.idx[par][f + i];
                    l = fminf(l, S.lo[a][q]);
                    h = fmaxf(h, S.hi[a][q]);
                }
                s.llo[a] = s.rlo[a] = o2f(__reduce_min_sync(m, f2o(l)));
                s.lhi[a] = s.rhi[a] = o2f(__reduce_max_sync(m, f2o(h)));
            }
        }
        int ol = f, orr = f + s.nl;
        for (int i0 = 0; i0 < c; i0 += 32) {
            const int i = i0 + lane;
            const bool in = i < c;
            const int q = in ? S.idx[par][f + i] : 0;
            bool right = false;
            if (in) {
                if (s.axis < 0) {
                    right = i >= s.nl;
                } else {
                    const float cn = s.axis == 0 ? (S.lo[0][q] + S.hi[0][q]) * 0.5f
                                                 : (s.axis == 1 ? (S.lo[1][q] + S.hi[1][q]) * 0.5f
                                                                : (S.lo[2][q] + S.hi[2][q]) * 0.5f);
                    const float lo = s.axis == 0 ? mn[0] : (s.axis == 1 ? mn[1] : mn[2]);
                    const float hi = s.axis == 0 ? mx[0] : (s.axis == 1 ? mx[1] : mx[2]);
                    right = bin_of(cn, lo, hi, B) > s.bin;
                }
            }
            const unsigned ml = __ballot_sync(m, in && !right), mr = __ballot_sync(m, in && right);
            const unsigned lt = (1u << lane) - 1u;
            if (in) {
                const int np = right ? orr + __popc(mr & lt) : ol + __popc(ml & lt);
                S.idx[par ^ 1][np] = (unsigned short)q;
                if (right ? c - s.nl == 1 : s.nl == 1) A.prim[first + np] = S.id[q];
            }
            ol += __popc(ml);
            orr += __popc(mr);
        }
        if (lane == 0) sub_split(A, S, id, first, f, c, level, s.llo, s.lhi, s.rlo, s.rhi, s.nl);
    }
}

__global__ void __launch_bounds__(kSubThreads) k_subtree(const SubArgs A) {
    extern __shared__ __align__(16) unsigned char sub_smem[];
    SubShared& S = *reinterpret_cast<SubShared*>(sub_smem);
    const int tid = threadIdx.x;
    const int nsub = A.ctr->nsub;
    for (;;) {
        __syncthreads();
        if (tid == 0) S.ticket = atomicAdd(&A.ctr->ticket, 1);
        __syncthreads();
        const int t = S.ticket;
        if (t >= nsub) return;
        const SubTask task = A.subs[t];
        const int first = task.x, root = task.y, m = task.z & 0x7fff;
        const float4* rec = A.rec[task.z >> 15];
        for (int i = tid; i < m; i += kSubThreads) {
            const Rec r = load_rec(rec, first + i);
            for (int a = 0; a < 3; ++a) { S.lo[a][i] = r.lo[a]; S.hi[a][i] = r.hi[a]; }
            S.id[i] = r.id;
            S.idx[0][i] = (unsigned short)i;
            S.lev[i] = kNoLevel;
        }
        if (tid < 6) (&S.nq[0][0])[tid] = 0;
        if (tid == 0) {
            S.splits = 0;
            S.depth = 1;
        }
        __syncthreads();
        if (tid == 0) {
            if (m == 1) {
                const BNode b = A.nodes[root];
                sub_leaf(A, root, first, 1, bnode_area(b));
                A.prim[first] = S.id[0];
            } else {
                const int cls = size_class(m);
                S.qid[0][cls][0] = root;
                S.qfc[0][cls][0] = (unsigned)m << 16;
                S.nq[0][cls] = 1;
            }
        }
        __syncthreads();
        int level = 0;
        for (;; ++level) {
            const int par = level & 1;
            if (S.nq[par][0] + S.nq[par][1] + S.nq[par][2] == 0) break;
            sub_large(A, S, first, level);
            sub_small<16>(A, S, 1, first, level);
            sub_small<8>(A, S, 0, first, level);
            __syncthreads();
            if (tid < 3) S.nq[par][tid] = 0;
            __syncthreads();
        }
        // every level splits or ends each of its ranges, so a subtree has at most kSub - 1 of them
        for (int l = level - 1; l >= 0; --l) {
            for (int s = 1 + tid; s < m; s += kSubThreads) {
                if (S.lev[s] != (unsigned short)l) continue;
                const int id = S.self[s], pair = child_pair(first + s);
                const BNode b = A.nodes[id];
                A.dp[id] = dp_inner(bnode_area(b), A.dp[pair], A.dp[pair + 1], A.c_node, A.c_tri);
            }
            __syncthreads();
        }
        if (tid == 0) {
            if (S.splits) atomicAdd(&A.ctr->splits, S.splits);
            atomicMax(&A.ctr->depth, task.w + S.depth);
        }
    }
}

// The children of the 8-wide node made from binary node `bid`: D(bid, 8) unfolded.  Each
// child is a binary node standing for itself (leaf[] tells whether as a leaf of the wide
// tree or as an 8-wide node).  Returns the number of children (1..8).
__device__ int collapse_children(const BNode* __restrict__ bn, const CollapseDP* __restrict__ dp, int bid,
                                 int* set, bool* leaf) {
    int k = 0;
    if (bn[bid].count > 0) {  // a binary leaf at the root: one leaf child
        set[0] = bid;
        leaf[0] = true;
        return 1;
    }
    int sn[16], sj[16], sp = 0;
    sn[sp] = bid; sj[sp] = 8; ++sp;
    bool top = true;
    while (sp > 0) {
        --sp;
        const int m = sn[sp];
        int j = sj[sp];
        const BNode b = bn[m];
        const unsigned dec = dp[m].dec;
        if (!top) {
            if (b.count > 0) { set[k] = m; leaf[k] = true; ++k; continue; }
            while (j > 1 && j <= 7 && !((dec >> (j - 1)) & 1u)) --j;  // C(m, j) = C(m, j - 1)
            if (j == 1) { set[k] = m; leaf[k] = (dec & 1u) != 0; ++k; continue; }
        }
        top = false;
        const int kl = (dec >> (8 + 3 * (j - 2))) & 7u;
        sn[sp] = b.a + 1; sj[sp] = j - kl; ++sp;  // right, visited after left
        sn[sp] = b.a; sj[sp] = kl; ++sp;
    }
    return k;
}

// One level of the wide tree, one thread per node.  The level's nodes are out[off8[level] ..]
// and work[..] names their binary nodes; their children follow them in out, counted in
// cnt8[level + 1].  Quantisation is exact in FP32: a plane's grid index is the floor (ceiling)
// of (plane - origin) / 2^e, every index of 8 bits times 2^e is a float, so rounding the
// difference down (up) first cannot move it across an index; where the quotient is so small that
// it rounds to zero, the ceiling of a positive difference is still one (64-bit divisions took half
// of this kernel: 1.11 -> 0.41 ms for 1M triangles, with one atomic per warp instead of per node).
__global__ void __launch_bounds__(128) k_collapse(int level, const BNode* __restrict__ bn, const int* __restrict__ work,
                                                  Bvh8Node* __restrict__ out, float4* __restrict__ tris,
                                                  const int* __restrict__ prim, const float* __restrict__ pos,
                                                  int* __restrict__ work_next, int* __restrict__ cnt8,
                                                  int* __restrict__ off8, Counters* ctr,
                                                  const CollapseDP* __restrict__ dp) {
    const int nwork = cnt8[level], out0 = off8[level];
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0) off8[level + 1] = out0 + nwork;
    for (int w0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); w0 < nwork; w0 += gridDim.x * blockDim.x) {
        const int wi = w0 + lane;
        const bool act = wi < nwork;
        int set[8];
        bool as_leaf[8];
        int k = 0;
        BNode b;
        if (act) {
            const int bid = work[wi];
            b = bn[bid];
            k = collapse_children(bn, dp, bid, set, as_leaf);
        }
        int n_int = 0, n_tri = 0;
        for (int i = 0; i < k; ++i) {
            if (!as_leaf[i]) ++n_int; else n_tri += dp[set[i]].count;
        }
        // one allocation per warp for the children and the leaf triangles
        int si = n_int, st = n_tri;
        for (int o = 1; o < 32; o <<= 1) {
            const int a1 = __shfl_up_sync(0xffffffffu, si, o), a2 = __shfl_up_sync(0xffffffffu, st, o);
            if (lane >= o) { si += a1; st += a2; }
        }
        int ci = 0, ct = 0;
        if (lane == 31) {
            if (si) ci = atomicAdd(&cnt8[level + 1], si);
            if (st) ct = atomicAdd(&ctr->ntris, st);
        }
        const int child0 = __shfl_sync(0xffffffffu, ci, 31) + si - n_int;  // within the next level
        const int tri_base = __shfl_sync(0xffffffffu, ct, 31) + st - n_tri;
        const int child_base = out0 + nwork + child0;
        double sah = 0.0;
        if (act) {
            // slot assignment by octant of the child centre around the node centre
            const float cx = (b.lo[0] + b.hi[0]) * 0.5f, cy = (b.lo[1] + b.hi[1]) * 0.5f, cz = (b.lo[2] + b.hi[2]) * 0.5f;
            int slot_child[8];
            for (int s = 0; s < 8; ++s) slot_child[s] = -1;
            // place larger children first so they get their preferred slot
            int order[8];
            float osa[8];
            for (int i = 0; i < k; ++i) { order[i] = i; osa[i] = bnode_area(bn[set[i]]); }
            for (int i = 1; i < k; ++i) {
                int o = order[i]; float s = osa[o]; int j = i - 1;
                while (j >= 0 && osa[order[j]] < s) { order[j + 1] = order[j]; --j; }
                order[j + 1] = o;
            }
            for (int ii = 0; ii < k; ++ii) {
                int i = order[ii];
                BNode c = bn[set[i]];
                int pref = (((c.lo[0] + c.hi[0]) * 0.5f > cx) ? 1 : 0) | (((c.lo[1] + c.hi[1]) * 0.5f > cy) ? 2 : 0) |
                           (((c.lo[2] + c.hi[2]) * 0.5f > cz) ? 4 : 0);
                int bs = -1, bd = 99;
                for (int s = 0; s < 8; ++s) {
                    if (slot_child[s] >= 0) continue;
                    int d = __popc(s ^ pref);
                    if (d < bd) { bd = d; bs = s; }
                }
                slot_child[bs] = i;
            }
            int ex[3];
            float inv[3];
            for (int a = 0; a < 3; ++a) {
                ex[a] = quant_exponent(b.lo[a], b.hi[a]);
                inv[a] = __int_as_float((127 - ex[a]) << 23);  // 2^-e
            }
            unsigned char qlo[3][8], qhi[3][8], meta[8];
            unsigned imask = 0;
            int r_int = 0, off = 0;
            sah = (double)bnode_area(b);
            for (int s = 0; s < 8; ++s) {
                meta[s] = 0;
                int i = slot_child[s];
                if (i < 0) {
                    for (int a = 0; a < 3; ++a) { qlo[a][s] = 255; qhi[a][s] = 0; }
                    continue;
                }
                BNode c = bn[set[i]];
                for (int a = 0; a < 3; ++a) {
                    const float lo = floorf(__fsub_rd(c.lo[a], b.lo[a]) * inv[a]);
                    const float up = __fsub_ru(c.hi[a], b.lo[a]);
                    const float hi = fmaxf(ceilf(up * inv[a]), up > 0.0f ? 1.0f : 0.0f);
                    qlo[a][s] = (unsigned char)fminf(fmaxf(lo, 0.0f), 255.0f);
                    qhi[a][s] = (unsigned char)fminf(fmaxf(hi, 0.0f), 255.0f);
                }
                // a leaf child holds the triangles of its whole binary subtree
                c.a = dp[set[i]].first;
                c.count = as_leaf[i] ? dp[set[i]].count : 0;
                if (c.count == 0) {
                    imask |= 1u << s;
                    meta[s] = (unsigned char)((1u << 5) | (24u + s));  // one hit bit at 24 + slot
                    work_next[child0 + r_int++] = set[i];
                } else {
                    // unary triangle count in the top three bits, first triangle in the low five
                    meta[s] = (unsigned char)((((1u << c.count) - 1u) << 5) | off);
                    for (int j = 0; j < c.count; ++j) {
                        int q = prim[c.a + j];
                        const float* p = pos + (size_t)q * 9;
                        float4* dst = tris + (size_t)(tri_base + off + j) * kTriFloat4;
                        dst[0] = make_float4(p[0], p[1], p[2], __int_as_float(q));
                        dst[1] = make_float4(p[3], p[4], p[5], 0.0f);
                        dst[2] = make_float4(p[6], p[7], p[8], 0.0f);
                    }
                    off += c.count;
                    sah += (double)c.count * (double)bnode_area(c);
                }
            }
            Bvh8Node nd;
            nd.w[0] = make_uint4(__float_as_uint(b.lo[0]), __float_as_uint(b.lo[1]), __float_as_uint(b.lo[2]),
                                 (unsigned)(ex[0] + 127) | ((unsigned)(ex[1] + 127) << 8) |
                                     ((unsigned)(ex[2] + 127) << 16) | (imask << 24));
            auto pack4 = [](const unsigned char* v) {
                return (unsigned)v[0] | ((unsigned)v[1] << 8) | ((unsigned)v[2] << 16) | ((unsigned)v[3] << 24);
            };
            nd.w[1] = make_uint4((unsigned)(n_int ? child_base : 0), (unsigned)(n_tri ? tri_base : 0), pack4(meta),
                                 pack4(meta + 4));
            nd.w[2] = make_uint4(pack4(qlo[0]), pack4(qlo[0] + 4), pack4(qlo[1]), pack4(qlo[1] + 4));
            nd.w[3] = make_uint4(pack4(qlo[2]), pack4(qlo[2] + 4), pack4(qhi[0]), pack4(qhi[0] + 4));
            nd.w[4] = make_uint4(pack4(qhi[1]), pack4(qhi[1] + 4), pack4(qhi[2]), pack4(qhi[2] + 4));
            out[out0 + wi] = nd;
        }
        for (int o = 16; o > 0; o >>= 1) sah += __shfl_xor_sync(0xffffffffu, sah, o);
        if (lane == 0) atomicAdd(&ctr->sah, sah);
    }
}

__global__ void k_init_counters(Counters* c) {
    Counters z;
    memset(&z, 0, sizeof(z));
    for (int a = 0; a < 3; ++a) {
        z.rootbox[a] = f2o(FLT_MAX); z.rootbox[3 + a] = f2o(-FLT_MAX);
        z.rootcen[a] = f2o(FLT_MAX); z.rootcen[3 + a] = f2o(-FLT_MAX);
    }
    *c = z;
}

__global__ void k_fill_one(int* p) { *p = 1; }

inline unsigned grid_for(long long n, int block) { return (unsigned)((n + block - 1) / block); }

inline float host_o2f(int i) {
    i = i >= 0 ? i : i ^ 0x7fffffff;
    float f;
    std::memcpy(&f, &i, 4);
    return f;
}

}  // namespace

static salty_status build_scene(salty_ctx* ctx, salty_scene* sc, const salty_build_opts& opts) {
    if (sc->n_inst > 0) return build_instanced(ctx, sc, opts);
    if (sc->n_sph > 0) return build_with_spheres(ctx, sc, opts);
    if (sc->n_tris <= 0) return ctx->err.fail(SALTY_ERR_INVALID_ARG, "scene has no triangles");
    if (sc->n_tris > (int64_t)0x3fffffff)
        return ctx->err.fail(SALTY_ERR_CAPACITY, "too many triangles (%lld)", (long long)sc->n_tris);
    float box[6];
    return build_bvh_tris(ctx, sc->pos.p, (int)sc->n_tris, opts, sc->bvh, box);
}

// The workspace outlives a build only for a scene that is built again (a changing scene), and
// goes with that scene: a scene built once leaves nothing behind.
salty_status build_bvh(salty_ctx* ctx, salty_scene* sc, const salty_build_opts& opts) {
    const bool again = sc->bvh.generation != 0;
    const salty_status s = build_scene(ctx, sc, opts);
    if (again && s == SALTY_OK) ctx->build_ws_owner = sc;
    if (!ctx->build_ws_owner) ctx->build_ws.release();
    return s;
}

salty_status build_bvh_tris(salty_ctx* ctx, const float* d_pos, int n, const salty_build_opts& opts, Bvh& out,
                            float root_box[6]) {
    auto& E = ctx->err;
    if (n <= 0) return E.fail(SALTY_ERR_INVALID_ARG, "no triangles to build a BVH over");
    BuildParams prm;
    prm.B = opts.bins;
    prm.max_leaf = opts.max_leaf;
    prm.trav_cost = opts.trav_cost;
    cudaStream_t st = ctx->stream;

    // Workspace: one allocation, carved up; up to kKeepBuildBytes (about 2M triangles) the
    // context's (build_bvh), a larger one is given back at the end.
    const size_t max_top = (size_t)n / (kSub + 1) + 2;  // tasks of one top level
    const size_t max_item = (size_t)n / kChunk + 1 + max_top;
    size_t total = 0;
    auto part = [&](size_t bytes) {
        const size_t o = total;
        total += (bytes + 255) / 256 * 256;
        return o;
    };
    const size_t o_ctr = part(sizeof(Counters));
    const size_t o_lvl = part((kMaxLevels + 2) * sizeof(int)), o_cnt8 = part((kMaxLevels + 2) * sizeof(int)),
                 o_off8 = part((kMaxLevels + 2) * sizeof(int));
    size_t o_rec[2], o_top[2], o_item[2], o_bins[2], o_work[2];
    for (int i = 0; i < 2; ++i) {
        o_rec[i] = part((size_t)n * 2 * sizeof(float4));
        o_top[i] = part(max_top * sizeof(Top));
        o_item[i] = part(max_item * sizeof(int2));
        o_bins[i] = part(max_top * kBinWords * sizeof(int));
        o_work[i] = part((size_t)n * sizeof(int));
    }
    const size_t o_sub = part((size_t)n * sizeof(SubTask)), o_hist = part((size_t)n * sizeof(int)),
                 o_prim = part((size_t)n * sizeof(int)), o_bn = part((size_t)2 * n * sizeof(BNode)),
                 o_dp = part((size_t)2 * n * sizeof(CollapseDP));
    DevBuf<unsigned char> once;
    DevBuf<unsigned char>& ws = total <= kKeepBuildBytes ? ctx->build_ws : once;
    SALTY_TRY_CUDA(E, ws.ensure(total));
    auto at = [&](size_t o) { return ws.p + o; };
    Counters* ctr = reinterpret_cast<Counters*>(at(o_ctr));
    int *lvl_off = reinterpret_cast<int*>(at(o_lvl)), *cnt8 = reinterpret_cast<int*>(at(o_cnt8)),
        *off8 = reinterpret_cast<int*>(at(o_off8));
    float4* rec[2];
    Top* tops[2];
    int2* items[2];
    int *bins[2], *work[2];
    for (int i = 0; i < 2; ++i) {
        rec[i] = reinterpret_cast<float4*>(at(o_rec[i]));
        tops[i] = reinterpret_cast<Top*>(at(o_top[i]));
        items[i] = reinterpret_cast<int2*>(at(o_item[i]));
        bins[i] = reinterpret_cast<int*>(at(o_bins[i]));
        work[i] = reinterpret_cast<int*>(at(o_work[i]));
    }
    SubTask* subs = reinterpret_cast<SubTask*>(at(o_sub));
    int *hist = reinterpret_cast<int*>(at(o_hist)), *prim = reinterpret_cast<int*>(at(o_prim));
    BNode* bnodes = reinterpret_cast<BNode*>(at(o_bn));
    CollapseDP* dp = reinterpret_cast<CollapseDP*>(at(o_dp));
    Counters* hc = (Counters*)ctx->pinned;
    int* hcnt = (int*)((unsigned char*)ctx->pinned + 1024);
    static_assert(sizeof(Counters) <= 1024, "pinned readback layout");
    SALTY_TRY_CUDA(E, out.nodes.ensure((size_t)n + 1));
    SALTY_TRY_CUDA(E, out.tris.ensure((size_t)n * kTriFloat4));

    cudaEvent_t e0 = ctx->ev[0], e1 = ctx->ev[1];
    cudaEventRecord(e0, st);
    k_init_counters<<<1, 1, 0, st>>>(ctr);
    const unsigned wide = (unsigned)ctx->num_sms * 4;  // blocks of the passes over primitives
    k_prim_setup<<<std::min(grid_for(n, 256), wide), 256, 0, st>>>(d_pos, n, rec[0], ctr);
    k_root_init<<<1, 256, 0, st>>>(ctr, tops[0], items[0], bins[0], subs, lvl_off, bnodes, n);
    // Top levels: the lists live on the device, so levels are launched in groups -- the first
    // as many as an even split needs -- and only then is the next level's length read.
    int levels = 0, group = 1;
    for (int r = n; r > kSub; r = (r + 1) / 2) ++group;
    if (n > kSub) {
        const unsigned gi = (unsigned)std::min<size_t>(max_item, wide), gs = (unsigned)std::min<size_t>((max_top + 3) / 4, wide);
        for (;;) {
            for (int g = 0; g < group; ++g, ++levels) {
                const int c = levels & 1;
                k_top_bin<<<gi, kTopThreads, 0, st>>>(levels, rec[c], tops[c], items[c], bins[c], prm.B, ctr);
                k_top_split<<<gs, kSplitWarps * 32, 0, st>>>(levels, tops[c], tops[c ^ 1], bins[c], bins[c ^ 1], items[c ^ 1],
                                                             subs, bnodes, hist, lvl_off, prm.B, ctr);
                k_top_partition<<<gi, kTopThreads, 0, st>>>(levels, rec[c], rec[c ^ 1], tops[c], tops[c ^ 1], items[c],
                                                            prm.B, ctr);
            }
            SALTY_TRY_CUDA(E, cudaMemcpyAsync(hc, ctr, sizeof(Counters), cudaMemcpyDeviceToHost, st));
            SALTY_TRY_CUDA(E, cudaStreamSynchronize(st));
            if (hc->error) return E.fail(SALTY_ERR_CUDA, "BVH partition disagreed with its bins by level %d", levels);
            if (hc->ntop[levels & 1] == 0) break;
            group = 3;
            if (levels + group > kMaxLevels) return E.fail(SALTY_ERR_CAPACITY, "binary build did not terminate");
        }
    }
    SubArgs sa{{rec[0], rec[1]}, subs, bnodes, dp, prim, ctr, prm, kCollapseNodeCost, kCollapseTriCost};
    SALTY_TRY_CUDA(E, cudaFuncSetAttribute(k_subtree, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SubShared)));
    int per_sm = 0;
    SALTY_TRY_CUDA(E, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_subtree, kSubThreads, sizeof(SubShared)));
    const unsigned nsub = n > kSub ? (unsigned)hc->nsub : 1u;
    k_subtree<<<std::min(nsub, (unsigned)(ctx->num_sms * std::max(per_sm, 1))), kSubThreads, sizeof(SubShared), st>>>(sa);
    if (levels > 0)
        k_top_dp<<<1, 1024, 0, st>>>(bnodes, dp, hist, lvl_off, levels, kCollapseNodeCost, kCollapseTriCost);
    // the wide nodes, level by level from the root (binary node 0)
    SALTY_TRY_CUDA(E, cudaMemsetAsync(cnt8, 0, (kMaxLevels + 2) * sizeof(int), st));
    SALTY_TRY_CUDA(E, cudaMemsetAsync(off8, 0, sizeof(int), st));
    SALTY_TRY_CUDA(E, cudaMemsetAsync(work[0], 0, sizeof(int), st));
    k_fill_one<<<1, 1, 0, st>>>(cnt8);
    int depth8 = 0;
    group = 3;
    for (long long r = n; r > 64; r /= 6) ++group;  // about 6 children per wide node
    for (;;) {
        for (int g = 0; g < group; ++g, ++depth8) {
            const int c = depth8 & 1;
            k_collapse<<<std::min(grid_for(n, 128), wide * 2), 128, 0, st>>>(depth8, bnodes, work[c], out.nodes.p, out.tris.p,
                                                                            prim, d_pos, work[c ^ 1], cnt8, off8, ctr, dp);
        }
        SALTY_TRY_CUDA(E, cudaMemcpyAsync(hcnt, cnt8, (depth8 + 1) * sizeof(int), cudaMemcpyDeviceToHost, st));
        SALTY_TRY_CUDA(E, cudaMemcpyAsync(hc, ctr, sizeof(Counters), cudaMemcpyDeviceToHost, st));
        cudaEventRecord(e1, st);
        SALTY_TRY_CUDA(E, cudaEventSynchronize(e1));
        if (hcnt[depth8] == 0) break;
        group = 3;
        if (depth8 + group > kMaxLevels) return E.fail(SALTY_ERR_CAPACITY, "collapse did not terminate");
    }
    SALTY_TRY_CUDA(E, cudaGetLastError());
    long long n8 = 0;
    for (int l = 0; l < depth8; ++l) n8 += hcnt[l];
    while (depth8 > 0 && hcnt[depth8 - 1] == 0) --depth8;
    for (int a = 0; a < 6; ++a) root_box[a] = host_o2f(hc->rootbox[a]);
    const float rdx = root_box[3] - root_box[0], rdy = root_box[4] - root_box[1], rdz = root_box[5] - root_box[2];
    float root_sa = 2.0f * (rdx * rdy + rdx * rdz + rdy * rdz);
    if (!(root_sa > 0.0f)) root_sa = 1.0f;
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    if (hc->ntris != n) return E.fail(SALTY_ERR_CUDA, "collapse wrote %d of %d triangles", hc->ntris, n);
    out.n_nodes = n8;
    out.n_tris = n;
    out.depth = depth8;
    out.built = true;
    static std::atomic<uint64_t> builds{0};
    out.generation = ++builds;  // unique in the process
    out.info.n_nodes = n8;
    out.info.n_binary = 2 * (int64_t)hc->splits + 1;
    out.info.depth = depth8;
    out.info.binary_depth = hc->depth;
    out.info.sah_cost = hc->sah / (double)root_sa;
    out.info.build_ms = ms;
    return SALTY_OK;
}

}  // namespace salty
