// Device H2 matrix of the t-SNE repulsive kernel K(x, y) = (1 + |x - y|^2)^-2.
//
// The reference builds and applies its H2 matrix through the H2Pack library
// (src/tsne_h2pack.c:772-953 update_h2_matrix, src/tsne_h2_matmul.c:225-452 fused product),
// which is absent from the reference checkout. This file is the engine's own design:
//
//   tree   : root box = bounding-box midpoint with half-width MIN_HALF_WIDTH * 2^k; 64-bit
//            Morton keys of the points' cells at depth L; stable sort -> tree order; every
//            level at once from the digits that neighbouring keys share, nodes split while they
//            hold more than leaf_size points and are numbered level by level in key order.
//   lists  : per-target far / near partners of the symmetric dual-tree traversal, derived
//            from the parent's inadmissible-source set (NSET), a warp per target.
//   bases  : for every node at level >= 2, an interpolative decomposition of K(candidates,
//            proxy points): column-pivoted Gram-Schmidt, one CTA per node, candidates = a
//            leaf's points or the children's skeletons (nested bases); the upward sums at its end.
//   product: far field (warp per compressed target), finer far entries and near field (CTA
//            per leaf, source tiles in shared memory) on a side stream, downward pass, then the
//            Z identity and the force.
// The CPU oracle (oracle/tsne_oracle.c) restates the same design; tree and lists agree bit
// for bit.
#include <cub/cub.cuh>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "devbuf.h"
#include "h2.h"
#include "kernels.h"

namespace tsne {
namespace {

template <int D> using Vec = typename Dim<D>::vec;

constexpr int IDG_THREADS = 256;     // shared-memory ID kernel (3D, large 2D leaves)
constexpr int IDG_GROUP = 4;         // its threads per candidate row in a Gram-Schmidt step
constexpr int NEAR_THREADS = 128;
constexpr int STACK_CAP = 192;       // leaf-target descent stack (depth * (2^D - 1) + 2^D)

struct TreeView {
    int n, L, leaf_size, cap_node, nset_cap;
    const unsigned long long *keys;
    int *start, *end, *level, *parent, *fchild, *nchild, *leaf, *ix;
    int4 *rec;               // per node, packed for the list pass: see node_rec
    float4 *proxies;         // per level: see proxy_table
    int *fm;                 // per point: first | last level << 8 of the nodes it starts, or -1
    int *blkcnt, *blkoff;    // per block of TREE_BLOCK points, 2 x 32 counts / offsets
    int *bset, *nid;         // per level l: boundary starts B_l and their node ids (stride cap_node)
    int *btot;               // |B_l|
    int *tickets;            // work-item counters of the dependency-ordered launches
    TreeInfo *info;
};

// each is zeroed by a kernel that runs before the launch that draws from it
enum { TICKET_LISTS = 0, TICKET_BASES = 1, TICKET_DOWN = 2, N_TICKET = 3 };

__device__ __forceinline__ void fma4(float4 &acc, float w, const float4 &v)
{
    acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y);
    acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
}
__device__ __forceinline__ void add4(float4 &a, const float4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }

// ---------------------------------------------------------------------------------
// root box and keys
// ---------------------------------------------------------------------------------
template <int D>
__device__ void root_from_parts(int n, int nblk, const double *part, const TreeView &tv);

// Bounding box in one launch: a grid of partial boxes, and the block that finishes last reduces
// them to the root box and writes the root node (`done` counts the finished blocks and is left
// at zero for the next launch). A second launch for the root alone cost 5 us plus its gap.
template <int D>
__global__ void __launch_bounds__(256) k_bbox(int n, const Vec<D> *Y, double *part, TreeView tv,
                                              int *done)
{
    after_previous();
    float lo[D], hi[D];
    int bad = 0;
    for (int k = 0; k < D; k++) { lo[k] = INFINITY; hi[k] = -INFINITY; }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const Vec<D> y = Y[i];
        for (int k = 0; k < D; k++) {
            const float v = vget(y, k);
            if (!isfinite(v)) { bad++; continue; }
            lo[k] = fminf(lo[k], v);
            hi[k] = fmaxf(hi[k], v);
        }
    }
    __shared__ float sl[256][D], sh[256][D];
    __shared__ int sb[256];
    for (int k = 0; k < D; k++) { sl[threadIdx.x][k] = lo[k]; sh[threadIdx.x][k] = hi[k]; }
    sb[threadIdx.x] = bad;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            for (int k = 0; k < D; k++) {
                sl[threadIdx.x][k] = fminf(sl[threadIdx.x][k], sl[threadIdx.x + s][k]);
                sh[threadIdx.x][k] = fmaxf(sh[threadIdx.x][k], sh[threadIdx.x + s][k]);
            }
            sb[threadIdx.x] += sb[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < D; k++) {
            part[(size_t)blockIdx.x * (2 * D + 1) + k] = sl[0][k];
            part[(size_t)blockIdx.x * (2 * D + 1) + D + k] = sh[0][k];
        }
        part[(size_t)blockIdx.x * (2 * D + 1) + 2 * D] = sb[0];
        __threadfence();
        sb[1] = atomicAdd(done, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!sb[1]) return;
    __threadfence();
    root_from_parts<D>(n, gridDim.x, part, tv);
    if (threadIdx.x == 0) *done = 0;
}

// Root box from the bounding box (min / max are exact in any order), then the root node; the
// counters that the build's later kernels add to are cleared here.
template <int D>
__device__ void root_from_parts(int n, int nblk, const double *part, const TreeView &tv)
{
    __shared__ double slo[256][D], shi[256][D], sbad[256];
    double lo[D], hi[D], bad = 0.0;
    for (int k = 0; k < D; k++) { lo[k] = INFINITY; hi[k] = -INFINITY; }
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        for (int k = 0; k < D; k++) {
            lo[k] = fmin(lo[k], __ldcg(part + (size_t)b * (2 * D + 1) + k));
            hi[k] = fmax(hi[k], __ldcg(part + (size_t)b * (2 * D + 1) + D + k));
        }
        bad += __ldcg(part + (size_t)b * (2 * D + 1) + 2 * D);
    }
    for (int k = 0; k < D; k++) { slo[threadIdx.x][k] = lo[k]; shi[threadIdx.x][k] = hi[k]; }
    sbad[threadIdx.x] = bad;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            for (int k = 0; k < D; k++) {
                slo[threadIdx.x][k] = fmin(slo[threadIdx.x][k], slo[threadIdx.x + s][k]);
                shi[threadIdx.x][k] = fmax(shi[threadIdx.x][k], shi[threadIdx.x + s][k]);
            }
            sbad[threadIdx.x] += sbad[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    TreeInfo *info = tv.info;
    double ext = 0.0, ctr[D];
    for (int k = 0; k < D; k++) {
        ctr[k] = 0.5 * (slo[0][k] + shi[0][k]);
        const double e = 0.5 * (shi[0][k] - slo[0][k]);
        if (e > ext) ext = e;
    }
    double R = MIN_HALF_WIDTH;
    for (int it = 0; it < 2100 && R < ext; it++) R *= 2.0;
    info->nonfinite = sbad[0] > 0.0 ? 1 : 0;
    info->radius = R;
    for (int k = 0; k < 3; k++) info->corner[k] = k < D ? ctr[k] - R : 0.0;
    info->n_node = 1;
    info->max_level = 0;
    info->max_leaf = 0;
    info->nset_overflow = 0;
    info->pad[0] = 0;   // node-capacity overflow
    info->pad[2] = 0;   // list slot overflow
    tv.tickets[TICKET_LISTS] = 0;
    for (int l = 0; l < 32; l++) info->n_level_nodes[l] = 0;
    for (int l = 0; l < 33; l++) info->level_begin[l] = 0;
    info->n_level_nodes[0] = 1;
    info->level_begin[1] = 1;
    tv.start[0] = 0; tv.end[0] = n; tv.level[0] = 0; tv.parent[0] = -1;
    tv.fchild[0] = -1; tv.nchild[0] = 0; tv.leaf[0] = 1;
    tv.ix[0] = tv.ix[1] = tv.ix[2] = 0;
}

// Morton keys of the cells at depth L, FP64 with IEEE operations only
template <int D>
struct KeyMaker {
    double cell, qmax, corner[D];
    __device__ __forceinline__ KeyMaker(const TreeInfo *info, int L)
        : cell(2.0 * info->radius / (double)(1LL << L)), qmax((double)((1LL << L) - 1))
    {
        for (int k = 0; k < D; k++) corner[k] = info->corner[k];
    }
    __device__ __forceinline__ unsigned long long key(const Vec<D> &y, int L) const
    {
        unsigned int q[D];
        for (int k = 0; k < D; k++) {
            const double t = ((double)vget(y, k) - corner[k]) / cell;
            double f;
            if (!(t >= 0.0)) f = 0.0;
            else if (t > qmax) f = qmax;
            else f = floor(t);
            q[k] = (unsigned int)f;
        }
        unsigned long long key = 0;
        for (int b = L - 1; b >= 0; b--)
            for (int k = D - 1; k >= 0; k--) key = (key << 1) | ((q[k] >> b) & 1u);
        return key;
    }
};

template <int D>
__global__ void k_keys(int n, int L, const Vec<D> *Y, const TreeInfo *info, unsigned long long *keys, int *idx)
{
    after_previous();
    const KeyMaker<D> km(info, L);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        keys[i] = km.key(Y[i], L);
        idx[i] = i;
    }
}

// The sort of up to SORT_MOST points. The device-wide radix sort is nine launches with the keys'
// whatever the size, about 70 us at 20K points; this is two, 36 us. Tiles of SORT_TILE points are
// made (keys and all) and sorted by a CTA each, stably; a point's place in the whole order is its
// place in its tile plus, for every other tile, the keys there that come before it: those <= its
// key in the tiles before (equal keys keep their order), those < its key in the tiles after. The
// bisections grow with the square of the points: a rebuild gains 35 us at 50K and at 66K points and
// 17 us at 131K; beyond, the radix sort.
constexpr int SORT_THREADS = 512, SORT_ITEMS = 4, SORT_TILE = SORT_THREADS * SORT_ITEMS;
constexpr int SORT_MOST = 131072;

struct KeyLess {
    __device__ bool operator()(unsigned long long a, unsigned long long b) const { return a < b; }
};

template <int D>
__global__ void __launch_bounds__(SORT_THREADS)
k_tile_sort(int n, int L, const Vec<D> *Y, const TreeInfo *info, unsigned long long *keys, int *idx)
{
    after_previous();
    using Sort = cub::BlockMergeSort<unsigned long long, SORT_THREADS, SORT_ITEMS, int>;
    __shared__ typename Sort::TempStorage tmp;
    const KeyMaker<D> km(info, L);
    const int base = blockIdx.x * SORT_TILE + threadIdx.x * SORT_ITEMS;
    unsigned long long k[SORT_ITEMS];
    int v[SORT_ITEMS];
#pragma unroll
    for (int q = 0; q < SORT_ITEMS; q++) {   // past the end: above every key (a key has 60 bits at most)
        v[q] = base + q;
        k[q] = base + q < n ? km.key(Y[base + q], L) : ~0ULL;
    }
    Sort(tmp).StableSort(k, v, KeyLess());
#pragma unroll
    for (int q = 0; q < SORT_ITEMS; q++)
        if (base + q < n) {
            keys[base + q] = k[q];
            idx[base + q] = v[q];
        }
}

__global__ void __launch_bounds__(256) k_tile_rank(int n, const unsigned long long *tk, const int *ti,
                                                   unsigned long long *keys, int *perm)
{
    after_previous();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = tk[i];
    const int mine = i / SORT_TILE, tiles = (n + SORT_TILE - 1) / SORT_TILE;
    int rank = i % SORT_TILE;
    constexpr int T = 4;   // bisections side by side: each step is a dependent load
    for (int t0 = 0; t0 < tiles; t0 += T) {
        int pos[T];
#pragma unroll
        for (int q = 0; q < T; q++) pos[q] = 0;
        // keys of tile t that come before point i: those < k + 1 before its own tile, < k after
        for (int step = SORT_TILE; step > 0; step >>= 1)
#pragma unroll
            for (int q = 0; q < T; q++) {
                const int t = t0 + q, p = t * SORT_TILE + pos[q] + step;   // (past the last tile: p > n)
                if (pos[q] + step <= SORT_TILE && p <= n && tk[p - 1] < (t < mine ? k + 1 : k)) pos[q] += step;
            }
#pragma unroll
        for (int q = 0; q < T; q++) rank += t0 + q == mine ? 0 : pos[q];
    }
    keys[rank] = k;
    perm[rank] = ti[i];
}

// ---------------------------------------------------------------------------------
// tree: all levels at once from the sorted keys.
//
// delta[i] = number of leading base-2^D digits that key[i - 1] and key[i] share (L when equal;
// -1 at i = 0 and at the sentinel i = n). A node of level l is a maximal run of points with
// one l-digit prefix: it starts at a point s with delta[s] < l and ends at the next point
// with delta < l. A node exists when its parent holds more than leaf_size points (and it is
// at most at level L); the counts shrink down the tree, so that is the whole condition.
//
// Point s starts the nodes of levels f_s = delta[s] + 1 .. m_s when the node of level
// delta[s] around it holds more than leaf_size points (E_s); m_s is the first level whose
// node starting at s holds at most leaf_size points (the leaf), capped at L. Nodes are
// numbered level by level in key order; the starts of level l's node boundaries,
// B_l = {E points with f <= l}, give every node's end (the next entry of B_l), parent (the
// entry of B_{l-1} at or before it) and children (the entries of B_{l+1} inside it).
// ---------------------------------------------------------------------------------
constexpr int TREE_BLOCK = 1024;   // points per block of the marking and numbering kernels

template <int D>
__device__ __forceinline__ int shared_digits(unsigned long long a, unsigned long long b, int L)
{
    const unsigned long long x = a ^ b;
    if (x == 0ULL) return L;
    return (__clzll((long long)x) - (64 - D * L)) / D;
}

// coordinate k of a key: every D-th bit, brought together by halving steps
template <int D>
__device__ __forceinline__ unsigned int key_coord(unsigned long long key, int k)
{
    unsigned long long x = key >> k;
    if constexpr (D == 2) {
        x &= 0x5555555555555555ULL;
        x = (x | x >> 1) & 0x3333333333333333ULL;
        x = (x | x >> 2) & 0x0f0f0f0f0f0f0f0fULL;
        x = (x | x >> 4) & 0x00ff00ff00ff00ffULL;
        x = (x | x >> 8) & 0x0000ffff0000ffffULL;
        x = (x | x >> 16) & 0x00000000ffffffffULL;
    } else {
        x &= 0x1249249249249249ULL;
        x = (x | x >> 2) & 0x10c30c30c30c30c3ULL;
        x = (x | x >> 4) & 0x100f00f00f00f00fULL;
        x = (x | x >> 8) & 0x001f0000ff0000ffULL;
        x = (x | x >> 16) & 0x001f00000000ffffULL;
        x = (x | x >> 32) & 0x00000000001fffffULL;
    }
    return (unsigned int)x;
}

// per point: E, f, m packed in fm (-1: starts no node); per block and level the number of
// node starts and of boundary starts; the tree-order coordinates
__device__ __forceinline__ void tree_bits(int fm, int l, bool &bn, bool &bb)
{
    const int f = fm & 0xff, m = fm >> 8;
    bb = fm >= 0 && f <= l;
    bn = bb && l <= m;
}

// In the sorted keys the least delta of (a, b] is the number of digits key[a] and key[b] share, so
// neither question needs a walk: the run of points that share delta[s] digits with s starts at p,
// found by bisection over the leaf_size points before s, and E_s is whether point p + leaf_size
// still belongs to it; m_s comes from the digits that points s and s + leaf_size share. The
// block's keys and leaf_size on each side are staged in shared memory while that fits. Walking
// point by point, up to leaf_size each way, took 82 us at 1M points and 18 at 20K with a launch of
// its own for the coordinates (10 and 4 us); this takes 37 and 9 us.
constexpr int TREE_HALO = 256;     // longest leaf_size whose keys are staged

template <int D>
__global__ void __launch_bounds__(TREE_BLOCK) k_tree_marks(TreeView tv, const int *perm, const Vec<D> *Y,
                                                           Vec<D> *xt)
{
    after_previous();
    __shared__ int wc[2][32][TREE_BLOCK / 32];
    __shared__ int s_max[TREE_BLOCK / 32];
    __shared__ unsigned long long sk[TREE_BLOCK + 2 * TREE_HALO];
    const int n = tv.n, L = tv.L, leaf = tv.leaf_size;
    const int b0 = blockIdx.x * TREE_BLOCK, s = b0 + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool staged = leaf <= TREE_HALO;
    if (staged)
        for (int i = max(0, b0 - leaf) + threadIdx.x; i < min(n, b0 + TREE_BLOCK + leaf); i += TREE_BLOCK)
            sk[i - b0 + TREE_HALO] = tv.keys[i];
    if (s < n) xt[s] = Y[perm[s]];
    __syncthreads();
    auto key = [&](int i) { return staged ? sk[i - b0 + TREE_HALO] : tv.keys[i]; };
    int fm = -1;
    if (s < n) {
        const unsigned long long ks = key(s);
        const int ds = s == 0 ? -1 : shared_digits<D>(key(s - 1), ks, L), f = ds + 1;
        bool E = s == 0;
        if (s > 0) {
            auto with_s = [&](int i) { return shared_digits<D>(key(i), ks, L) >= ds; };
            if (s >= leaf && with_s(s - leaf)) E = true;
            else {
                int lo = max(0, s - leaf), p = s - 1;   // point s - 1 shares delta[s] digits
                while (lo < p) {
                    const int mid = (lo + p) >> 1;
                    if (with_s(mid)) p = mid;
                    else lo = mid + 1;
                }
                E = leaf < n - p && with_s(p + leaf);
            }
        }
        if (f > L) E = false;
        if (E) {
            const int mu = leaf < n - s ? shared_digits<D>(ks, key(s + leaf), L) : -1;
            fm = f | (min(L, max(f, mu + 1)) << 8);
        }
        tv.fm[s] = fm;
    }
    // counts of the levels up to the block's deepest node; below it every mark is a boundary
    int mm = fm >= 0 ? fm >> 8 : -1;
    mm = __reduce_max_sync(0xffffffffu, mm);
    const unsigned marks = __ballot_sync(0xffffffffu, fm >= 0);
    if (lane == 0) s_max[w] = mm;
    __syncthreads();
    const int deepest = __reduce_max_sync(0xffffffffu, s_max[lane]);
    for (int l = 0; l <= L; l++) {
        unsigned vn = 0, vb = marks;
        if (l <= deepest) {
            bool bn, bb;
            tree_bits(fm, l, bn, bb);
            vn = __ballot_sync(0xffffffffu, bn);
            vb = __ballot_sync(0xffffffffu, bb);
        }
        if (lane == 0) { wc[0][l][w] = __popc(vn); wc[1][l][w] = __popc(vb); }
    }
    __syncthreads();
    if (threadIdx.x < 64) {
        const int arr = threadIdx.x >> 5, l = threadIdx.x & 31;
        int c = 0;
        if (l <= L)
            for (int k = 0; k < TREE_BLOCK / 32; k++) c += wc[arr][l][k];
        tv.blkcnt[((size_t)blockIdx.x * 2 + arr) * 32 + l] = c;
    }
}

// Exclusive scans of the 64 per-block count columns (a CTA per column; each thread takes a
// contiguous run of blocks, then a block-wide scan of the runs). Column totals: the node
// counts per level (columns 0-31) into btot[32 + l], the boundary counts |B_l| (columns 32-63)
// into btot[l]; every block of k_tree_emit turns the level counts into the level ranges.
constexpr int TREE_SCAN_THREADS = 1024;

__global__ void __launch_bounds__(TREE_SCAN_THREADS) k_tree_scan(int nblk, TreeView tv)
{
    after_previous();
    __shared__ int wsum[TREE_SCAN_THREADS / 32];
    const int col = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int per = (nblk + TREE_SCAN_THREADS - 1) / TREE_SCAN_THREADS;
    const int b0 = min(nblk, tid * per), b1 = min(nblk, b0 + per);
    auto at = [&](int b) { return ((size_t)b * 2 + (col >> 5)) * 32 + (col & 31); };
    int own = 0;
    for (int b = b0; b < b1; b++) own += tv.blkcnt[at(b)];
    int x = own;   // inclusive scan of the runs: warps, then the warp totals
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        wsum[lane] = t;
    }
    __syncthreads();
    int run = x - own + (w > 0 ? wsum[w - 1] : 0);
    for (int b = b0; b < b1; b++) {
        const int v = tv.blkcnt[at(b)];
        tv.blkoff[at(b)] = run;
        run += v;
    }
    if (tid == TREE_SCAN_THREADS - 1) {
        const int total = wsum[31];
        if (col < 32) tv.btot[32 + col] = total;
        else tv.btot[col - 32] = (col - 32) <= tv.L ? total : 0;
    }
}

// numbers the nodes and writes their start, level, leaf flag, box index and first child;
// end, parent and child count are stored as positions in the boundary lists for k_tree_finish.
// Every block scans the 32 level counts itself (a warp; no launch of its own for that), block 0
// writes the level table.
template <int D>
__global__ void __launch_bounds__(TREE_BLOCK) k_tree_emit(TreeView tv)
{
    after_previous();
    __shared__ int wo[2][32][TREE_BLOCK / 32];
    __shared__ int sboff[2][32], slb[32], s_over, s_deep;
    const int n = tv.n, L = tv.L;
    const int s = blockIdx.x * TREE_BLOCK + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w == 0) {   // level ranges
        const int c = lane <= L ? tv.btot[32 + lane] : 0;
        int x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        const int total = __shfl_sync(0xffffffffu, x, 31);
        const unsigned used = __ballot_sync(0xffffffffu, c > 0);
        const int over = total > tv.cap_node;   // node table full: the host regrows it; nothing downstream runs
        slb[lane] = x - c;
        if (lane == 0) { s_over = over; s_deep = 31 - __clz((int)used); }
        if (blockIdx.x == 0) {
            TreeInfo *info = tv.info;
            info->level_begin[lane] = x - c;
            info->n_level_nodes[lane] = over ? 0 : c;
            if (lane == 0) {
                info->level_begin[32] = total;
                info->n_node = over ? 0 : total;
                info->max_level = over ? 0 : 31 - __clz((int)used);
                if (over) info->pad[0] = 1;
            }
        }
    }
    __syncthreads();
    if (s_over) return;
    const int deepest = s_deep;   // no level below it has a node: its boundaries are not needed
    const unsigned lt = (1u << lane) - 1u;
    const int fm = s < n ? tv.fm[s] : -1;
    for (int l = 0; l <= deepest; l++) {
        bool bn, bb;
        tree_bits(fm, l, bn, bb);
        const unsigned vn = __ballot_sync(0xffffffffu, bn), vb = __ballot_sync(0xffffffffu, bb);
        if (lane == 0) { wo[0][l][w] = __popc(vn); wo[1][l][w] = __popc(vb); }
    }
    __syncthreads();
    if (threadIdx.x < 64) {   // exclusive scan over the warps, per array and level
        const int arr = threadIdx.x >> 5, l = threadIdx.x & 31;
        if (l <= deepest) {
            int run = 0;
            for (int k = 0; k < TREE_BLOCK / 32; k++) { const int c = wo[arr][l][k]; wo[arr][l][k] = run; run += c; }
        }
        // the block's level offsets, read once (not once per level by every warp)
        sboff[arr][l] = l <= L ? tv.blkoff[((size_t)blockIdx.x * 2 + arr) * 32 + l] : 0;
    }
    __syncthreads();
    const size_t cap = (size_t)tv.cap_node;
    const unsigned long long key = s < n ? tv.keys[s] : 0ULL;
    const int f = fm & 0xff, m = fm >> 8;
    unsigned int q[3] = {0, 0, 0};
    if (fm >= 0)
        for (int k = 0; k < D; k++) q[k] = key_coord<D>(key, k);
    int prev_br = 0, prev_id = -1;
    for (int l = 0; l <= deepest; l++) {
        bool bn, bb;
        tree_bits(fm, l, bn, bb);
        const unsigned vn = __ballot_sync(0xffffffffu, bn), vb = __ballot_sync(0xffffffffu, bb);
        const int br = sboff[1][l] + wo[1][l][w] + __popc(vb & lt);
        if (bb) {
            int id = -1;
            if (bn) {
                const int nr = sboff[0][l] + wo[0][l][w] + __popc(vn & lt);
                id = slb[l] + nr;
                tv.start[id] = s;
                tv.level[id] = l;
                tv.leaf[id] = l == m ? 1 : 0;
                for (int k = 0; k < 3; k++) tv.ix[(size_t)id * 3 + k] = (int)(q[k] >> (L - l));
                tv.end[id] = br;
                tv.parent[id] = l == 0 ? -1 : (f <= l - 1 ? prev_br : prev_br - 1);
                tv.fchild[id] = -1;
                tv.nchild[id] = 0;
                if (prev_id >= 0) { tv.fchild[prev_id] = id; tv.nchild[prev_id] = br; }
            }
            tv.bset[(size_t)l * cap + br] = s;
            tv.nid[(size_t)l * cap + br] = id;
            prev_id = id;
        }
        prev_br = br;
    }
}

// The node record of the list pass, two 16-byte loads for what lies in seven arrays:
// [2t] = (first child, children | leaf << 8 | level << 16, parent, 0), [2t + 1] = box index.
struct NodeRec {
    int fchild, nchild, level, parent;
    bool leaf;
    int ix[3];
};
__device__ __forceinline__ NodeRec node_rec(const TreeView &tv, int t)
{
    const int4 a = tv.rec[2 * (size_t)t], b = tv.rec[2 * (size_t)t + 1];
    NodeRec r;
    r.fchild = a.x;
    r.nchild = a.y & 0xff;
    r.leaf = (a.y >> 8) & 1;
    r.level = a.y >> 16;
    r.parent = a.z;
    r.ix[0] = b.x; r.ix[1] = b.y; r.ix[2] = b.z;
    return r;
}

// ---------------------------------------------------------------------------------
// proxy points (shells |y - c|_inf = rho h around a box of half-width h)
// ---------------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void proxy_point(int p, double h, float *out)
{
    if constexpr (D == 2) {
        const int sh = p / SHELL_PTS_2D, k = p % SHELL_PTS_2D;
        const double rad = shell_rho(sh) * h;
        const double off = (sh & 1) ? 0.0 : 0.5;
        const double u = ((double)k + off) * (8.0 / SHELL_PTS_2D);
        const int side = (int)(u * 0.5);
        const double a = u - 2.0 * side - 1.0;
        double x, y;
        switch (side) {
            case 0: x = a; y = -1.0; break;
            case 1: x = 1.0; y = a; break;
            case 2: x = -a; y = 1.0; break;
            default: x = -1.0; y = -a; break;
        }
        out[0] = (float)(x * rad);
        out[1] = (float)(y * rad);
    } else {
        constexpr int g = SHELL_GRID_3D, per = 6 * g * g;
        const int sh = p / per, r = p % per, f = r / (g * g), ij = r % (g * g), i = ij / g, j = ij % g;
        const double rad = shell_rho(sh) * h;
        const int ax = f >> 1;
        const double sgn = (f & 1) ? 1.0 : -1.0;
        const double a = ((double)i + 0.5) * (2.0 / g) - 1.0;
        const double b = ((double)j + 0.5) * (2.0 / g) - 1.0;
        double c[3];
        c[ax] = sgn;
        c[(ax + 1) % 3] = a;
        c[(ax + 2) % 3] = b;
        for (int k = 0; k < 3; k++) out[k] = (float)(c[k] * rad);
    }
}

// The proxies of every level, relative to a node's centre, once per build (they are FP64 work that
// every node of a level repeated: 26,000 of a 3D node's 550,000 cycles, 1,500 of a 2D node's 70,000).
// 2D: (x, y) per proxy; 3D: the pairs (2j, 2j + 1) as (-2x, -2x', -2y, -2y'), then, ID3_PB further,
// (-2z, -2z', |p|^2, |p'|^2).
constexpr int PROXY_F4 = 216;   // float4 per level
template <int D>
__device__ __forceinline__ void proxy_table(int l, double radius, float4 *table)
{
    constexpr int P = Dim<D>::NPROXY;
    static_assert(D == 2 ? P * sizeof(float2) <= PROXY_F4 * sizeof(float4) : P == PROXY_F4, "table row");
    const double h = radius / (double)(1LL << l);
    float4 *row = table + (size_t)l * PROXY_F4;
    if constexpr (D == 2) {
        for (int p = threadIdx.x; p < P; p += blockDim.x) {
            float y[2];
            proxy_point<2>(p, h, y);
            reinterpret_cast<float2 *>(row)[p] = make_float2(y[0], y[1]);
        }
    } else {
        for (int j = threadIdx.x; j < P / 2; j += blockDim.x) {
            float p0[3], p1[3];
            proxy_point<3>(2 * j, h, p0);
            proxy_point<3>(2 * j + 1, h, p1);
            row[j] = make_float4(-2.f * p0[0], -2.f * p1[0], -2.f * p0[1], -2.f * p1[1]);
            row[P / 2 + j] = make_float4(-2.f * p0[2], -2.f * p1[2], fmaf(p0[0], p0[0], fmaf(p0[1], p0[1], p0[2] * p0[2])),
                                         fmaf(p1[0], p1[0], fmaf(p1[1], p1[1], p1[2] * p1[2])));
        }
    }
}

// end, parent and child count of every node from the boundary lists; its record; the largest
// leaf; the proxy table
template <int D>
__global__ void k_tree_finish(TreeView tv)
{
    after_previous();
    TreeInfo *info = tv.info;
    if (info->pad[0]) return;
    for (int l = blockIdx.x; l <= tv.L; l += gridDim.x) proxy_table<D>(l, info->radius, tv.proxies);
    const int n_node = info->n_node;
    const size_t cap = (size_t)tv.cap_node;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n_node; t += gridDim.x * blockDim.x) {
        const int l = tv.level[t], s = tv.start[t], pos = tv.end[t];
        const int e = pos + 1 < tv.btot[l] ? tv.bset[(size_t)l * cap + pos + 1] : tv.n;
        tv.end[t] = e;
        int par = -1, c = 0;
        if (l > 0) tv.parent[t] = par = tv.nid[(size_t)(l - 1) * cap + tv.parent[t]];
        const int lf = tv.leaf[t];
        if (lf) {
            atomicMax(&info->max_leaf, e - s);
        } else {
            const int c0 = tv.nchild[t], lim = tv.btot[l + 1];
            while (c0 + c < lim && tv.bset[(size_t)(l + 1) * cap + c0 + c] < e) c++;
            tv.nchild[t] = c;
        }
        tv.rec[2 * (size_t)t] = make_int4(tv.fchild[t], c | lf << 8 | l << 16, par, 0);
        tv.rec[2 * (size_t)t + 1] = make_int4(tv.ix[3 * (size_t)t], tv.ix[3 * (size_t)t + 1], tv.ix[3 * (size_t)t + 2], 0);
    }
}

// ---------------------------------------------------------------------------------
// dependency-ordered launches
//
// A kernel that processes the nodes of several levels in one launch takes its work items from
// a ticket counter, so items start in ticket order whatever order the hardware dispatches
// blocks in. An item waits only for items with smaller tickets, which are held by running
// blocks or finished, so every wait ends. The waits are bounded all the same: after
// DEP_WAIT_LIMIT polls the waiting thread records the failure (the host reports it) and goes on.
// ---------------------------------------------------------------------------------
constexpr int DEP_WAIT_LIMIT = 1 << 22;

struct DepArgs {
    int *flag;      // per node: epoch of the last launch that finished it
    int *ticket;    // work-item counter, zeroed before the launch
    int *err;       // set when a wait gave up
    int epoch;
    int limit = DEP_WAIT_LIMIT;   // polls before a wait gives up
    int *flag2 = nullptr;         // a second per-node flag (launches that publish twice)
};

__device__ __forceinline__ int ld_acquire_gpu(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(int *p, int v)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// one thread: poll until node's flag holds this launch's epoch (bounded)
__device__ __forceinline__ void dep_wait(const DepArgs &dp, int node)
{
    const int *f = dp.flag + node;
    for (int it = 0; it < dp.limit; it++) {
        if (ld_acquire_gpu(f) == dp.epoch) return;
        __nanosleep(it < 64 ? 32 : 128);
    }
    atomicExch(dp.err, 1);
}
// one thread, after a block barrier that follows every write of the item
__device__ __forceinline__ void dep_publish(const DepArgs &dp, int node)
{
    __threadfence();
    st_release_gpu(dp.flag + node, dp.epoch);
}

// the second flag of a node (launches that publish twice: the bases publish the skeleton and
// rank first, the upward coefficients last)
__device__ __forceinline__ void dep_wait_y0(const DepArgs &dp, int node)
{
    DepArgs d2 = dp;
    d2.flag = dp.flag2;
    dep_wait(d2, node);
}
__device__ __forceinline__ void dep_publish_y0(const DepArgs &dp, int node)
{
    __threadfence();
    st_release_gpu(dp.flag2 + node, dp.epoch);
}

// one bounded wait for `node` (the failure path of the dependency-ordered launches, for tests)
__global__ void k_dep_probe(DepArgs dp, int node)
{
    after_previous();
    if (threadIdx.x == 0) dep_wait(dp, node);
}

// ---------------------------------------------------------------------------------
// interaction lists
// ---------------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ bool admissible(int L, const NodeRec &t, const NodeRec &s)
{
    const long long wt = 1LL << (L - t.level);
    const long long ws = 1LL << (L - s.level);
    long long dist = 0;
#pragma unroll
    for (int k = 0; k < D; k++) {
        const long long ct = 2LL * t.ix[k] * wt + wt;
        const long long cs = 2LL * s.ix[k] * ws + ws;
        const long long df = ct > cs ? ct - cs : cs - ct;
        dist = df > dist ? df : dist;
    }
    return dist >= wt + ws + (long long)ADM_EXTRA * (wt < ws ? wt : ws);
}

// The count pass also parks each target's entries in fixed slots, so that the list write is a
// compaction; a target with more entries sets slot_over and the whole build falls back to the
// traversing write pass, in 3D with a segmented sort. Targets with far entries hold about 20 of them in 2D
// (69 the most, 300K points) and 50-115 in 3D, where the most is 160 at 20K points, 262-278 at 60K and
// 384 at 300K: so large 3D trees fall back in every build (at 100K 0.24 ms of write and 0.18 of sorts, on the
// side stream). Near entries are 8-23, the most 91.
constexpr int far_slots(int d) { return d == 2 ? 128 : 256; }
constexpr int NEAR_SLOTS = 128;

struct ListOut {
    int *far_cnt, *near_cnt;             // count pass
    int *fine_cnt;                       // of a leaf's far entries, those finer than the leaf
    const int *far_ptr, *near_ptr;       // write pass
    int *far_idx, *near_idx;
    int *nset, *nset_cnt;                // inadmissible sources, packed: see nset_pack
    int *far_slot, *near_slot;           // count pass: far_slots(D) / NEAR_SLOTS entries per target
    int *slot_over;
};

// A source s that is inadmissible for a target, as the target's children will meet it: the range
// of its children, or s itself when it is a leaf (first node << 4 | nodes; that holds 2^27 nodes, whose
// skeletons and coefficients alone, 2.5 KB a node, are more than the device's memory)
__device__ __forceinline__ int nset_pack(int s, const NodeRec &r)
{
    return r.leaf ? (s << 4 | 1) : (r.fchild << 4 | r.nchild);
}

// ---- the traversing write pass: a thread per target (only when a target overflowed its slots)
template <int D>
__device__ void descend(const TreeView &tv, ListOut &lo, int t, const NodeRec &rt, const NodeRec &rc, int &fc, int &nc)
{
    int stk[STACK_CAP];
    int sp = 0;
    for (int k = rc.nchild - 1; k >= 0; k--) stk[sp++] = rc.fchild + k;
    while (sp > 0) {
        const int s = stk[--sp];
        const NodeRec rs = node_rec(tv, s);
        if (admissible<D>(tv.L, rt, rs)) { lo.far_idx[lo.far_ptr[t] + fc++] = s; continue; }
        if (rs.leaf) { lo.near_idx[lo.near_ptr[t] + nc++] = s; continue; }
        if (sp + rs.nchild > STACK_CAP) { atomicExch(&tv.info->nset_overflow, 1); return; }
        for (int k = rs.nchild - 1; k >= 0; k--) stk[sp++] = rs.fchild + k;
    }
}

template <int D>
__global__ void __launch_bounds__(128) k_lists_write(int n_node, TreeView tv, ListOut lo)
{
    after_previous();
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n_node; t += gridDim.x * blockDim.x) {
        const NodeRec rt = node_rec(tv, t);
        int fc = 0, nc = 0;
        if (t == 0) {
            if (rt.leaf) lo.near_idx[lo.near_ptr[0] + nc++] = 0;
        } else {
            const int pn = lo.nset_cnt[rt.parent];
            for (int a = 0; a < pn; a++) {
                const int e = lo.nset[(size_t)rt.parent * tv.nset_cap + a];
                for (int c = e >> 4; c < (e >> 4) + (e & 15); c++) {
                    if (c == t) {
                        if (rt.leaf) lo.near_idx[lo.near_ptr[t] + nc++] = t;
                        continue;
                    }
                    const NodeRec rc = node_rec(tv, c);
                    if (admissible<D>(tv.L, rt, rc)) lo.far_idx[lo.far_ptr[t] + fc++] = c;
                    else if (rt.leaf) {
                        if (rc.leaf) lo.near_idx[lo.near_ptr[t] + nc++] = c;
                        else descend<D>(tv, lo, t, rt, rc, fc, nc);
                    }
                }
            }
        }
        if (D == 2) {
            // ascending partners (insertion sort of this target's short segments; 3D lists are
            // longer and are sorted afterwards by a segmented sort)
            int *f = lo.far_idx + lo.far_ptr[t];
            for (int a = 1; a < fc; a++) { const int v = f[a]; int z = a - 1; while (z >= 0 && f[z] > v) { f[z + 1] = f[z]; z--; } f[z + 1] = v; }
            int *g = lo.near_idx + lo.near_ptr[t];
            for (int a = 1; a < nc; a++) { const int v = g[a]; int z = a - 1; while (z >= 0 && g[z] > v) { g[z + 1] = g[z]; z--; } g[z + 1] = v; }
        }
    }
}

// Count pass of every target in one dependency-ordered launch: persistent warps, a warp per
// target, in increasing node id, so a target's parent comes first. The lanes take the entries of
// the parent's inadmissible set, each with its nodes c. An internal target t sends c to its far
// list when c != t and (t, c) is admissible, else to its own inadmissible set. A leaf target
// sends an admissible c to its far list, a leaf c to its near list, and puts any other c on the
// warp's stack, whose nodes are then expanded 32 children at a time, deepest first: a round pops
// G = 32 / 2^D nodes, so a level of the tree holds at most G - 1 + 32 stack entries, under 1024
// over the depth, plus one chunk's 32 * 2^D.
// What bounds it is the chain from the root (a level each: the parent's flag, its set, the nodes'
// records, the publication), so the next ticket is drawn while a target is worked on, the set
// holds ready child ranges and a node is one record. Leaves had a thread each in a launch of
// their own, every step of whose traversal was a dependent load: with the internal pass 98 us
// at 20K points 2D and 200 us at 1M, 403 us at 100K in 3D (and the traversal again to write).
constexpr int LIST_WARPS = 4;
constexpr int LIST_CTAS = 8;   // per SM
template <int D> constexpr int list_stack() { return 1024 + 32 * (1 << D); }

template <int D>
__global__ void __launch_bounds__(32 * LIST_WARPS) k_lists(TreeView tv, ListOut lo, DepArgs dp)
{
    after_previous();
    constexpr int NCH = 1 << D, G = 32 / NCH, FS = far_slots(D);
    __shared__ int stack_[LIST_WARPS][list_stack<D>()];
    int *stack = stack_[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int n_node = tv.info->n_node, cap = tv.nset_cap, L = tv.L;
    int next = 0;
    if (lane == 0) next = atomicAdd(dp.ticket, 1);
    for (;;) {
        const int t = __shfl_sync(0xffffffffu, next, 0);
        if (t >= n_node) break;
        if (lane == 0) next = atomicAdd(dp.ticket, 1);
        const NodeRec rt = node_rec(tv, t);
        int *fslot = lo.far_slot + (size_t)t * FS, *nslot = lo.near_slot + (size_t)t * NEAR_SLOTS;
        int nf = 0, nn = 0, ns = 0;   // far, near and inadmissible entries so far
        int fine = 0;                 // far entries below the target's level
        // every lane's c (its flags say whether it has one): appended in lane order
        auto put_far = [&](bool on, int c) {
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) {
                const int w = nf + __popc(m & lt);
                if (w < FS) fslot[w] = c;
            }
            nf += __popc(m);
        };
        auto put_near = [&](bool on, int c) {
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) {
                const int w = nn + __popc(m & lt);
                if (w < NEAR_SLOTS) nslot[w] = c;
            }
            nn += __popc(m);
        };
        if (t == 0) {
            if (rt.leaf) put_near(lane == 0, 0);
            else {
                if (lane == 0) lo.nset[0] = nset_pack(0, rt);
                ns = 1;
            }
        } else {
            const int p = rt.parent;
            if (lane == 0) dep_wait(dp, p);
            __syncwarp();
            const int pn = __ldcg(lo.nset_cnt + p);
            for (int a0 = 0; a0 < pn; a0 += 32) {
                const int e = a0 + lane < pn ? __ldcg(lo.nset + (size_t)p * cap + a0 + lane) : 0;
                const int c0 = e >> 4, cn = e & 15;
                int sp = 0;
#pragma unroll
                for (int k = 0; k < NCH; k++) {
                    const bool on = k < cn;
                    const int c = c0 + k;
                    const NodeRec rc = node_rec(tv, on ? c : 0);
                    const bool self = on && c == t;
                    const bool far = on && !self && admissible<D>(L, rt, rc);
                    put_far(far, c);
                    if (!rt.leaf) {
                        const bool in = on && !far;
                        const unsigned m = __ballot_sync(0xffffffffu, in);
                        if (in) {
                            const int w = ns + __popc(m & lt);
                            if (w < cap) lo.nset[(size_t)t * cap + w] = nset_pack(c, rc);
                        }
                        ns += __popc(m);
                    } else {
                        put_near(on && !far && rc.leaf, c);   // the target itself is a leaf too
                        const bool in = on && !far && !rc.leaf;
                        const unsigned m = __ballot_sync(0xffffffffu, in);
                        if (in) stack[sp + __popc(m & lt)] = rc.fchild << 4 | rc.nchild;
                        sp += __popc(m);
                    }
                }
                while (sp > 0) {   // leaf targets only
                    __syncwarp();
                    const int take = min(G, sp), g = lane / NCH, k = lane % NCH;
                    const int q = g < take ? stack[sp - take + g] : 0;
                    sp -= take;
                    __syncwarp();
                    const bool on = k < (q & 15);
                    const int c = (q >> 4) + k;
                    const NodeRec rc = node_rec(tv, on ? c : 0);
                    const bool far = on && admissible<D>(L, rt, rc);
                    fine -= nf;
                    put_far(far, c);
                    fine += nf;
                    put_near(on && !far && rc.leaf, c);
                    const bool in = on && !far && !rc.leaf;
                    const unsigned m = __ballot_sync(0xffffffffu, in);
                    if (in) stack[sp + __popc(m & lt)] = rc.fchild << 4 | rc.nchild;
                    sp += __popc(m);
                }
                __syncwarp();
            }
        }
        if (lane == 0) {
            lo.far_cnt[t] = nf;
            lo.near_cnt[t] = nn;
            lo.fine_cnt[t] = fine;
            if (nf > FS || nn > NEAR_SLOTS) *lo.slot_over = 1;
            if (ns > cap) { atomicExch(&tv.info->nset_overflow, 1); ns = cap; }
            lo.nset_cnt[t] = ns;
        }
        __syncwarp();
        if (!rt.leaf && lane == 0) dep_publish(dp, t);
    }
}

// The list write from the count pass's slots: a warp per target copies its entries to its list
// segment, ascending (each entry's place is its rank among the segment's distinct entries,
// counted from the warp's staged copy; the traversing write pass emits and sorts the same set)
__device__ __forceinline__ void warp_copy_sorted(const int *slot, int cnt, int *dst, int *stage, int lane)
{
    for (int a = lane; a < cnt; a += 32) stage[a] = slot[a];
    __syncwarp();
    for (int a = lane; a < cnt; a += 32) {
        const int v = stage[a];
        int r = 0;
        for (int b = 0; b < cnt; b++) r += stage[b] < v;
        dst[r] = v;
    }
    __syncwarp();
}

template <int D>
__global__ void __launch_bounds__(256) k_lists_compact(TreeView tv, ListOut lo)
{
    after_previous();
    constexpr int FS = far_slots(D);
    __shared__ int stage_[8][FS > NEAR_SLOTS ? FS : NEAR_SLOTS];
    const int n_node = tv.info->n_node;
    const int lane = threadIdx.x & 31;
    int *stage = stage_[threadIdx.x >> 5];
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n_node; t += (gridDim.x * blockDim.x) >> 5) {
        warp_copy_sorted(lo.far_slot + (size_t)t * FS, lo.far_cnt[t], lo.far_idx + lo.far_ptr[t], stage, lane);
        warp_copy_sorted(lo.near_slot + (size_t)t * NEAR_SLOTS, lo.near_cnt[t], lo.near_idx + lo.near_ptr[t], stage, lane);
    }
}

// Positions of every node's entries, from its counts: far_ptr, near_ptr (list segments), rowoff
// (its rows of the interpolation matrices: a leaf's points, or the upper bound of the children's
// skeletons; nodes above MIN_ADM_LEVEL have none), the item lists of the basis launches
// (ilist: the internal nodes at level >= MIN_ADM_LEVEL; llist / blist: the leaves there of at most
// TINY_LEAF / SMALL_LEAF points, clist: the larger ones) and flist, the leaves with far entries
// finer than themselves; each list in increasing node id.
// Two launches over the nodes there are (block sums, then every block adds the sums before its
// own): six device-wide scans over the node capacity and their flag and memset launches took
// 25 launches, 75 us of a rebuild at 20K points and 85 us at 1M.
constexpr int TINY_LEAF = 32;    // the leaves of the smallest basis CTAs,
constexpr int SMALL_LEAF = 64;   // and of the next
constexpr int NODE_BLOCK = 1024;

struct NodeSums {
    long long rows;
    int far, near, in, small, big, large, fine, pad;
};
struct NodeScan {
    const int *far_cnt, *near_cnt, *fine_cnt;
    int *far_ptr, *near_ptr;
    long long *rowoff;
    int *ilist, *llist, *blist, *clist, *flist, *rank;
    NodeSums *blk;
};

__device__ __forceinline__ NodeSums node_add(const NodeSums &a, const NodeSums &b)
{
    NodeSums c;
    c.rows = a.rows + b.rows;
    c.far = a.far + b.far; c.near = a.near + b.near;
    c.in = a.in + b.in; c.small = a.small + b.small; c.big = a.big + b.big;
    c.large = a.large + b.large; c.fine = a.fine + b.fine; c.pad = 0;
    return c;
}
__device__ __forceinline__ NodeSums node_shfl_up(const NodeSums &a, int o)
{
    NodeSums c;
    c.rows = __shfl_up_sync(0xffffffffu, a.rows, o);
    c.far = __shfl_up_sync(0xffffffffu, a.far, o);
    c.near = __shfl_up_sync(0xffffffffu, a.near, o);
    c.in = __shfl_up_sync(0xffffffffu, a.in, o);
    c.small = __shfl_up_sync(0xffffffffu, a.small, o);
    c.big = __shfl_up_sync(0xffffffffu, a.big, o);
    c.large = __shfl_up_sync(0xffffffffu, a.large, o);
    c.fine = __shfl_up_sync(0xffffffffu, a.fine, o);
    c.pad = 0;
    return c;
}
__device__ __forceinline__ NodeSums node_zero()
{
    NodeSums c;
    c.rows = 0; c.far = c.near = c.in = c.small = c.big = c.large = c.fine = c.pad = 0;
    return c;
}
template <int D>
__device__ __forceinline__ NodeSums node_counts(const TreeView &tv, const NodeScan &q, int t)
{
    NodeSums c = node_zero();
    c.far = q.far_cnt[t];
    c.near = q.near_cnt[t];
    c.fine = q.fine_cnt[t] > 0;
    if (tv.level[t] < MIN_ADM_LEVEL) return c;
    if (!tv.leaf[t]) {
        c.rows = (1 << D) * Dim<D>::MAXR;
        c.in = 1;
    } else {
        const int r = tv.end[t] - tv.start[t];
        c.rows = r;
        if (r <= TINY_LEAF) c.small = 1;
        else if (r <= SMALL_LEAF) c.big = 1;
        else c.large = 1;
    }
    return c;
}
// inclusive scan over the block; `total` receives the block's sum in every thread
__device__ __forceinline__ NodeSums node_block_scan(NodeSums x, NodeSums *sh, NodeSums &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const NodeSums y = node_shfl_up(x, o);
        if (lane >= o) x = node_add(x, y);
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        NodeSums v = sh[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const NodeSums y = node_shfl_up(v, o);
            if (lane >= o) v = node_add(v, y);
        }
        sh[lane] = v;
    }
    __syncthreads();
    total = sh[31];
    if (w > 0) x = node_add(x, sh[w - 1]);
    __syncthreads();
    return x;
}

template <int D>
__global__ void __launch_bounds__(NODE_BLOCK) k_node_sums(TreeView tv, NodeScan q)
{
    after_previous();
    __shared__ NodeSums sh[32];
    const int n_node = tv.info->n_node, t = blockIdx.x * NODE_BLOCK + threadIdx.x;
    if (blockIdx.x * NODE_BLOCK >= n_node) return;
    NodeSums total;
    node_block_scan(t < n_node ? node_counts<D>(tv, q, t) : node_zero(), sh, total);
    if (threadIdx.x == 0) q.blk[blockIdx.x] = total;
}

template <int D>
__global__ void __launch_bounds__(NODE_BLOCK) k_node_scan(TreeView tv, NodeScan q)
{
    after_previous();
    __shared__ NodeSums sh[32];
    TreeInfo *info = tv.info;
    const int n_node = info->n_node, t = blockIdx.x * NODE_BLOCK + threadIdx.x;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        q.far_ptr[0] = 0; q.near_ptr[0] = 0; q.rowoff[0] = 0;
        tv.tickets[TICKET_BASES] = 0;
        if (n_node == 0) { info->n_far = info->n_near = info->n_int = info->n_small = info->n_big = info->n_large = info->n_fine = 0; info->n_rows = 0; }
    }
    if (blockIdx.x * NODE_BLOCK >= n_node) return;
    // the blocks before this one
    NodeSums before = node_zero(), total;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += NODE_BLOCK) before = node_add(before, q.blk[b]);
    node_block_scan(before, sh, before);
    const NodeSums own = t < n_node ? node_counts<D>(tv, q, t) : node_zero();
    const NodeSums inc = node_add(node_block_scan(own, sh, total), before);
    if (t >= n_node) return;
    q.far_ptr[t + 1] = inc.far;
    q.near_ptr[t + 1] = inc.near;
    q.rowoff[t + 1] = inc.rows;
    if (own.in) q.ilist[inc.in - 1] = t;
    if (own.small) q.llist[inc.small - 1] = t;
    if (own.big) q.blist[inc.big - 1] = t;
    if (own.large) q.clist[inc.large - 1] = t;
    if (own.fine) q.flist[inc.fine - 1] = t;
    if (tv.level[t] < MIN_ADM_LEVEL) q.rank[t] = 0;   // no basis; the others' ranks come with theirs
    if (t == n_node - 1) {
        info->n_far = inc.far;
        info->n_near = inc.near;
        info->n_rows = inc.rows;
        info->n_int = inc.in;
        info->n_small = inc.small;
        info->n_big = inc.big;
        info->n_large = inc.large;
        info->n_fine = inc.fine;
    }
}

struct IdArgs {
    TreeView tv;
    const void *xt;
    void *skel;
    int *rank;
    const long long *rowoff;
    float *U;
    float *gA, *gnrm;
    int *gsel;
    void *gcand;
    int mcap;      // candidate rows that fit the launch's shared memory
    float tol2;
    float4 *y0;    // upward-pass coefficients of [1 | Y], computed right after the basis
};

template <int D>
constexpr size_t id_smem_bytes(int mcap)
{
    constexpr int P = Dim<D>::NPROXY, MAXR = Dim<D>::MAXR;
    return sizeof(float) * (size_t)P * D                 // proxies
           + sizeof(Vec<D>) * (size_t)mcap               // candidates
           + sizeof(float) * (size_t)mcap                // residual norms
           + sizeof(int) * (size_t)mcap                  // pivot position per row (-1: not selected)
           + sizeof(int) * (size_t)MAXR                  // pivot rows
           + sizeof(float) * (size_t)mcap * (P + 1);     // the matrix (row stride P + 1)
}

// Interpolative decomposition of one node (one CTA): A = K(candidates - c, proxies),
// column-pivoted Gram-Schmidt over the rows of A until the largest residual row norm is
// <= tol * the largest initial one; U = [I ; R11^-1 R12]^T in candidate order.
// The dot products of every step go to the node's U rows (R12), and the column of R11 that
// a step produces is stored in the pivot row of A, which no later step reads.
// LEAVES = true: every leaf at level >= 2 (leaves depend on nothing), blockIdx.x counts
// from the first node of level 2; false: the internal nodes of one level.
// One Gram-Schmidt step over the candidate rows of A (row stride PP): every unselected row a
// loses its component along the unit pivot row q; its dot product goes to U[a][r] and its new
// squared norm to nrm[a]. G threads per row, each over every G-th proxy.
template <int G, int P, int PP>
__device__ __forceinline__ void gs_rows(float *A, const float *q, int m, int tid, const int *selpos, float *nrm,
                                        float *U, int MAXR, int r)
{
    static_assert(P % G == 0, "proxies split evenly over a row's threads");
    for (int a0 = 0; a0 < m; a0 += IDG_THREADS / G) {
        const int a = a0 + tid / G, gl = tid % G;
        const bool act = a < m && selpos[a] < 0;
        float *row = A + (size_t)(act ? a : 0) * PP;
        float d2[2] = {0.f, 0.f};
        if (act) {
#pragma unroll 6
            for (int i = 0; i < P / G; i++) {
                const int p = gl + i * G;
                d2[i & 1] = fmaf(q[p], row[p], d2[i & 1]);
            }
        }
        float dot = d2[0] + d2[1];
        for (int o = 1; o < G; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        float z2[2] = {0.f, 0.f};
        if (act) {
#pragma unroll 6
            for (int i = 0; i < P / G; i++) {
                const int p = gl + i * G;
                const float v = fmaf(-dot, q[p], row[p]);
                row[p] = v;
                z2[i & 1] = fmaf(v, v, z2[i & 1]);
            }
        }
        float s2 = z2[0] + z2[1];
        for (int o = 1; o < G; o <<= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        if (act && gl == 0) {
            nrm[a] = s2;
            U[(size_t)a * MAXR + r] = dot;
        }
    }
}

// items != nullptr: the internal nodes of every level in one dependency-ordered launch (items
// in increasing node id, taken deepest first; a node waits for its internal children's flags);
// otherwise the nodes of `level` (or every leaf). Children's ranks, skeletons and coefficients
// are read through L2.
template <int D, bool LEAVES>
__global__ void __launch_bounds__(IDG_THREADS) k_id(int level, IdArgs g, int n_item, const int *items,
                                                    DepArgs dp)
{
    after_previous();
    constexpr int P = Dim<D>::NPROXY, PP = P + 1, MAXR = Dim<D>::MAXR, NCH = 1 << D;
    extern __shared__ __align__(16) unsigned char smraw[];
    const TreeView &tv = g.tv;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    __shared__ int s_item;
    __shared__ int s_coff[NCH + 1];   // children's first candidate row
    __shared__ float4 s_part[IDG_THREADS];
    int t;
    if (items != nullptr) {
        if (tid == 0) s_item = atomicAdd(dp.ticket, 1);
        __syncthreads();
        if (s_item >= n_item) return;
        t = items[n_item - 1 - s_item];
        if (!LEAVES && tid < tv.nchild[t] && !tv.leaf[tv.fchild[t] + tid]) dep_wait(dp, tv.fchild[t] + tid);
        __syncthreads();
    } else {
        t = tv.info->level_begin[LEAVES ? MIN_ADM_LEVEL : level] + blockIdx.x;
        if (LEAVES ? !tv.leaf[t] : tv.leaf[t] != 0) return;
    }
    const int lvl = tv.level[t];
    const Vec<D> *xt = (const Vec<D> *)g.xt;
    Vec<D> *skel = (Vec<D> *)g.skel;

    unsigned char *ptr = smraw;
    float *prox = (float *)ptr; ptr += sizeof(float) * P * D;
    Vec<D> *cand_s = (Vec<D> *)ptr; ptr += sizeof(Vec<D>) * g.mcap;
    float *nrm_s = (float *)ptr; ptr += sizeof(float) * g.mcap;
    int *selpos_s = (int *)ptr; ptr += sizeof(int) * g.mcap;
    int *sel = (int *)ptr; ptr += sizeof(int) * MAXR;
    float *A_s = (float *)ptr;

    __shared__ float s_bv[IDG_THREADS / 32];
    __shared__ int s_bi[IDG_THREADS / 32];
    __shared__ int s_best, s_stop;
    __shared__ float s_n0;

    int m = 0;
    if (LEAVES) m = tv.end[t] - tv.start[t];
    else {
        if (tid == 0) {
            int acc = 0;
            for (int c = 0; c < tv.nchild[t]; c++) {
                s_coff[c] = acc;
                acc += __ldcg(g.rank + tv.fchild[t] + c);
            }
            s_coff[tv.nchild[t]] = acc;
        }
        __syncthreads();
        m = s_coff[tv.nchild[t]];
    }
    const long long roff = g.rowoff[t];
    const bool glob = m > g.mcap;
    float *A = glob ? g.gA + roff * PP : A_s;
    float *nrm = glob ? g.gnrm + roff : nrm_s;
    int *selpos = glob ? g.gsel + roff : selpos_s;
    Vec<D> *cand = glob ? (Vec<D> *)g.gcand + roff : cand_s;
    float *U = g.U + roff * MAXR;

    const double h = tv.info->radius / (double)(1LL << lvl);
    for (int p = tid; p < P; p += IDG_THREADS) proxy_point<D>(p, h, prox + p * D);
    float ctr[D];
    for (int k = 0; k < D; k++)
        ctr[k] = (float)(tv.info->corner[k] + (double)(2 * tv.ix[(size_t)t * 3 + k] + 1) * h);
    if (LEAVES) {
        for (int a = tid; a < m; a += IDG_THREADS) cand[a] = xt[tv.start[t] + a];
    } else {
        for (int a = tid; a < m; a += IDG_THREADS) {
            int c = 0;
            while (a >= s_coff[c + 1]) c++;
            cand[a] = __ldcg(skel + (size_t)(tv.fchild[t] + c) * MAXR + (a - s_coff[c]));
        }
    }
    __syncthreads();

    float lmax = 0.f;
    for (int a = tid; a < m; a += IDG_THREADS) {
        const Vec<D> x = cand[a];
        float rel[D];
        for (int k = 0; k < D; k++) rel[k] = vget(x, k) - ctr[k];
        float s2 = 0.f;
        float *row = A + (size_t)a * PP;
        for (int p = 0; p < P; p++) {
            float r2 = 0.f;
            for (int k = 0; k < D; k++) { const float df = rel[k] - prox[p * D + k]; r2 = fmaf(df, df, r2); }
            const float w = rkernel(r2);
            row[p] = w;
            s2 = fmaf(w, w, s2);
        }
        nrm[a] = s2;
        selpos[a] = -1;
        lmax = fmaxf(lmax, s2);
    }
    for (int o = 16; o > 0; o >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
    if (lane == 0) s_bv[wid] = lmax;
    __syncthreads();
    if (tid == 0) {
        float v = 0.f;
        for (int w = 0; w < IDG_THREADS / 32; w++) v = fmaxf(v, s_bv[w]);
        s_n0 = v;
    }
    __syncthreads();
    const float stop2 = g.tol2 * s_n0;
    const int rmax = min(min(m, P), MAXR);
    int r = 0;
    while (r < rmax) {
        float bv = -1.f;
        int bi = INT_MAX;
        for (int a = tid; a < m; a += IDG_THREADS)
            if (selpos[a] < 0 && (nrm[a] > bv)) { bv = nrm[a]; bi = a; }
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) { s_bv[wid] = bv; s_bi[wid] = bi; }
        __syncthreads();
        if (tid == 0) {
            float v = s_bv[0];
            int i = s_bi[0];
            for (int w = 1; w < IDG_THREADS / 32; w++)
                if (s_bv[w] > v || (s_bv[w] == v && s_bi[w] < i)) { v = s_bv[w]; i = s_bi[w]; }
            s_best = i;
            s_stop = (i == INT_MAX) || !(v > stop2) || !(v > 0.f);
        }
        __syncthreads();
        if (s_stop) break;
        const int best = s_best;
        const float rr = sqrtf(nrm[best]);
        const float inv = 1.0f / rr;
        float *q = A + (size_t)best * PP;
        for (int p = tid; p < P; p += IDG_THREADS) {
            const float v = q[p] * inv;
            q[p] = v;
            if (glob) A_s[p] = v;   // the shared-memory matrix area is free for a global-memory node
        }
        if (tid == 0) { selpos[best] = r; sel[r] = best; }
        __syncthreads();
        // G threads per row, each over every G-th proxy; the partial sums meet by shuffles inside
        // the group (whole warps take part in them). A matrix in global memory uses G = 8 and the
        // pivot row staged in shared memory, for more loads in flight per row.
        if (glob) gs_rows<8, P, PP>(A, A_s, m, tid, selpos, nrm, U, MAXR, r);
        else gs_rows<IDG_GROUP, P, PP>(A, q, m, tid, selpos, nrm, U, MAXR, r);
        __syncthreads();
        // column r of R11 (R[0..r-1][best] from the earlier steps, then the norm) into the
        // pivot row, which is dead from now on
        for (int k = tid; k <= r; k += IDG_THREADS) q[k] = k < r ? U[(size_t)best * MAXR + k] : rr;
        r++;
    }
    __syncthreads();
    for (int k = tid; k < r; k += IDG_THREADS) skel[(size_t)t * MAXR + k] = cand[sel[k]];
    if (tid == 0) g.rank[t] = r;
    // R11[k][j] = A[sel[j]][k]; a node whose matrix lives in global memory first copies R11 into
    // the (unused) shared-memory matrix area, column j at j (j + 1) / 2
    const float *R11 = A;
    if (glob) {
        float *R = A_s;
        for (int idx = tid; idx < r * r; idx += IDG_THREADS) {
            const int j = idx / r, k = idx % r;
            if (k <= j) R[j * (j + 1) / 2 + k] = A[(size_t)sel[j] * PP + k];
        }
        __syncthreads();
        R11 = R;
    }
    for (int a = tid; a < m; a += IDG_THREADS) {
        float *u = U + (size_t)a * MAXR;
        const int pos = selpos[a];
        if (pos >= 0) {
            for (int k = 0; k < r; k++) u[k] = (k == pos) ? 1.f : 0.f;
        } else if (glob) {
            for (int k = r - 1; k >= 0; k--) {
                float acc = u[k];
                for (int j = k + 1; j < r; j++) acc = fmaf(-R11[j * (j + 1) / 2 + k], u[j], acc);
                u[k] = acc / R11[k * (k + 1) / 2 + k];
            }
        } else {
            for (int k = r - 1; k >= 0; k--) {
                float acc = u[k];
                for (int j = k + 1; j < r; j++) acc = fmaf(-R11[(size_t)sel[j] * PP + k], u[j], acc);
                u[k] = acc / R11[(size_t)sel[k] * PP + k];
            }
        }
    }
    // upward pass of this node: y0[t] = U^T (the leaf's [1 | x] | the children's y0), groups of
    // RG threads over k and IDG_THREADS / RG groups over the rows, summed in a fixed order
    __syncthreads();
    {
        const int RG = r <= 16 ? 16 : (r <= 32 ? 32 : 64);
        const int C = IDG_THREADS / RG, kk = tid % RG, cg = tid / RG;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kk < r) {
            for (int a = cg; a < m; a += C) {
                const float w = U[(size_t)a * MAXR + kk];
                if (LEAVES) {
                    const Vec<D> x = cand[a];
                    acc.x += w;
                    acc.y = fmaf(w, vget(x, 0), acc.y);
                    acc.z = fmaf(w, vget(x, 1), acc.z);
                    if (D == 3) acc.w = fmaf(w, vget(x, 2), acc.w);
                } else {
                    int c = 0;
                    while (a >= s_coff[c + 1]) c++;
                    fma4(acc, w, __ldcg(g.y0 + (size_t)(tv.fchild[t] + c) * MAXR + (a - s_coff[c])));
                }
            }
        }
        s_part[tid] = acc;
        __syncthreads();
        if (tid < r) {
            float4 y = s_part[tid];
            for (int c = 1; c < C; c++) add4(y, s_part[c * RG + tid]);
            g.y0[(size_t)t * MAXR + tid] = y;
        }
    }
    if (items != nullptr && !LEAVES) {
        __syncthreads();
        if (tid == 0) dep_publish(dp, t);
    }
}



__device__ __forceinline__ float f2_sum(F2 a)
{
    float a0, a1;
    f2_unpack(a, a0, a1);
    return a0 + a1;
}

// Warp argmax of (norm, row): the largest norm, ties to the lowest row. Norms are >= 0 or -1
// (no candidate), so their bit patterns order like the values.
__device__ __forceinline__ void warp_argmax(float &bv, int &bi)
{
    const int key = __float_as_int(bv);
    const int mx = __reduce_max_sync(0xffffffffu, key);
    bi = __reduce_min_sync(0xffffffffu, key == mx ? bi : INT_MAX);
    bv = __int_as_float(mx);
}

// Interpolative decompositions of the 2D nodes at level >= 2, one CTA per node, two lanes per
// candidate row of A = K(candidate - c, proxies): lane l holds the row's entries of the proxies
// 4j + 2l, 4j + 2l + 1 as pairs for the paired FP32 instructions, NS rows per pair of lanes.
// LEAVES: the leaves of `items` (candidates = their points).
// Otherwise every internal node in one dependency-ordered launch (candidates = the children's
// skeletons): items in decreasing node id (deepest level first), so a node's internal children
// come before it; it waits for their first flags (skeleton and rank, published right after their
// Gram-Schmidt steps) and, before its own upward sums, for their second flags (coefficients,
// published last), and reads all of these through L2. When the children's ranks add up to more
// than 128, thread tid < 128 also owns row 128 + tid, kept in global memory (in the node's first U
// rows, unused until the end).
// Column-pivoted Gram-Schmidt until the largest residual row norm is <= tol * the largest
// initial one (ties: the lower row); the dot products of every step are kept in shared
// memory (row-major, stride MAXR + 1), R11 is gathered from the pivot rows into shared
// memory, and the back substitution U = [I ; R11^-1 R12]^T runs there, two columns per lane and
// four at a time. Then U goes out to global memory, with the skeleton and the
// rank, and the upward coefficients y0 = U^T (the leaf's [1 | x] | the children's y0) are summed
// in a fixed order (yt threads).
// What bounds it is a node's serial chain (rank x (pivot, barrier, dot product, update, argmax,
// barrier)) and, along the tree, the levels' chain. With a row per thread a step was 64 loads,
// 192 FMAs and the pivot's 64 stores by one thread, and a node's rows took 8,000 cycles to evaluate
// (one long stretch of code); two lanes have 48 paired FMAs (the same four partial sums p mod 4,
// joined in the same order). Four lanes per row had the same chain and twice the instructions (leaves at 1M
// points 563 us a rebuild). From a row per thread: leaves 62 -> 36 us at 20K points and 538 -> 443 us at
// 1M, internal nodes 143 -> 103 us and 537 -> 426 us (three CTAs of 168 registers per SM; four of 128
// spilled 184 bytes: 131 and 555 us).
constexpr int ID2_DSTRIDE = Dim<2>::MAXR + 1;
constexpr int ID2_HELD = 128;                     // rows in registers of the internal nodes' CTAs
constexpr int ID2_TINY = 32, ID2_SMALL = 64;      // leaves of the smaller CTAs
constexpr int ID2_ONE_LAUNCH = 148 * 4;           // leaves that one launch of the largest CTAs runs at once
template <int THREADS, int NS> constexpr size_t id2_smem() { return sizeof(float) * (THREADS / 2 * NS) * ID2_DSTRIDE; }
template <bool LEAVES, int THREADS, int NS>
constexpr int id2_min_blocks() { return !LEAVES ? 3 : NS == 2 ? 4 : (THREADS == 128 ? 5 : 10); }
// the leaves of a launch: the items of up to three lists, one after another
struct LeafItems {
    const int *list[3];
    int n[3];
};
__device__ __forceinline__ int leaf_item(const LeafItems &x, int i)
{
    if (i < x.n[0]) return x.list[0][i];
    i -= x.n[0];
    if (i < x.n[1]) return x.list[1][i];
    return x.list[2][i - x.n[1]];
}
static_assert(ID2_TINY == TINY_LEAF && ID2_SMALL == SMALL_LEAF, "the leaf lists are the launches'");

template <bool LEAVES, int THREADS, int NS>
__global__ void __launch_bounds__(THREADS, id2_min_blocks<LEAVES, THREADS, NS>())
k_id2d(int n_item, const int *items, LeafItems leaves, IdArgs g, DepArgs dp)
{
    after_previous();
    constexpr int P = Dim<2>::NPROXY, MAXR = Dim<2>::MAXR, NW = THREADS / 32;
    constexpr int PAIRS = THREADS / 2, HELD = PAIRS * NS, E = P / 4;
    constexpr int ROWS = LEAVES ? HELD : 4 * MAXR;   // candidate rows a CTA can hold
    constexpr int QS = 36;                           // stride of a lane's share of the pivot row
    static_assert(LEAVES || (HELD == ID2_HELD && ROWS <= 2 * HELD && P == MAXR), "overflow rows reuse U rows of MAXR floats");
    static_assert(P == 64 && NW <= 32 && THREADS >= MAXR, "16 pairs per lane");
    extern __shared__ float dots[];            // [HELD][ID2_DSTRIDE]
    __shared__ __align__(8) float px[P], py[P];
    __shared__ __align__(16) float qsh[2 * QS];   // the pivot row: proxy 4j + 2l + e at l QS + 2j + e
    __shared__ float rdiag[MAXR];
    __shared__ int piv[MAXR];
    __shared__ float R11[MAXR * (MAXR + 1) / 2];   // column jj at jj (jj + 1) / 2
    __shared__ float4 sin_[ROWS];
    __shared__ float4 part[THREADS];
    __shared__ float2 sxy[ROWS];
    __shared__ float s_bv[2][NW];
    __shared__ int s_bi[2][NW];
    __shared__ float s_lmax[NW];
    __shared__ int s_crank[4], s_item;
    const TreeView &tv = g.tv;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, ln = tid & 1;
    // internal nodes by level (items == nullptr): one launch per level, node n_item + block,
    // its children finished by the launches before, so nothing waits or publishes
    const bool bylevel = !LEAVES && items == nullptr;
    if (!LEAVES && !bylevel && tid == 0) s_item = atomicAdd(dp.ticket, 1);
    __syncthreads();
    int t;
    if (bylevel) {
        t = n_item + (int)blockIdx.x;
        if (tv.leaf[t]) return;   // uniform over the CTA
    } else {
        const int item = LEAVES ? (int)blockIdx.x : s_item;
        if (item >= n_item) return;
        t = LEAVES ? leaf_item(leaves, item) : items[n_item - 1 - item];
    }
    const int lvl = tv.level[t];
    const float2 *xt = (const float2 *)g.xt;
    float2 *skel = (float2 *)g.skel;
    const int cfirst = tv.fchild[t], nch = LEAVES ? 0 : tv.nchild[t];
    const int s0 = tv.start[t];
    const long long roff = g.rowoff[t];
    float *U = g.U + roff * MAXR;
    const double h = tv.info->radius / (double)(1LL << lvl);
    if (tid < P) {
        const float2 y = reinterpret_cast<const float2 *>(tv.proxies + (size_t)lvl * PROXY_F4)[tid];
        px[tid] = y.x;
        py[tid] = y.y;
    }
    const float cx = (float)(tv.info->corner[0] + (double)(2 * tv.ix[(size_t)t * 3 + 0] + 1) * h);
    const float cy = (float)(tv.info->corner[1] + (double)(2 * tv.ix[(size_t)t * 3 + 1] + 1) * h);
    if (!LEAVES && tid < nch) {
        if (!bylevel && !tv.leaf[cfirst + tid]) dep_wait(dp, cfirst + tid);   // leaves: the launch before
        s_crank[tid] = __ldcg(g.rank + cfirst + tid);
    }
    __syncthreads();
    int m = 0;
    if (LEAVES) m = tv.end[t] - s0;
    else for (int c = 0; c < nch; c++) m += s_crank[c];
    // candidates and the upward-pass inputs
    for (int a = tid; a < m; a += THREADS) {
        float2 pt;
        if (LEAVES) {
            pt = xt[s0 + a];
            sin_[a] = make_float4(1.f, pt.x, pt.y, 0.f);
        } else {
            int c = 0, aa = a;
            while (aa >= s_crank[c]) { aa -= s_crank[c]; c++; }
            pt = __ldcg(skel + (size_t)(cfirst + c) * MAXR + aa);
            if (bylevel) sin_[a] = __ldcg(g.y0 + (size_t)(cfirst + c) * MAXR + aa);
        }
        sxy[a] = pt;
    }
    __syncthreads();

    const int a0 = tid >> 1;                     // the lanes' rows: a0 + PAIRS s
    const int w0 = wid * 16;                     // the warp's first row; a set whose w0 + PAIRS s >= m is empty
    const bool big = !LEAVES && m > HELD;        // uniform over the block
    const bool xvalid = big && HELD + tid < m;
    F2 row[NS][E];
    float nrm[NS];
    int pos[NS], xpos = xvalid ? -1 : -2;        // -1: open row, -2: no row, >= 0: pivot position
    float xnrm = -1.f, lmax = 0.f, bv = -1.f;
    int bi = INT_MAX;
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const int a = a0 + PAIRS * s;
        const bool valid = a < m;
        pos[s] = valid ? -1 : -2;
        nrm[s] = -1.f;
        if (w0 + PAIRS * s >= m) continue;
        const float2 x = sxy[valid ? a : 0];
        const F2 rx = f2_pack(x.x - cx, x.x - cx), ry = f2_pack(x.y - cy, x.y - cy);
        F2 zz = f2_pack(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < E; j++) {
            const float2 qx = *reinterpret_cast<const float2 *>(px + 4 * j + 2 * ln);
            const float2 qy = *reinterpret_cast<const float2 *>(py + 4 * j + 2 * ln);
            const F2 dx = f2_sub(rx, f2_pack(qx.x, qx.y)), dy = f2_sub(ry, f2_pack(qy.x, qy.y));
            const F2 d = f2_add(f2_pack(1.f, 1.f), f2_fma(dx, dx, f2_mul(dy, dy)));
            float d0, d1;
            f2_unpack(d, d0, d1);
            const F2 w = f2_pack(fast_rcp(d0), fast_rcp(d1));
            row[s][j] = f2_mul(w, w);
            zz = f2_fma(row[s][j], row[s][j], zz);
        }
        float z = f2_sum(zz);
        z += __shfl_xor_sync(0xffffffffu, z, 1);
        if (valid) {
            nrm[s] = z;
            if (z > bv) { bv = z; bi = a; }
        }
    }
    float *xr = U + (size_t)tid * MAXR;   // overflow row, in the node's first U rows
    if (xvalid) {
        const float2 xx = sxy[HELD + tid];
        const float qx = xx.x - cx, qy = xx.y - cy;
        float z2 = 0.f;
        for (int p = 0; p < P; p++) {
            const float dx = qx - px[p], dy = qy - py[p];
            const float w = rkernel(fmaf(dx, dx, dy * dy));
            xr[p] = w;
            z2 = fmaf(w, w, z2);
        }
        xnrm = z2;
        if (xnrm > bv) { bv = xnrm; bi = HELD + tid; }
    }
    lmax = fmaxf(lmax, bv);
    lmax = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(lmax)));
    warp_argmax(bv, bi);
    if (lane == 0) { s_lmax[wid] = lmax; s_bv[0][wid] = bv; s_bi[0][wid] = bi; }
    __syncthreads();
    const float n0 = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(lane < NW ? s_lmax[lane] : 0.f)));
    const float stop2 = g.tol2 * n0;
    const int rmax = min(min(m, P), MAXR);
    int r = 0, buf = 0;
    while (r < rmax) {
        float v = lane < NW ? s_bv[buf][lane] : -1.f;
        int best = lane < NW ? s_bi[buf][lane] : INT_MAX;
        warp_argmax(v, best);
        if (best == INT_MAX || !(v > stop2) || !(v > 0.f)) break;
#pragma unroll
        for (int s = 0; s < NS; s++)
            if (best == a0 + PAIRS * s) {
                const float rr = __fsqrt_rn(nrm[s]);
                const float inv = __frcp_rn(rr);
                const F2 i2 = f2_pack(inv, inv);
#pragma unroll
                for (int j = 0; j < E; j += 2) {
                    float4 y;
                    f2_unpack(f2_mul(row[s][j], i2), y.x, y.y);
                    f2_unpack(f2_mul(row[s][j + 1], i2), y.z, y.w);
                    *reinterpret_cast<float4 *>(qsh + ln * QS + 2 * j) = y;
                }
                if (ln == 0) { rdiag[r] = rr; piv[r] = best; }
                pos[s] = r;
                nrm[s] = -1.f;
            }
        if (xvalid && best == HELD + tid) {
            const float rr = __fsqrt_rn(xnrm);
            const float inv = __frcp_rn(rr);
            for (int p = 0; p < P; p++) qsh[((p >> 1) & 1) * QS + 2 * (p >> 2) + (p & 1)] = xr[p] * inv;
            rdiag[r] = rr;
            piv[r] = best;
            xpos = r;
            xnrm = -1.f;
        }
        __syncthreads();
        bv = -1.f;
        bi = INT_MAX;
        if (w0 < m) {   // uniform over the warp
            F2 q[E];
#pragma unroll
            for (int j = 0; j < E; j += 2) {
                const float4 y = *reinterpret_cast<const float4 *>(qsh + ln * QS + 2 * j);
                q[j] = f2_pack(y.x, y.y);
                q[j + 1] = f2_pack(y.z, y.w);
            }
#pragma unroll
            for (int s = 0; s < NS; s++) {
                if (w0 + PAIRS * s >= m) continue;
                F2 d2 = f2_pack(0.f, 0.f), zz = d2;
#pragma unroll
                for (int j = 0; j < E; j++) d2 = f2_fma(q[j], row[s][j], d2);
                float dot = f2_sum(d2);
                dot += __shfl_xor_sync(0xffffffffu, dot, 1);
                const F2 nd = f2_pack(-dot, -dot);
#pragma unroll
                for (int j = 0; j < E; j++) {
                    row[s][j] = f2_fma(nd, q[j], row[s][j]);
                    zz = f2_fma(row[s][j], row[s][j], zz);
                }
                float z = f2_sum(zz);
                z += __shfl_xor_sync(0xffffffffu, z, 1);
                if (pos[s] == -1) {
                    nrm[s] = z;
                    if (ln == 0) dots[(a0 + PAIRS * s) * ID2_DSTRIDE + r] = dot;
                    if (z > bv) { bv = z; bi = a0 + PAIRS * s; }
                }
            }
        }
        if (xpos == -1) {
            float dot = 0.f;
            for (int p = 0; p < P; p++) dot = fmaf(qsh[((p >> 1) & 1) * QS + 2 * (p >> 2) + (p & 1)], xr[p], dot);
            float s2 = 0.f;
            for (int p = 0; p < P; p++) {
                const float y = fmaf(-dot, qsh[((p >> 1) & 1) * QS + 2 * (p >> 2) + (p & 1)], xr[p]);
                xr[p] = y;
                s2 = fmaf(y, y, s2);
            }
            xnrm = s2;
            U[(size_t)(HELD + tid) * MAXR + r] = dot;
            if (s2 > bv) { bv = s2; bi = HELD + tid; }
        }
        warp_argmax(bv, bi);
        buf ^= 1;
        if (lane == 0) { s_bv[buf][wid] = bv; s_bi[buf][wid] = bi; }
        r++;
        __syncthreads();
    }
    __syncthreads();
    // skeleton and rank; R11 from the pivot rows' dot products (column jj: its entries k < jj)
#pragma unroll
    for (int s = 0; s < NS; s++)
        if (ln == 0 && pos[s] >= 0) skel[(size_t)t * MAXR + pos[s]] = sxy[a0 + PAIRS * s];
    if (xpos >= 0) skel[(size_t)t * MAXR + xpos] = sxy[HELD + tid];
    if (tid == 0) g.rank[t] = r;
    for (int jj = wid; jj < r; jj += NW) {
        const int pr = piv[jj];
        for (int k = lane; k <= jj; k += 32)
            R11[jj * (jj + 1) / 2 + k] = k == jj ? rdiag[jj]
                                                 : (pr < HELD ? dots[pr * ID2_DSTRIDE + k] : U[(size_t)pr * MAXR + k]);
    }
    __syncthreads();
    // the skeleton and the rank are what the parent's decomposition needs: published here;
    // the children's upward coefficients, published last, are waited for before the sums
    if (!LEAVES && !bylevel) {
        if (tid == 0) dep_publish(dp, t);
        if (tid < nch && !tv.leaf[cfirst + tid]) dep_wait_y0(dp, cfirst + tid);
        __syncthreads();
        for (int a = tid; a < m; a += THREADS) {
            int c = 0, aa = a;
            while (aa >= s_crank[c]) { aa -= s_crank[c]; c++; }
            sin_[a] = __ldcg(g.y0 + (size_t)(cfirst + c) * MAXR + aa);
        }
    }
    // back substitution of the open rows: columns top, top - 1 by the first lane, top - 2, top - 3 by
    // the second, each column taking the later columns k in decreasing order, then its division
#pragma unroll
    for (int s = 0; s < NS; s++) {
        if (w0 + PAIRS * s >= m) continue;
        float *u = dots + (a0 + PAIRS * s) * ID2_DSTRIDE;
        const bool open = pos[s] == -1;
        for (int top = r - 1; top >= 0; top -= 4) {
            const int ca = max(top - 2 * ln, 0), cb = max(top - 2 * ln - 1, 0);
            float acc0 = u[ca], acc1 = u[cb];
            const float *col = R11 + (r - 1) * r / 2;   // column r - 1; column k - 1 lies k before column k
            for (int k = r - 1; k > top; col -= k, k--) {
                const float uk = u[k];
                acc0 = fmaf(-col[ca], uk, acc0);
                acc1 = fmaf(-col[cb], uk, acc1);
            }
#pragma unroll
            for (int z = 0; z < 4; z++) {
                if (top - z < 0) break;
                const float *cz = R11 + (top - z) * (top - z + 1) / 2;
                const float uk = __shfl_sync(0xffffffffu, ((z & 1) ? acc1 : acc0) / cz[top - z], z >> 1, 2);
                if (ln == z >> 1 && open) u[top - z] = uk;
                if (2 * ln > z) acc0 = fmaf(-cz[ca], uk, acc0);
                if (2 * ln + 1 > z) acc1 = fmaf(-cz[cb], uk, acc1);
            }
            __syncwarp();
        }
        if (pos[s] >= 0)   // pivot rows are rows of the identity
            for (int k = ln; k < r; k += 2) u[k] = k == pos[s] ? 1.f : 0.f;
    }
    if (xpos == -1) {
        float *u = U + (size_t)(HELD + tid) * MAXR;
        for (int k = r - 1; k >= 0; k--) {
            float acc = u[k];
            for (int jj = k + 1; jj < r; jj++) acc = fmaf(-R11[jj * (jj + 1) / 2 + k], u[jj], acc);
            u[k] = acc / R11[k * (k + 1) / 2 + k];
        }
    }
    if (xpos >= 0)
        for (int k = 0; k < r; k++) U[(size_t)(HELD + tid) * MAXR + k] = k == xpos ? 1.f : 0.f;
    __syncthreads();
    // U rows 0 .. min(m, HELD) - 1 out of shared memory (over the overflow rows' scratch)
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const int a = a0 + PAIRS * s;
        if (a >= m) continue;
        const float *u = dots + a * ID2_DSTRIDE;
        float *o = U + (size_t)a * MAXR;
        for (int k = 4 * ln; k < r; k += 8) {
            if (k + 3 < r) *reinterpret_cast<float4 *>(o + k) = make_float4(u[k], u[k + 1], u[k + 2], u[k + 3]);
            else
                for (int z = k; z < r; z++) o[z] = u[z];
        }
    }
    // y0[k] = sum_a U[a][k] in[a]: groups of RG threads over k, C = yt / RG groups over a
    const int yt = LEAVES && m <= ID2_SMALL ? 64 : 128;
    const int RG = r <= 16 ? 16 : (r <= 32 ? 32 : 64);
    const int C = yt / RG, kk = tid & (RG - 1), cg = tid / RG;
    static_assert(THREADS >= (LEAVES && HELD <= ID2_SMALL ? 64 : 128), "a thread per part");
    if (tid < yt) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kk < r) {
            for (int a = cg; a < m; a += C) {
                const float w = a < HELD ? dots[a * ID2_DSTRIDE + kk] : U[(size_t)a * MAXR + kk];
                fma4(acc, w, sin_[a]);
            }
        }
        part[tid] = acc;
    }
    __syncthreads();
    if (tid < r) {
        float4 y = part[tid];
        for (int c = 1; c < C; c++) add4(y, part[c * RG + tid]);
        g.y0[(size_t)t * MAXR + tid] = y;
    }
    if (!LEAVES && !bylevel) {
        __syncthreads();
        if (tid == 0) dep_publish_y0(dp, t);
    }
}

// ---------------------------------------------------------------------------------
// 3D interpolative decompositions
// ---------------------------------------------------------------------------------
// The 3D proxy matrix has 216 columns and up to 512 candidate rows (eight children of rank
// <= 64). The column-pivoted Gram-Schmidt runs left-looking, so the matrix is never changed:
// step r takes the row b of the largest residual norm and orthonormalises it against the earlier
// directions q_0..q_{r-1} by classical Gram-Schmidt applied twice (the first pass from b's stored
// projections, the second recomputed, so the directions stay orthonormal to rounding); every
// other row a then takes its dot product c = a . q_r (= its residual's, as q_r is orthogonal to
// the earlier directions), kept in shared memory as R12, with its squared residual norm
// downdated in FP64 by c^2. R11's column r is b's projections on q_0..q_{r-1} and its residual
// norm. The stop rule, tie rule, back substitution U = [I ; R11^-1 R12]^T and the upward
// coefficients are those of k_id.
//
// The rows' entries (1 + |x|^2 + |p|^2 - 2 x.p)^-2 (x: candidate relative to the node's centre, p:
// proxy; one reciprocal each) are evaluated once and held: the first THREADS / 4 rows in
// registers (at most 28 pairs of proxies per lane, four lanes or more per row), of a node with more
// candidates the next ones in the shared memory that is left, and only rows beyond that are
// evaluated again in every step. Evaluating every row in every step kept the reciprocal pipe at a
// quarter of its rate and the rows' pass at 18 instructions per pair of entries; held, a pair is
// one load and one paired FMA. At 100K points (h2_tol 3e-2, late in a run; nodes of 178 candidates
// and rank 42 on average) the internal launch went from 2,034 to 1,580 us, the leaves' from 928 to
// 731 us a rebuild. It is bound by the chain of the largest nodes (420 candidates, of which about
// 245 are evaluated in every step) and by the latencies of a step: the pivot's two
// orthonormalisations take about half of it.
//
// The proxies go in pairs (2j, 2j + 1) for the paired FP32 instructions. A row's dot product is S
// chains over the pairs j = c mod S in increasing j (S = 16, 8, 4, 2 by the number of rows against
// the threads), joined by butterfly shuffles. A row held by as many lanes as chains has a chain
// per lane; with S = 2, four lanes hold a row, and the chain's first 28 pairs and its last 26 are
// two lanes', the second going on from the first's sum. S and the order of a chain are part of
// the result's rounding, so they do not depend on where a row is held.
//
// One CTA per node: 128 threads (leaves of at most 32 points), 256 (33..64), 512 (the others).
//
// Internal nodes run in one dependency-ordered launch: a node waits for its internal
// children's skeletons and ranks (flag), published right after their pivot loop, and, before
// its upward coefficients, for their coefficients (second flag, published last).
constexpr int ID3_P = Dim<3>::NPROXY;
constexpr int ID3_NP = ID3_P / 2;            // proxy pairs
constexpr int ID3_ROWS = 8 * Dim<3>::MAXR;   // candidate rows of an internal node
constexpr int ID3_QS = 220;                  // row stride of the directions (16-byte rows,
                                             // conflict-free for 4 lanes x 8 directions)
constexpr int ID3_TINY = 32;                 // leaves of the 128-thread CTAs
constexpr int ID3_SMALL = 64;                // leaves of the 256-thread CTAs
constexpr int ID3_MID = 128;                 // leaves whose rows a 512-thread CTA holds in registers
constexpr int ID3_HELD = 28;                 // most pairs per lane
constexpr int ID3_VP = 400;                  // the residual in the lanes' order (id3_place)
static_assert(ID3_TINY == TINY_LEAF && ID3_SMALL == SMALL_LEAF, "the leaf lists are the launches'");
static_assert(ID3_P % 8 == 0 && ID3_QS >= ID3_P && ID3_QS % 4 == 0, "proxy pairs, 16-byte rows");

template <int THREADS, int ROWS>
struct Id3 {
    static constexpr int QR = ROWS < Dim<3>::MAXR ? ROWS : Dim<3>::MAXR;   // rank bound
    static constexpr int CS = QR + 1;                                      // row stride of R12 / U
    static constexpr int NW = THREADS / 32;
    static constexpr int REG_ROWS = THREADS / 4;                           // rows held in registers
    static constexpr int NK = ROWS > REG_ROWS ? (ROWS - REG_ROWS + THREADS / 2 - 1) / (THREADS / 2) : 0;
    static_assert(THREADS >= 4 * QR || ROWS < QR * 2, "four lanes per direction");
    struct Smem {
        float Q[QR * ID3_QS];                  // directions q_0..q_{r-1}; at the end: y0 partials
        float4 pa[ID3_NP];                     // proxy pairs: (-2x, -2x', -2y, -2y')
        float4 pb[ID3_NP];                     //              (-2z, -2z', |p|^2, |p'|^2)
        float R11[QR * (QR + 1) / 2];          // column j at j (j + 1) / 2
        float4 vp[ID3_VP / 4];                 // the residual's pairs in the order of the rows' lanes
        float4 red[(NW + 3) / 4];
        float res[ID3_P];                      // the pivot's residual
        float dc[QR];                          // its second-pass projections
        int piv[QR];
        float bv[2][NW];
        int bi[2][NW];
        int coff[9];
        int item;
    };
    static_assert(QR * ID3_QS * sizeof(float) >= THREADS * sizeof(float4), "y0 partials in the directions");
    // the parts sized by the node's rows m follow: candidates ((x, y, z) - centre, 1 + |.|^2),
    // pivot position of each row or -1, R12 (the rows' dots, then U), held entries
    static constexpr size_t fixed() { return (sizeof(Smem) + 15) / 16 * 16; }
    static constexpr size_t sized(int m) { return (size_t)m * (sizeof(float4) + sizeof(int) + sizeof(float) * CS); }
    static constexpr size_t row_bytes() { return sizeof(float2) * ID3_NP; }
    static constexpr size_t most() { return 227 * 1024; }
    static constexpr size_t smem() { return ROWS > REG_ROWS ? most() : fixed() + sized(ROWS) + 16; }
    static_assert(fixed() + sized(ROWS) + 16 <= most(), "a node of ROWS candidates fits");
};

// entry of proxy p (scalar form of the paired arithmetic below: the same operations in the
// same order, so both give the same value)
template <typename SM>
__device__ __forceinline__ float id3_entry(const SM &s, const float4 &c, int p)
{
    const float4 A = s.pa[p >> 1], B = s.pb[p >> 1];
    const bool o = p & 1;
    const float mx = o ? A.y : A.x, my = o ? A.w : A.z, mz = o ? B.y : B.x, e = o ? B.w : B.z;
    const float d = fmaf(c.z, mz, fmaf(c.y, my, fmaf(c.x, mx, c.w + e)));
    const float w = fast_rcp(d);
    return w * w;
}
// entries of the pair j of candidate c
template <typename SM>
__device__ __forceinline__ F2 id3_pair(const SM &s, const float4 &c, int j)
{
    const float4 A = s.pa[j], B = s.pb[j];
    const F2 mx = f2_pack(A.x, A.y), my = f2_pack(A.z, A.w), mz = f2_pack(B.x, B.y), e = f2_pack(B.z, B.w);
    const F2 d = f2_fma(f2_pack(c.z, c.z), mz,
                        f2_fma(f2_pack(c.y, c.y), my, f2_fma(f2_pack(c.x, c.x), mx, f2_add(f2_pack(c.w, c.w), e))));
    float d0, d1;
    f2_unpack(d, d0, d1);
    const F2 w = f2_pack(fast_rcp(d0), fast_rcp(d1));
    return f2_mul(w, w);
}
__device__ __forceinline__ void id3_norm2(F2 w, double &dn)
{
    float a0, a1;
    f2_unpack(w, a0, a1);
    dn = fma((double)a0, (double)a0, dn);
    dn = fma((double)a1, (double)a1, dn);
}
__device__ __forceinline__ F2 id3_v(const float *v, int j)
{
    const float2 x = *reinterpret_cast<const float2 *>(v + 2 * j);
    return f2_pack(x.x, x.y);
}

// The lane's part of a row in registers. S >= 4: a lane per chain, lane q holds the pairs q + S i.
// S == 2: four lanes, lane q (chain q & 1, half q >> 1) holds the pairs (q & 1) + 2 (28 (q >> 1) + i).
__device__ __forceinline__ int id3_log2(int S) { return S == 2 ? 1 : S == 4 ? 2 : S == 8 ? 3 : 4; }
__device__ __forceinline__ int id3_count(int S, int q)
{
    return S == 2 ? (q >> 1 ? 26 : 28) : (ID3_NP - q + S - 1) >> id3_log2(S);
}
__device__ __forceinline__ int id3_held_pair(int S, int q, int i) { return S == 2 ? (q & 1) + 2 * (28 * (q >> 1) + i) : q + S * i; }
// The place of pair j of the residual, so that a lane's pairs lie together and two are one 16-byte
// load (the lanes' starts fall on different banks).
__device__ __forceinline__ int id3_stride(int S) { return S <= 4 ? 28 : S == 8 ? 16 : 12; }
__device__ __forceinline__ int id3_place(int S, int j)
{
    return S == 2 ? (j & 1) * 56 + (j >> 1) : (j & (S - 1)) * id3_stride(S) + (j >> id3_log2(S));
}
__device__ __forceinline__ int id3_start(int S, int q) { return S == 2 ? (q & 1) * 56 + (q >> 1) * 28 : q * id3_stride(S); }

// w: the lane's entries, zeros after its last; dn: the row's squared norm
template <typename SM>
__device__ __forceinline__ void id3_hold(const SM &s, const float4 &c, int S, int q, F2 (&w)[ID3_HELD], double &dn)
{
    const int n = id3_count(S, q);
    dn = 0.0;
#pragma unroll
    for (int i = 0; i < ID3_HELD; i++) {
        w[i] = f2_pack(0.f, 0.f);
        if (i < n) w[i] = id3_pair(s, c, id3_held_pair(S, q, i));
        id3_norm2(w[i], dn);   // (a zero leaves it as it is)
    }
    if (S == 2) {
        const double head = __shfl_xor_sync(0xffffffffu, dn, 2);
        dn = head;   // in the second half: the chain's sum so far
#pragma unroll
        for (int i = 0; i < 26; i++) {
            asm volatile("" : "+l"(w[i].v));   // converted again here, not held as 56 doubles
            id3_norm2(w[i], dn);
        }
    }
    for (int o = 1; o < S; o <<= 1) dn += __shfl_xor_sync(0xffffffffu, dn, o);
}
// acc = fma(w[i], v[i], acc) over the lane's pairs, four at a time. Past its last pair the lane
// holds zeros, and the residual's places there hold finite values: the sum is unchanged.
__device__ __forceinline__ F2 id3_chain(const F2 (&w)[ID3_HELD], const float4 *v, int n, F2 acc)
{
#pragma unroll
    for (int i = 0; i < ID3_HELD; i += 4) {
        if (i >= n) break;   // uniform: n is the longest lane's
        const float4 x = v[i / 2], y = v[i / 2 + 1];
        acc = f2_fma(w[i], f2_pack(x.x, x.y), acc);
        acc = f2_fma(w[i + 1], f2_pack(x.z, x.w), acc);
        acc = f2_fma(w[i + 2], f2_pack(y.x, y.y), acc);
        acc = f2_fma(w[i + 3], f2_pack(y.z, y.w), acc);
    }
    return acc;
}
// The row's dot product with the residual (complete in every lane; S == 2: in the lanes of the
// second half). n: the longest lane's pairs.
__device__ __forceinline__ float id3_dot_held(const float4 *v, int n, int S, const F2 (&w)[ID3_HELD])
{
    F2 acc = id3_chain(w, v, n, f2_pack(0.f, 0.f));
    if (S == 2) {
        acc.v = __shfl_xor_sync(0xffffffffu, acc.v, 2);   // in the second half: the chain's sum so far
        const float y = f2_sum(id3_chain(w, v, n, acc));
        return __fadd_rn(y, __shfl_xor_sync(0xffffffffu, y, 1));   // = the FP64 sum of two, rounded
    }
    double out = (double)f2_sum(acc);
    for (int o = 1; o < S; o <<= 1) out += __shfl_xor_sync(0xffffffffu, out, o);
    return (float)out;
}

// d[j] = q_j . res for the directions j < r (four lanes per direction, 54 proxies each)
template <typename SM>
__device__ __forceinline__ void id3_proj(SM &s, int r, int tid, float *d)
{
    const int j = tid >> 2, sub = tid & 3;
    float d0 = 0.f, d1 = 0.f;
    if (j < r) {
        const float *qj = s.Q + j * ID3_QS;
#pragma unroll
        for (int i = 0; i < ID3_P / 8; i++) {
            const int p = sub + 8 * i;
            d0 = fmaf(qj[p], s.res[p], d0);
            d1 = fmaf(qj[p + 4], s.res[p + 4], d1);
        }
    }
    float x = d0 + d1;
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    if (sub == 0 && j < r) d[j] = x;
}

// v - sum_{j < r} d[j] q_j[p]
__device__ __forceinline__ float id3_sub(const float *Q, int r, int p, const float *d, float v)
{
    float a0 = v, a1 = 0.f, a2 = 0.f, a3 = 0.f;
    int j = 0;
#pragma unroll 2
    for (; j + 3 < r; j += 4) {
        a0 = fmaf(-d[j], Q[j * ID3_QS + p], a0);
        a1 = fmaf(-d[j + 1], Q[(j + 1) * ID3_QS + p], a1);
        a2 = fmaf(-d[j + 2], Q[(j + 2) * ID3_QS + p], a2);
        a3 = fmaf(-d[j + 3], Q[(j + 3) * ID3_QS + p], a3);
    }
    for (; j < r; j++) a0 = fmaf(-d[j], Q[j * ID3_QS + p], a0);
    return (a0 + a1) + (a2 + a3);
}

template <int THREADS>
constexpr int id3_min_blocks() { return THREADS >= 512 ? 1 : (THREADS >= 256 ? 2 : 4); }

// LEAVES: the leaves of `items` with mlo < points <= ROWS (others are another launch's); `chains`
// is the thread count by which S is chosen.
template <bool LEAVES, int THREADS, int ROWS>
__global__ void __launch_bounds__(THREADS, id3_min_blocks<THREADS>())
k_id3(int n_item, const int *items, int mlo, int chains, IdArgs g, DepArgs dp)
{
    after_previous();
    using K = Id3<THREADS, ROWS>;
    using SM = typename K::Smem;
    constexpr int P = ID3_P, MAXR = Dim<3>::MAXR, QR = K::QR, CS = K::CS, NW = K::NW, NK = K::NK;
    constexpr int PPT = (P + THREADS - 1) / THREADS;   // proxies per thread in the pivot's steps
    extern __shared__ __align__(16) unsigned char smraw[];
    SM &s = *reinterpret_cast<SM *>(smraw);
    const TreeView &tv = g.tv;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (!LEAVES && tid == 0) s.item = atomicAdd(dp.ticket, 1);
    __syncthreads();
    const int item = LEAVES ? (int)blockIdx.x : s.item;
    if (item >= n_item) return;
    const int t = items[LEAVES ? item : n_item - 1 - item];
    if (LEAVES) {
        const int mm = tv.end[t] - tv.start[t];
        if (mm <= mlo || mm > ROWS) return;   // uniform over the CTA
    }
    const int cfirst = tv.fchild[t], nch = LEAVES ? 0 : tv.nchild[t];
    const int s0 = tv.start[t];
    const int lvl = tv.level[t];
    const long long roff = g.rowoff[t];
    float *U = g.U + roff * MAXR;
    const float4 *xt = (const float4 *)g.xt;
    float4 *skel = (float4 *)g.skel;
    for (int j = tid; j < ID3_NP; j += THREADS) {
        const float4 *row = tv.proxies + (size_t)lvl * PROXY_F4;
        s.pa[j] = row[j];
        s.pb[j] = row[ID3_NP + j];
    }
    for (int j = tid; j < ID3_VP / 4; j += THREADS) s.vp[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    const double h = tv.info->radius / (double)(1LL << lvl);
    float ctr[3];
    for (int k = 0; k < 3; k++)
        ctr[k] = (float)(tv.info->corner[k] + (double)(2 * tv.ix[(size_t)t * 3 + k] + 1) * h);
    if (!LEAVES && tid < nch && !tv.leaf[cfirst + tid]) dep_wait(dp, cfirst + tid);
    __syncthreads();
    if (!LEAVES) {
        if (tid < nch) s.coff[tid + 1] = __ldcg(g.rank + cfirst + tid);
        __syncthreads();
        if (tid == 0) {
            s.coff[0] = 0;
            for (int c = 0; c < nch; c++) s.coff[c + 1] += s.coff[c];
        }
        __syncthreads();
    }
    const int m = LEAVES ? tv.end[t] - tv.start[t] : s.coff[nch];
    float4 *cand = reinterpret_cast<float4 *>(smraw + K::fixed());
    int *selpos = reinterpret_cast<int *>(cand + m);
    float *C = reinterpret_cast<float *>(selpos + m);
    for (int a = tid; a < m; a += THREADS) {
        float4 x;
        if (LEAVES) x = xt[s0 + a];
        else {
            int c = 0;
            while (a >= s.coff[c + 1]) c++;
            x = __ldcg(skel + (size_t)(cfirst + c) * MAXR + (a - s.coff[c]));
        }
        const float rx = x.x - ctr[0], ry = x.y - ctr[1], rz = x.z - ctr[2];
        cand[a] = make_float4(rx, ry, rz, 1.f + fmaf(rx, rx, fmaf(ry, ry, rz * rz)));
        selpos[a] = -1;
    }
    __syncthreads();

    int S = 2;   // chains per row; uniform over the CTA
    while (S < 16 && chains / (2 * S) >= m) S <<= 1;
    const int lanes = S > 4 ? S : 4, q = tid & (lanes - 1), ra = tid >> (S > 4 ? id3_log2(S) : 2);
    // the lane that keeps a register row's state (its sums are complete there)
    const bool keeper = q == (S == 2 ? 2 : 0);
    const int held_n = id3_count(S, 0);
    const float4 *vrow = s.vp + id3_start(S, q) / 2;
    F2 w[ID3_HELD];
    double nrm = -1.0, nrx[NK > 0 ? NK : 1];
    int pos = -2, pox[NK > 0 ? NK : 1];   // -1: open row, -2: no row, >= 0: pivot position
    {
        const float4 c = cand[ra < m ? ra : 0];
        id3_hold(s, c, S, q, w, nrm);
        if (ra < m && keeper) pos = -1;
        else nrm = -1.0;
    }
    // further rows (S = 2): two lanes each, in shared memory while it lasts
    const int mx = NK > 0 ? max(0, m - K::REG_ROWS) : 0;
    float4 *held = reinterpret_cast<float4 *>(((uintptr_t)(C + (size_t)m * CS) + 15) & ~(uintptr_t)15);
    const int nheld = NK > 0 ? min(mx, (int)((smraw + K::most() - reinterpret_cast<unsigned char *>(held)) / (int)K::row_bytes())) : 0;
    const int ch = tid & 1;
#pragma unroll
    for (int k = 0; k < NK; k++) {
        const int x = tid / 2 + k * (THREADS / 2);
        double dn = 0.0;
        pox[k] = -2;
        if (x < mx) {
            const float4 c = cand[K::REG_ROWS + x];
            for (int i = 0; i < ID3_NP / 4; i++) {   // the chain's pairs 2i and 2i + 1
                const F2 e0 = id3_pair(s, c, ch + 4 * i), e1 = id3_pair(s, c, ch + 4 * i + 2);
                if (x < nheld) {
                    float4 e;
                    f2_unpack(e0, e.x, e.y);
                    f2_unpack(e1, e.z, e.w);
                    held[i * 2 * nheld + 2 * x + ch] = e;
                }
                id3_norm2(e0, dn);
                id3_norm2(e1, dn);
            }
        }
        dn += __shfl_xor_sync(0xffffffffu, dn, 1);
        nrx[k] = -1.0;
        if (x < mx && ch == 0) { pox[k] = -1; nrx[k] = dn; }
    }
    float bv = -1.f, lmax = 0.f;
    int bi = INT_MAX;
    if (pos == -1) {
        const float v = (float)nrm;
        lmax = fmaxf(lmax, v);
        if (v > bv) { bv = v; bi = ra; }
    }
#pragma unroll
    for (int k = 0; k < NK; k++)
        if (pox[k] == -1) {
            const float v = (float)nrx[k];
            lmax = fmaxf(lmax, v);
            if (v > bv) { bv = v; bi = K::REG_ROWS + tid / 2 + k * (THREADS / 2); }
        }
    lmax = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(lmax)));
    warp_argmax(bv, bi);
    if (lane == 0) { reinterpret_cast<float *>(s.red)[wid] = lmax; s.bv[0][wid] = bv; s.bi[0][wid] = bi; }
    __syncthreads();
    float *red = reinterpret_cast<float *>(s.red);
    const float n0 = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(lane < NW ? red[lane] : 0.f)));
    __syncthreads();   // red is used again
    const float stop2 = g.tol2 * n0;
    const int rmax = min(min(m, P), QR);
    int r = 0, buf = 0;
    while (r < rmax) {
        float v = lane < NW ? s.bv[buf][lane] : -1.f;
        int best = lane < NW ? s.bi[buf][lane] : INT_MAX;
        warp_argmax(v, best);
        if (best == INT_MAX || !(v > stop2) || !(v > 0.f)) break;
        // the pivot's residual: thread tid takes the proxies tid + THREADS i
        const float *cb = C + best * CS;   // the pivot's projections on q_0..q_{r-1}
        float rv[PPT];
#pragma unroll
        for (int i = 0; i < PPT; i++) {
            const int p = tid + THREADS * i;
            rv[i] = 0.f;
            if (p < P) {
                rv[i] = id3_sub(s.Q, r, p, cb, id3_entry(s, cand[best], p));
                s.res[p] = rv[i];
            }
        }
        __syncthreads();
        if (r > 0) id3_proj(s, r, tid, s.dc);   // uniform
        __syncthreads();
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < PPT; i++) {
            const int p = tid + THREADS * i;
            if (p < P) {
                rv[i] = id3_sub(s.Q, r, p, s.dc, rv[i]);
                reinterpret_cast<float *>(s.vp)[2 * id3_place(S, p >> 1) + (p & 1)] = rv[i];
                sq = fmaf(rv[i], rv[i], sq);
            }
        }
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (lane == 0) red[wid] = sq;
        __syncthreads();
        float rr2 = 0.f;   // the warps that have proxies, in order
        constexpr int PW = NW < (P + 31) / 32 ? NW : (P + 31) / 32;
#pragma unroll
        for (int x = 0; x < PW; x += 4) {
            const float4 y = s.red[x / 4];
            rr2 += y.x;
            if (x + 1 < PW) rr2 += y.y;
            if (x + 2 < PW) rr2 += y.z;
            if (x + 3 < PW) rr2 += y.w;
        }
        const float rr = __fsqrt_rn(rr2);
        if (!(rr > 0.f) || !(rr < INFINITY)) break;   // uniform: every thread sums the same values
        const float inv = __frcp_rn(rr);
#pragma unroll
        for (int i = 0; i < PPT; i++)
            if (tid + THREADS * i < P) s.Q[r * ID3_QS + tid + THREADS * i] = rv[i] * inv;
        if (tid < r) s.R11[r * (r + 1) / 2 + tid] = cb[tid] + s.dc[tid];
        if (tid == r) s.R11[r * (r + 1) / 2 + r] = rr;
        if (tid == 0) { s.piv[r] = best; selpos[best] = r; }
        if (pos == -1 && ra == best) pos = r;
        // every open row: c = a . q_r (from the unscaled residual), its R12 entry; squared
        // residual norm -= c^2
        bv = -1.f;
        bi = INT_MAX;
        const float part = id3_dot_held(vrow, held_n, S, w);
        if (pos == -1) {
            const float c = part * inv;
            nrm = fmax(nrm - (double)c * (double)c, 0.0);
            C[ra * CS + r] = c;
            const float nv = (float)nrm;
            if (nv > bv) { bv = nv; bi = ra; }
        }
#pragma unroll
        for (int k = 0; k < NK; k++) {
            if (k * (THREADS / 2) >= mx) break;   // uniform
            const int x = tid / 2 + k * (THREADS / 2), a = K::REG_ROWS + x;
            F2 acc = f2_pack(0.f, 0.f);
            if (x < nheld) {
                const float4 *e = held + 2 * x + ch, *v4 = s.vp + ch * 28;
#pragma unroll 9
                for (int i = 0; i < ID3_NP / 4; i++) {
                    const float4 y = e[i * 2 * nheld], v = v4[i];
                    acc = f2_fma(f2_pack(y.x, y.y), f2_pack(v.x, v.y), acc);
                    acc = f2_fma(f2_pack(y.z, y.w), f2_pack(v.z, v.w), acc);
                }
            } else if (x < mx) {
                const float4 c = cand[a];
                const float *v2 = reinterpret_cast<const float *>(s.vp);
#pragma unroll 2
                for (int i = 0; i < ID3_NP / 2; i++)
                    acc = f2_fma(id3_pair(s, c, ch + 2 * i), id3_v(v2, ch * 56 + i), acc);
            }
            const float y = f2_sum(acc), px = __fadd_rn(y, __shfl_xor_sync(0xffffffffu, y, 1));
            if (pox[k] == -1 && a == best) pox[k] = r;
            if (pox[k] == -1) {
                const float c = px * inv;
                nrx[k] = fmax(nrx[k] - (double)c * (double)c, 0.0);
                C[a * CS + r] = c;
                const float nv = (float)nrx[k];
                if (nv > bv) { bv = nv; bi = a; }
            }
        }
        warp_argmax(bv, bi);
        buf ^= 1;
        if (lane == 0) { s.bv[buf][wid] = bv; s.bi[buf][wid] = bi; }
        r++;
        __syncthreads();
    }
    __syncthreads();
    // skeleton and rank, published before the rest (the parent's candidates)
    for (int k = tid; k < r; k += THREADS) {
        const int a = s.piv[k];
        float4 x;
        if (LEAVES) x = xt[s0 + a];
        else {
            int c = 0;
            while (a >= s.coff[c + 1]) c++;
            x = __ldcg(skel + (size_t)(cfirst + c) * MAXR + (a - s.coff[c]));
        }
        skel[(size_t)t * MAXR + k] = x;
    }
    if (tid == 0) g.rank[t] = r;
    if (!LEAVES) {
        __syncthreads();
        if (tid == 0) dep_publish(dp, t);
    }
    // U = R12 times R11^-1 for the open rows (back substitution, one thread per row, four columns
    // at a time in registers: column i takes the later columns k in decreasing order, then its
    // division), the pivot rows rows of the identity
    for (int a = tid; a < m; a += THREADS) {
        float *u = C + a * CS;
        const int sp = selpos[a];
        if (sp >= 0) {
            for (int i = 0; i < r; i++) u[i] = i == sp ? 1.f : 0.f;
            continue;
        }
        for (int top = r - 1; top >= 0; top -= 4) {
            float acc[4];
#pragma unroll
            for (int z = 0; z < 4; z++) acc[z] = top - z >= 0 ? u[top - z] : 0.f;
            for (int k = r - 1; k > top; k--) {
                const float uk = u[k];
                const float *col = s.R11 + k * (k + 1) / 2 + top;
#pragma unroll
                for (int z = 0; z < 4; z++)
                    if (top - z >= 0) acc[z] = fmaf(-col[-z], uk, acc[z]);
            }
#pragma unroll
            for (int z = 0; z < 4; z++) {
                if (top - z < 0) break;
                const float *col = s.R11 + (top - z) * (top - z + 1) / 2;
                const float uk = acc[z] / col[top - z];
                u[top - z] = uk;
#pragma unroll
                for (int y = z + 1; y < 4; y++)
                    if (top - y >= 0) acc[y] = fmaf(-col[top - y], uk, acc[y]);
            }
        }
    }
    if (!LEAVES && tid < nch && !tv.leaf[cfirst + tid]) dep_wait_y0(dp, cfirst + tid);
    __syncthreads();
    for (int idx = tid; idx < m * r; idx += THREADS) {
        const int a = idx / r, k = idx - a * r;
        U[(size_t)a * MAXR + k] = C[a * CS + k];
    }
    // upward coefficients y0 = U^T (the leaf's [1 | x] | the children's y0): groups of RG
    // threads over k and YT / RG groups over the rows, summed in a fixed order
    {
        const int YT = min(THREADS, chains);
        float4 *part = reinterpret_cast<float4 *>(s.Q);
        const int RG = r <= 16 ? 16 : (r <= 32 ? 32 : 64);
        const int G = YT / RG, kk = tid % RG, cg = tid / RG;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kk < r && cg < G) {
            for (int a = cg; a < m; a += G) {
                const float w = C[a * CS + kk];
                if (LEAVES) {
                    const float4 x = xt[s0 + a];
                    acc.x += w;
                    acc.y = fmaf(w, x.x, acc.y);
                    acc.z = fmaf(w, x.y, acc.z);
                    acc.w = fmaf(w, x.z, acc.w);
                } else {
                    int c = 0;
                    while (a >= s.coff[c + 1]) c++;
                    fma4(acc, w, __ldcg(g.y0 + (size_t)(cfirst + c) * MAXR + (a - s.coff[c])));
                }
            }
        }
        part[tid] = acc;
        __syncthreads();
        if (tid < r) {
            float4 y = part[tid];
            for (int c = 1; c < G; c++) add4(y, part[c * RG + tid]);
            g.y0[(size_t)t * MAXR + tid] = y;
        }
    }
    if (!LEAVES) {
        __syncthreads();
        if (tid == 0) dep_publish_y0(dp, t);
    }
}

// ---------------------------------------------------------------------------------
// product kernels
// ---------------------------------------------------------------------------------
struct ProdArgs {
    TreeView tv;
    const void *xt;
    const void *skel;
    const int *rank;
    const long long *rowoff;
    const float *U;
    float4 *y0, *y1, *yp;
    const int *far_ptr, *far_idx, *near_ptr, *near_idx;
    const int *fine_cnt;
    const float4 *xin;   // input columns in tree order, or null for [1 | coordinates]
};

template <int D>
__device__ __forceinline__ float4 input_at(const ProdArgs &g, const typename Dim<D>::vec *xt, int j);

template <int D>
__device__ __forceinline__ float4 with_one(const Vec<D> &x)
{
    if constexpr (D == 2) return make_float4(1.f, x.x, x.y, 0.f);
    else return make_float4(1.f, x.x, x.y, x.z);
}
template <int D>
__device__ __forceinline__ float4 input_at(const ProdArgs &g, const typename Dim<D>::vec *xt, int j)
{
    return g.xin ? g.xin[j] : with_one<D>(xt[j]);
}

// upward pass, one warp per node of `level`: y0[t] = U_t^T (leaf points | children's y0)
template <int D>
__global__ void __launch_bounds__(256) k_up(int level, ProdArgs g)
{
    after_previous();
    constexpr int MAXR = Dim<D>::MAXR;
    const TreeView &tv = g.tv;
    const Vec<D> *xt = (const Vec<D> *)g.xt;
    const int lb = tv.info->level_begin[level], nl = tv.info->n_level_nodes[level];
    const int lane = threadIdx.x & 31;
    for (int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < nl; j += (gridDim.x * blockDim.x) >> 5) {
        const int t = lb + j;
        const int r = g.rank[t];
        const float *U = g.U + g.rowoff[t] * MAXR;
        float4 acc[MAXR / 32];
        for (int h = 0; h < MAXR / 32; h++) acc[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tv.leaf[t]) {
            const int m = tv.end[t] - tv.start[t];
            for (int a = 0; a < m; a++) {
                const float4 in = input_at<D>(g, xt, tv.start[t] + a);
                for (int h = 0; h < MAXR / 32; h++) {
                    const int k = lane + 32 * h;
                    if (k < r) fma4(acc[h], U[(size_t)a * MAXR + k], in);
                }
            }
        } else {
            int a = 0;
            for (int c = tv.fchild[t]; c < tv.fchild[t] + tv.nchild[t]; c++) {
                for (int kk = 0; kk < g.rank[c]; kk++, a++) {
                    const float4 in = g.y0[(size_t)c * MAXR + kk];
                    for (int h = 0; h < MAXR / 32; h++) {
                        const int k = lane + 32 * h;
                        if (k < r) fma4(acc[h], U[(size_t)a * MAXR + k], in);
                    }
                }
            }
        }
        for (int h = 0; h < MAXR / 32; h++) {
            const int k = lane + 32 * h;
            if (k < r) g.y0[(size_t)t * MAXR + k] = acc[h];
        }
    }
}

// The place of a node's slot k in skel, y0 and y1. In 64 bits: the node table is regrown while it is full, so
// no count of nodes is the last one that an int product would have to hold.
template <int D>
__host__ __device__ constexpr size_t slot_at(int node, int k) { return (size_t)node * Dim<D>::MAXR + k; }
static_assert(slot_at<2>(1 << 25, 1) == ((size_t)1 << 31) + 1 && slot_at<3>(1 << 25, 1) == ((size_t)1 << 31) + 1, "past an int");

// The sources of far entries [e0, e1) of a target at level lt, for one warp, in order. Sources of
// the target's level and (FINE) finer ones are skeletons with their coefficients; coarser ones
// (leaves) are points with the input columns; without FINE, finer sources are left out.
// The entries' node, size and kind are read 32 at a time by the lanes, the next 32 ahead. Their
// sources, each entry padded with zero coefficients to a multiple of S, are one sequence, which
// the lanes load 32 at a time, two rounds ahead, and hand to `body` in shared memory: body(x, y,
// count), which takes every S-th of them per lane group, sees the sources of an entry at places
// 0, S, 2 S, .. as if the entry stood alone. Read entry by entry, each one was a chain of four
// dependent loads before its first sum.
template <int D>
struct SrcBuf {
    float4 y[2][32];
    Vec<D> x[2][32];
};
template <int D>
struct SrcRegs {
    Vec<D> x;
    float4 y;
};

template <int D, bool FINE, typename Body>
__device__ __forceinline__ void for_sources(const ProdArgs &g, int e0, int e1, int lt, int S, int lane, SrcBuf<D> &buf,
                                            const Body &body)
{
    constexpr unsigned ALL = 0xffffffffu;
    // this lane's entry of a group of 32: its node (points: the first one), size, kind (0 skeleton, 1 points)
    auto entry = [&](int e, int &base, int &cnt, int &pts) {
        base = cnt = pts = 0;
        if (e + lane >= e1) return;
        const int s = g.far_idx[e + lane], ls = g.tv.level[s];
        if (ls >= lt) {
            base = s;
            cnt = (FINE || ls == lt) ? g.rank[s] : 0;
        } else {
            pts = 1;
            base = g.tv.start[s];
            cnt = g.tv.end[s] - base;
        }
    };
    int base, cnt, pts;
    entry(e0, base, cnt, pts);
    for (int e = e0; e < e1; e += 32) {
        int nbase, ncnt, npts;
        entry(e + 32, nbase, ncnt, npts);
        int first = (cnt + S - 1) & ~(S - 1);   // the entry's place in the sequence
        const int own = first;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(ALL, first, o);
            if (lane >= o) first += v;
        }
        const int total = __shfl_sync(ALL, first, 31);
        first -= own;
        auto load = [&](int round, SrcRegs<D> &r) {
            const int j = round * 32 + lane;
            int i = 0;   // the last entry that starts at or before j
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int v = __shfl_sync(ALL, first, i + o);
                if (v <= j) i += o;
            }
            const int b = j - __shfl_sync(ALL, first, i), c = __shfl_sync(ALL, cnt, i);
            const int from = __shfl_sync(ALL, base, i), p = __shfl_sync(ALL, pts, i);
            const size_t at = p ? (size_t)from + b : slot_at<D>(from, b);
            r.y = make_float4(0.f, 0.f, 0.f, 0.f);
            if constexpr (D == 2) r.x = make_float2(0.f, 0.f);
            else r.x = r.y;
            if (j < total && b < c) {
                r.x = p ? ((const Vec<D> *)g.xt)[at] : ((const Vec<D> *)g.skel)[at];
                r.y = !p ? g.y0[at] : (g.xin ? g.xin[at] : with_one<D>(r.x));
            }
        };
        SrcRegs<D> ra, rb;
        load(0, ra);
        load(1, rb);
        for (int round = 0; round * 32 < total; round += 2) {
            buf.x[0][lane] = ra.x;
            buf.y[0][lane] = ra.y;
            __syncwarp();
            load(round + 2, ra);
            body(buf.x[0], buf.y[0], min(32, total - round * 32));
            if ((round + 1) * 32 < total) {
                buf.x[1][lane] = rb.x;
                buf.y[1][lane] = rb.y;
                __syncwarp();
                load(round + 3, rb);
                body(buf.x[1], buf.y[1], min(32, total - (round + 1) * 32));
            }
        }
        __syncwarp();
        base = nbase; cnt = ncnt; pts = npts;
    }
}

// far field onto compressed targets at level >= 2:
//   same-level partner  : y1[t] += K(J_t, J_s) y0[s]
//   coarser leaf partner: y1[t] += K(J_t, X_s) [1 | x_s]
// A warp per target; of a target of rank above 32 (3D), a warp per 32 of its skeleton slots. A
// target of rank r <= 32 gives each slot a group of lanes (rp = r rounded up to a power of two
// slots) and the warp's 32 / rp groups split the sources; the group sums meet by shuffles in a
// fixed order. What bounds it is the longest target's sequence of sources (3D: about 9,000 near
// the root), so these are staged ahead (for_sources) and four are in the arithmetic at a time.
// Measured at 20K / 1M points in 2D and 100K in 3D: 22 / 165 / 453 us; read entry by entry,
// 63 / 160 / 1,021 us.
constexpr int FAR_WARPS = 4;
constexpr int far_halves(int d) { return (d == 2 ? MAX_RANK_2D : MAX_RANK_3D) / 32; }

template <int D>
__global__ void __launch_bounds__(32 * FAR_WARPS) k_far_c(int first, int n_node, ProdArgs g)
{
    after_previous();
    constexpr int MAXR = Dim<D>::MAXR, HALVES = far_halves(D);
    __shared__ SrcBuf<D> bufs[FAR_WARPS];
    const TreeView &tv = g.tv;
    const Vec<D> *skel = (const Vec<D> *)g.skel;
    const int lane = threadIdx.x & 31;
    SrcBuf<D> &buf = bufs[threadIdx.x >> 5];
    if (blockIdx.x == 0 && threadIdx.x == 0) tv.tickets[TICKET_DOWN] = 0;   // for the downward pass
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < HALVES * (n_node - first);
         w += (gridDim.x * blockDim.x) >> 5) {
        const int t = first + w / HALVES, k0 = 32 * (w % HALVES);
        const int r = g.rank[t];
        if (k0 > 0 && k0 >= r) continue;
        int rp = 1;
        while (rp < r && rp < 32) rp <<= 1;
        const int S = 32 / rp, k = k0 + lane % rp, sub = lane / rp;
        const Vec<D> J = skel[(size_t)t * MAXR + (k < r ? k : 0)];
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        const int e0 = g.far_ptr[t], e1 = g.far_ptr[t + 1], lt = tv.level[t];
        if (S == 1)   // rank above 16: whole rounds without a stride to carry
            for_sources<D, false>(g, e0, e1, lt, 1, lane, buf, [&](const Vec<D> *x, const float4 *y, int cnt) {
                if (cnt == 32) {
#pragma unroll 8
                    for (int b = 0; b < 32; b++) fma4(acc, rkernel(dist2(J, x[b])), y[b]);
                } else {
#pragma unroll 4
                    for (int b = 0; b < cnt; b++) fma4(acc, rkernel(dist2(J, x[b])), y[b]);
                }
            });
        else
            for_sources<D, false>(g, e0, e1, lt, S, lane, buf, [&](const Vec<D> *x, const float4 *y, int cnt) {
#pragma unroll 4
                for (int b = sub; b < cnt; b += S) fma4(acc, rkernel(dist2(J, x[b])), y[b]);
            });
        for (int o = rp; o < 32; o <<= 1) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
            acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
            acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
        }
        if (sub == 0 && k < r) g.y1[(size_t)t * MAXR + k] = acc;
    }
}

// near field onto a leaf's points (one CTA per leaf, sources tiled through shared memory):
//   near partner           : yp[i] += sum_{j != i} K(x_i, x_j) [1 | x_j]
//   finer far partner (s)  : yp[i] += K(x_i, J_s) y0[s]
// NC = number of accumulated columns (3 in 2D for [1 | x y], 4 in 3D or for general inputs);
// only the leaf's own tiles test for the diagonal.
template <int NC>
__device__ __forceinline__ void acc_cols(float4 &acc, float w, const float4 &v)
{
    acc.x = fmaf(w, v.x, acc.x);
    acc.y = fmaf(w, v.y, acc.y);
    acc.z = fmaf(w, v.z, acc.z);
    if (NC == 4) acc.w = fmaf(w, v.w, acc.w);
}

// Parts of the leaf targets' sums: NEAR_ALL = the near blocks and the far entries whose source
// is finer than the leaf (through the source's skeleton and upward coefficients), assigned;
// NEAR_BLOCKS = the near blocks alone (tree, points and lists only: no basis), assigned. The
// finer far entries alone are k_fine's.
constexpr int NEAR_ALL = 0, NEAR_BLOCKS = 1;

template <int D, int NC, int PART = NEAR_ALL>
__global__ void __launch_bounds__(NEAR_THREADS) k_near(ProdArgs g)
{
    after_previous();
    constexpr int MAXR = Dim<D>::MAXR;
    const TreeView &tv = g.tv;
    const int t = blockIdx.x;
    if (!tv.leaf[t]) return;
    const Vec<D> *xt = (const Vec<D> *)g.xt;
    const Vec<D> *skel = (const Vec<D> *)g.skel;
    __shared__ Vec<D> sx[NEAR_THREADS];
    __shared__ float4 sxin[NEAR_THREADS];
    __shared__ float4 sy[MAXR];
    const int s0 = tv.start[t], cnt = tv.end[t] - s0, lt = tv.level[t];
    for (int chunk = 0; chunk < cnt; chunk += NEAR_THREADS) {
        const int i = s0 + chunk + threadIdx.x;
        const bool valid = chunk + (int)threadIdx.x < cnt;
        const Vec<D> xi = xt[valid ? i : s0];
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int e = g.near_ptr[t]; e < g.near_ptr[t + 1]; e++) {
            const int s = g.near_idx[e];
            const int ss = tv.start[s], sc = tv.end[s] - ss;
            for (int tile = 0; tile < sc; tile += NEAR_THREADS) {
                __syncthreads();
                if ((int)threadIdx.x < sc - tile) {
                    sx[threadIdx.x] = xt[ss + tile + threadIdx.x];
                    sxin[threadIdx.x] = input_at<D>(g, xt, ss + tile + threadIdx.x);
                }
                __syncthreads();
                const int lim = min(NEAR_THREADS, sc - tile);
                if (s == t) {
                    const int self = i - (ss + tile);
                    for (int j = 0; j < lim; j++) {
                        float w = rkernel(dist2(xi, sx[j]));
                        w = (j == self) ? 0.f : w;
                        acc_cols<NC>(acc, w, sxin[j]);
                    }
                } else {
#pragma unroll 4
                    for (int j = 0; j < lim; j++) acc_cols<NC>(acc, rkernel(dist2(xi, sx[j])), sxin[j]);
                }
            }
        }
        for (int e = g.far_ptr[t]; PART != NEAR_BLOCKS && e < g.far_ptr[t + 1]; e++) {
            const int s = g.far_idx[e];
            if (tv.level[s] <= lt) continue;
            const int rs = g.rank[s];
            __syncthreads();
            for (int b = threadIdx.x; b < rs; b += NEAR_THREADS) {
                sx[b] = skel[(size_t)s * MAXR + b];
                sy[b] = g.y0[(size_t)s * MAXR + b];
            }
            __syncthreads();
            for (int b = 0; b < rs; b++) acc_cols<NC>(acc, rkernel(dist2(xi, sx[b])), sy[b]);
        }
        if (valid) g.yp[i] = acc;
    }
}

// Near field of the 2D force product ([1 | x y] columns), two targets per thread with the
// paired FP32 instructions: thread `tid` owns the leaf's points tid and tid + NEAR2_THREADS of
// each chunk of 2 * NEAR2_THREADS. Sources are staged with each coordinate duplicated
// ((x, x), (y, y)), so one shared-memory load feeds both targets; per source and target pair
// the kernel issues 5 arithmetic instructions and 2 reciprocals instead of 10 and 2.
// Same sums, same order of sources, as k_near.
constexpr int NEAR2_THREADS = 64;
constexpr int NEAR2_TILE = 2 * NEAR2_THREADS;

template <int PART = NEAR_ALL>
__global__ void __launch_bounds__(NEAR2_THREADS) k_near2d(ProdArgs g)
{
    after_previous();
    constexpr int MAXR = Dim<2>::MAXR;
    const TreeView &tv = g.tv;
    const int t = blockIdx.x;
    if (!tv.leaf[t]) return;
    const float2 *xt = (const float2 *)g.xt;
    const float2 *skel = (const float2 *)g.skel;
    __shared__ float4 sxy[NEAR2_TILE];      // (x, x, y, y)
    __shared__ float4 sw01[MAXR];           // (w0, w0, w1, w1) of a skeleton source
    __shared__ float2 sw2[MAXR];            // (w2, w2)
    const int tid = threadIdx.x;
    const int s0 = tv.start[t], cnt = tv.end[t] - s0, lt = tv.level[t];
    for (int chunk = 0; chunk < cnt; chunk += NEAR2_TILE) {
        const int a0 = chunk + tid, a1 = a0 + NEAR2_THREADS;
        const float2 x0 = xt[s0 + (a0 < cnt ? a0 : 0)], x1 = xt[s0 + (a1 < cnt ? a1 : 0)];
        const F2 ax = f2_pack(x0.x, x1.x), ay = f2_pack(x0.y, x1.y);
        F2 acc0 = f2_pack(0.f, 0.f), accx = acc0, accy = acc0;
        for (int e = g.near_ptr[t]; e < g.near_ptr[t + 1]; e++) {
            const int s = g.near_idx[e];
            const int ss = tv.start[s], sc = tv.end[s] - ss;
            for (int tile = 0; tile < sc; tile += NEAR2_TILE) {
                __syncthreads();
                for (int b = tid; b < NEAR2_TILE && b < sc - tile; b += NEAR2_THREADS) {
                    const float2 p = xt[ss + tile + b];
                    sxy[b] = make_float4(p.x, p.x, p.y, p.y);
                }
                __syncthreads();
                const int lim = min(NEAR2_TILE, sc - tile);
                if (s == t) {
                    const int self0 = a0 - tile, self1 = a1 - tile;
                    for (int j = 0; j < lim; j++) {
                        const float4 q = sxy[j];
                        const F2 sx = f2_pack(q.x, q.y), sy = f2_pack(q.z, q.w);
                        F2 w = f2_rkernel(ax, ay, sx, sy);
                        float w0, w1;
                        f2_unpack(w, w0, w1);
                        w = f2_pack(j == self0 ? 0.f : w0, j == self1 ? 0.f : w1);
                        acc0 = f2_add(acc0, w);
                        accx = f2_fma(w, sx, accx);
                        accy = f2_fma(w, sy, accy);
                    }
                } else {
#pragma unroll 4
                    for (int j = 0; j < lim; j++) {
                        const float4 q = sxy[j];
                        const F2 sx = f2_pack(q.x, q.y), sy = f2_pack(q.z, q.w);
                        const F2 w = f2_rkernel(ax, ay, sx, sy);
                        acc0 = f2_add(acc0, w);
                        accx = f2_fma(w, sx, accx);
                        accy = f2_fma(w, sy, accy);
                    }
                }
            }
        }
        for (int e = g.far_ptr[t]; PART != NEAR_BLOCKS && e < g.far_ptr[t + 1]; e++) {
            const int s = g.far_idx[e];
            if (tv.level[s] <= lt) continue;
            const int rs = g.rank[s];
            __syncthreads();
            for (int b = tid; b < rs; b += NEAR2_THREADS) {
                const float2 p = skel[(size_t)s * MAXR + b];
                const float4 y = g.y0[(size_t)s * MAXR + b];
                sxy[b] = make_float4(p.x, p.x, p.y, p.y);
                sw01[b] = make_float4(y.x, y.x, y.y, y.y);
                sw2[b] = make_float2(y.z, y.z);
            }
            __syncthreads();
            for (int b = 0; b < rs; b++) {
                const float4 q = sxy[b];
                const float4 y01 = sw01[b];
                const float2 y2 = sw2[b];
                const F2 w = f2_rkernel(ax, ay, f2_pack(q.x, q.y), f2_pack(q.z, q.w));
                acc0 = f2_fma(w, f2_pack(y01.x, y01.y), acc0);
                accx = f2_fma(w, f2_pack(y01.z, y01.w), accx);
                accy = f2_fma(w, f2_pack(y2.x, y2.y), accy);
            }
        }
        float c00, c01, cx0, cx1, cy0, cy1;
        f2_unpack(acc0, c00, c01);
        f2_unpack(accx, cx0, cx1);
        f2_unpack(accy, cy0, cy1);
        if (a0 < cnt) g.yp[s0 + a0] = make_float4(c00, cx0, cy0, 0.f);
        if (a1 < cnt) g.yp[s0 + a1] = make_float4(c01, cx1, cy1, 0.f);
    }
}

// The finer far entries of the leaves that have any (flist), added to their points' sums: a CTA
// per leaf, a warp per 32 of its points, the sources' skeletons and coefficients staged ahead
// (for_sources). A leaf's far list is ascending and nodes are numbered level by level, so the
// finer sources are its last fine_cnt entries. Same sums, in the same order and with the same
// operations, as k_near2d and k_near. At 20K / 1M points in 2D and 100K in 3D: 18 / 27 / 144 us, on
// the side stream; a block per node, every thread of which walked the far list to find the finer
// entries, took 44 / 87 / 234 us before the downward pass.
template <int D>
__global__ void __launch_bounds__(32 * FAR_WARPS) k_fine(const int *items, ProdArgs g)
{
    after_previous();
    __shared__ SrcBuf<D> bufs[FAR_WARPS];
    const TreeView &tv = g.tv;
    const Vec<D> *xt = (const Vec<D> *)g.xt;
    const int lane = threadIdx.x & 31;
    SrcBuf<D> &buf = bufs[threadIdx.x >> 5];
    const int t = items[blockIdx.x];
    const int s0 = tv.start[t], cnt = tv.end[t] - s0, e1 = g.far_ptr[t + 1], e0 = e1 - g.fine_cnt[t], lt = tv.level[t];
    for (int chunk = threadIdx.x & ~31; chunk < cnt; chunk += 32 * FAR_WARPS) {
        const bool valid = chunk + lane < cnt;
        const int i = s0 + (valid ? chunk + lane : 0);
        const Vec<D> xi = xt[i];
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        auto add = [&](const Vec<D> &sx, const float4 &v) {
            if constexpr (D == 2) {
                const float dx = xi.x - sx.x, dy = xi.y - sx.y;
                float w = fast_rcp(fmaf(dx, dx, fmaf(dy, dy, 1.f)));
                w *= w;
                acc.x = fmaf(w, v.x, acc.x);
                acc.y = fmaf(w, v.y, acc.y);
                acc.z = fmaf(w, v.z, acc.z);
            } else {
                fma4(acc, rkernel(dist2(xi, sx)), v);
            }
        };
        for_sources<D, true>(g, e0, e1, lt, 1, lane, buf, [&](const Vec<D> *x, const float4 *y, int c) {
            if (c == 32) {
#pragma unroll 8
                for (int b = 0; b < 32; b++) add(x[b], y[b]);
            } else {
#pragma unroll 4
                for (int b = 0; b < c; b++) add(x[b], y[b]);
            }
        });
        if (valid) {
            add4(acc, g.yp[i]);
            g.yp[i] = acc;
        }
    }
}

// downward pass of node t (one warp): the node's y1 through U onto its leaf points (yp) or
// its children's y1. y1 is staged in the warp's slice of shared memory (sy, MAXR entries); lane
// a takes candidate row a and reads its U row four entries at a time. FRESH: y1 is read
// through L2 (written in the same launch).
template <int D, bool FRESH>
__device__ __forceinline__ void down_node(const ProdArgs &g, int t, int lane, float4 *sy)
{
    constexpr int MAXR = Dim<D>::MAXR;
    const TreeView &tv = g.tv;
    const int r = g.rank[t];
    const float *U = g.U + g.rowoff[t] * MAXR;
    for (int k = lane; k < r; k += 32) {
        const float4 *src = g.y1 + (size_t)t * MAXR + k;
        sy[k] = FRESH ? __ldcg(src) : *src;
    }
    __syncwarp();
    const bool isleaf = tv.leaf[t] != 0;
    int m = 0;
    if (isleaf) m = tv.end[t] - tv.start[t];
    else for (int c = tv.fchild[t]; c < tv.fchild[t] + tv.nchild[t]; c++) m += g.rank[c];
    const int r4 = r & ~3;
    for (int a0 = 0; a0 < m; a0 += 32) {
        const int a = a0 + lane;
        if (a >= m) break;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        const float *u = U + (size_t)a * MAXR;
        for (int k = 0; k < r4; k += 4) {
            const float4 w = *reinterpret_cast<const float4 *>(u + k);
            fma4(acc, w.x, sy[k]);
            fma4(acc, w.y, sy[k + 1]);
            fma4(acc, w.z, sy[k + 2]);
            fma4(acc, w.w, sy[k + 3]);
        }
        for (int k = r4; k < r; k++) fma4(acc, u[k], sy[k]);
        if (isleaf) {
            float4 o = g.yp[tv.start[t] + a];
            add4(o, acc);
            g.yp[tv.start[t] + a] = o;
        } else {
            int c = tv.fchild[t], aa = a;
            while (aa >= g.rank[c]) { aa -= g.rank[c]; c++; }
            float4 *dst = g.y1 + (size_t)c * MAXR + aa;
            float4 o = FRESH ? __ldcg(dst) : *dst;
            add4(o, acc);
            *dst = o;
        }
    }
    __syncwarp();
}

// downward pass of every internal node at level >= 2 in one dependency-ordered launch
// (persistent warps, items in increasing node id): a node waits for its parent's push
template <int D>
__global__ void __launch_bounds__(256) k_down_internal(int n_item, const int *items, ProdArgs g,
                                                        DepArgs dp)
{
    after_previous();
    __shared__ float4 sy[256 / 32][Dim<D>::MAXR];
    const int lane = threadIdx.x & 31;
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(dp.ticket, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= n_item) break;
        const int t = items[item];
        const int p = g.tv.parent[t];
        if (lane == 0 && g.tv.level[p] >= MIN_ADM_LEVEL) dep_wait(dp, p);
        __syncwarp();
        down_node<D, true>(g, t, lane, sy[threadIdx.x >> 5]);
        __syncwarp();
        if (lane == 0) dep_publish(dp, t);
    }
}

// downward pass of every leaf at level >= 2 (after the internal nodes)
template <int D>
__global__ void __launch_bounds__(256) k_down_leaves(ProdArgs g)
{
    after_previous();
    __shared__ float4 sy[256 / 32][Dim<D>::MAXR];
    const TreeView &tv = g.tv;
    const int lb = tv.info->level_begin[MIN_ADM_LEVEL];
    const int nl = tv.info->n_node - lb;
    const int lane = threadIdx.x & 31;
    for (int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < nl; j += (gridDim.x * blockDim.x) >> 5) {
        const int t = lb + j;
        if (tv.leaf[t]) down_node<D, false>(g, t, lane, sy[threadIdx.x >> 5]);
    }
}

inline int grid_for(long long work, int block, int cap = 148 * 16)
{
    long long g = (work + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
template <int D>
class H2Impl final : public H2Matrix {
public:
    ~H2Impl() override
    {
        if (counts_ev_) cudaEventDestroy(counts_ev_);
        if (st2_) {
            cudaStreamSynchronize(st2_);
            cudaStreamDestroy(st2_);
        }
        if (fork_ev_) cudaEventDestroy(fork_ev_);
        if (near_ev_) cudaEventDestroy(near_ev_);
        if (lists_ev_) cudaEventDestroy(lists_ev_);
    }

    H2Impl(int n, cudaStream_t st) : n_(n), st_(st)
    {
        TSNE_CUDA_CHECK(cudaStreamCreateWithFlags(&st2_, cudaStreamNonBlocking));
        TSNE_CUDA_CHECK(cudaEventCreateWithFlags(&fork_ev_, cudaEventDisableTiming));
        TSNE_CUDA_CHECK(cudaEventCreateWithFlags(&near_ev_, cudaEventDisableTiming));
        TSNE_CUDA_CHECK(cudaEventCreateWithFlags(&lists_ev_, cudaEventDisableTiming));
        keys_in_.exact(n); keys_.exact(n); idx_in_.exact(n); perm_.exact(n); xt_.exact(n);
        yp_.exact(n);
        bbox_part_.exact((size_t)BBOX_BLOCKS * (2 * D + 1));
        fm_.exact(n);
        blkcnt_.exact((size_t)ceil_div(n, TREE_BLOCK) * 64);
        blkoff_.exact((size_t)ceil_div(n, TREE_BLOCK) * 64);
        btot_.exact(64);
        proxies_.exact((size_t)(Dim<D>::L + 1) * PROXY_F4);
        tickets_.exact(N_TICKET);
        done_.exact(1);
        TSNE_CUDA_CHECK(cudaMemsetAsync(tickets_.p, 0, sizeof(int) * N_TICKET, st_));
        TSNE_CUDA_CHECK(cudaMemsetAsync(done_.p, 0, sizeof(int), st_));
        info_.exact(1);
        TSNE_CUDA_CHECK(cudaMemsetAsync(info_.p, 0, sizeof(TreeInfo), st_));
        TSNE_CUDA_CHECK(cudaEventCreateWithFlags(&counts_ev_, cudaEventDisableTiming));
        size_t b1 = 0;
        TSNE_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(nullptr, b1, keys_in_.p, keys_.p, idx_in_.p,
                                                        perm_.p, n, 0, D * Dim<D>::L, st_));
        sort_bytes_ = b1;
        cub_tmp_.exact(b1 + 256);
        cap_node_ = first_cap_node(n);
        nset_cap_ = Dim<D>::NSET;
        alloc_nodes();
        TSNE_CUDA_CHECK(cudaFuncSetAttribute(k_id<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)id_smem_bytes<D>(id_mcap())));
        TSNE_CUDA_CHECK(cudaFuncSetAttribute(k_id<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)id_smem_bytes<D>(id_mcap())));
        if (D == 2) {
            id2_attr<true, 64, 1>();
            id2_attr<true, 128, 1>();
            id2_attr<true, 128, 2>();
            id2_attr<false, 128, 2>();
        }
        if (D == 3) {
            TSNE_CUDA_CHECK(cudaFuncSetAttribute(k_near<D, 4, NEAR_BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)NEAR_MOST));
            id3_attr<false, 512, ID3_ROWS>();
            id3_attr<true, 512, ID3_ROWS>();
            id3_attr<true, 512, ID3_MID>();
            id3_attr<true, 256, ID3_SMALL>();
            id3_attr<true, 128, ID3_TINY>();
        }
    }

    static int id_mcap()
    {
        // shared-memory rows of the ID: every internal node of the 2D tree (4 * MAXR rows)
        // and leaves up to that size; the 3D bound keeps the CTA under 227 KB
        return D == 2 ? (1 << D) * Dim<D>::MAXR : 240;
    }
    static int first_cap_node(int n) { return std::max(1024, 4 * (n / 16) + 1024); }   // regrown while it is full

    int build(const void *Y, int leaf_size, double tol, const std::function<void()> *overlap) override
    {
        join_near();   // the side stream's near field reads the tree this build rewrites
        leaf_size_ = leaf_size;
        const int L = Dim<D>::L;
        cudaEvent_t t_tree = mark_begin();
        sec_begin();
        // One batch: root box, keys, sort, the whole tree (four kernels over the points, no level
        // loop) and the counting pass of the interaction lists (kernels read the level and node
        // counts on the device), then one copy to pinned memory and one wait bring the tree, the
        // list totals and the basis rows (TreeInfo): copies to pageable members held the host,
        // and with it the work queued to overlap the wait, for about 50 us per rebuild. A full node table or a full inadmissible-source set are caught there and redone.
        bool tree_ok = false;
        for (int attempt = 0; attempt < 12; attempt++) {
            if (!tree_ok) {
                const int nblk = ceil_div(n_, TREE_BLOCK);
                launch_early(k_bbox<D>, BBOX_BLOCKS, 256, 0, st_, n_, (const Vec<D> *)Y, bbox_part_.p, view(),
                    done_.p);
                if (n_ <= SORT_MOST) {
                    const int tiles = ceil_div(n_, SORT_TILE);
                    const bool one = tiles == 1;
                    launch_early(k_tile_sort<D>, tiles, SORT_THREADS, 0, st_, n_, L, (const Vec<D> *)Y, info_.p,
                        one ? keys_.p : keys_in_.p, one ? perm_.p : idx_in_.p);
                    if (!one)
                        launch_early(k_tile_rank, ceil_div(n_, 256), 256, 0, st_, n_, keys_in_.p, idx_in_.p,
                            keys_.p, perm_.p);
                    launches_ += 2;
                } else {
                    launch_early(k_keys<D>, grid_for(n_, 256), 256, 0, st_, n_, L, (const Vec<D> *)Y, info_.p,
                        keys_in_.p, idx_in_.p);
                    size_t bytes = sort_bytes_;
                    TSNE_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(cub_tmp_.p, bytes, keys_in_.p, keys_.p, idx_in_.p,
                                                                    perm_.p, n_, 0, D * L, st_));
                    launches_ += 1 + 4;
                }
                launch_early(k_tree_marks<D>, nblk, TREE_BLOCK, 0, st_, view(), perm_.p, (const Vec<D> *)Y, xt_.p);
                launch_early(k_tree_scan, 64, TREE_SCAN_THREADS, 0, st_, nblk, view());
                launch_early(k_tree_emit<D>, nblk, TREE_BLOCK, 0, st_, view());
                launch_early(k_tree_finish<D>, grid_for(cap_node_, 256, 148 * 8), 256, 0, st_, view());
                launches_ += 5;
                tree_ok = true;
            }
            launch_list_counts();
            TSNE_CUDA_CHECK(cudaMemcpyAsync(hinfo_.p, info_.p, sizeof(TreeInfo), cudaMemcpyDeviceToHost, st_));
            TSNE_CUDA_CHECK(cudaEventRecord(counts_ev_, st_));
            if (overlap != nullptr && *overlap) {
                (*overlap)();
                overlap = nullptr;
            }
            TSNE_CUDA_CHECK(cudaEventSynchronize(counts_ev_));
            const TreeInfo &I = *hinfo_.p;
            if (I.nonfinite) return -1;
            if (I.pad[1]) {   // a dependency wait of an earlier launch gave up
                fprintf(stderr, "tsne_h2pack: an H2 kernel gave up waiting for a tree dependency\n");
                return -2;
            }
            if (I.pad[0]) {   // node table full: grow and start over
                cap_node_ *= 2;
                alloc_nodes();
                tree_ok = false;
                continue;
            }
            if (I.nset_overflow) {   // inadmissible-source set full: grow, recount
                nset_cap_ *= 2;
                alloc_lists();
                if (attempt < 11) {   // the counters that the root kernel cleared for the first count
                    TSNE_CUDA_CHECK(cudaMemsetAsync(&info_.p->nset_overflow, 0, sizeof(int), st_));
                    TSNE_CUDA_CHECK(cudaMemsetAsync(&info_.p->pad[2], 0, sizeof(int), st_));
                    TSNE_CUDA_CHECK(cudaMemsetAsync(&tickets_.p[TICKET_LISTS], 0, sizeof(int), st_));
                    continue;
                }
            }
            break;
        }
        mark_end(t_tree, 0);
        sec_end("tree+counts");
        const TreeInfo &I = *hinfo_.p;
        n_node_ = I.n_node;
        max_level_ = I.max_level;
        last_max_level_ = max_level_;
        stats_.n_node = n_node_;
        stats_.max_level = max_level_;
        stats_.max_leaf = I.max_leaf;
        hrows_ = I.n_rows;
        hint_ = I.n_int;
        hleaf_ = I.n_small;
        hbig_ = I.n_big;
        hlarge_ = I.n_large;
        hfine_ = I.n_fine;
        if (max_level_ <= 2) { built_ = false; return 1; }

        // The list write needs only the count pass, and the bases read no list, so it runs on the side stream beside the leaf
        // bases; the near blocks follow it there. Its buffers are allocated first, in the
        // workspace stream's order (the stream-ordered pool), and the side stream starts from
        // that point. Readers on the workspace stream join it first (join_lists).
        stats_.n_far = htot_[0] = I.n_far;
        stats_.n_near = htot_[1] = I.n_near;
        far_idx_.ensure(std::max(1, htot_[0]));
        near_idx_.ensure(std::max(1, htot_[1]));
        const bool slot_over = I.pad[2] != 0;   // a target with more entries than slots
        if (D == 3 && slot_over) {
            sort_reserve(far_idx_, far_alt_, htot_[0], far_ptr_.p);
            sort_reserve(near_idx_, near_alt_, htot_[1], near_ptr_.p);
        }
        {
            TSNE_CUDA_CHECK(cudaEventRecord(fork_ev_, st_));
            TSNE_CUDA_CHECK(cudaStreamWaitEvent(st2_, fork_ev_, 0));
            cudaEvent_t t_lists = mark_begin(st2_);
            if (!slot_over) {
                launch_early(k_lists_compact<D>, grid_for((long long)n_node_ * 32, 256, 148 * 8), 256, 0, st2_,
                    view(), list_out());
            } else {
                launch_early(k_lists_write<D>, grid_for(n_node_, 128, 148 * 8), 128, 0, st2_, n_node_, view(),
                    list_out());
                if (D == 3) {
                    sort_segments(far_idx_, far_alt_, htot_[0], far_ptr_.p, st2_);
                    sort_segments(near_idx_, near_alt_, htot_[1], near_ptr_.p, st2_);
                }
            }
            launches_++;
            mark_end(t_lists, 1, st2_);
            TSNE_CUDA_CHECK(cudaEventRecord(lists_ev_, st2_));
            lists_pending_ = true;
        }

        // bases, bottom-up
        cudaEvent_t t_bases = mark_begin();
        constexpr int MAXR = Dim<D>::MAXR, P = Dim<D>::NPROXY;
        skel_.ensure((size_t)n_node_ * MAXR);
        y0_.ensure((size_t)n_node_ * MAXR);
        y1_.ensure((size_t)n_node_ * MAXR);
        U_.ensure((size_t)std::max<long long>(hrows_, 1) * MAXR);
        const int mcap = id_mcap();
        const bool id3_path = D == 3 && id3_;   // no stored matrix, except for leaves above ID3_ROWS
        const bool need_glob = id3_path ? stats_.max_leaf > ID3_ROWS : stats_.max_leaf > mcap || (1 << D) * MAXR > mcap;
        if (need_glob) {
            gA_.ensure((size_t)std::max<long long>(hrows_, 1) * (P + 1));
            gnrm_.ensure(std::max<long long>(hrows_, 1));
            gsel_.ensure(std::max<long long>(hrows_, 1));
            gcand_.ensure(std::max<long long>(hrows_, 1));
        }
        const float tol2 = (float)((tol * ID_TOL_FACTOR) * (tol * ID_TOL_FACTOR));
        // leaves: one launch, shared memory sized for the largest leaf
        const int mleaf = std::max(1, std::min(stats_.max_leaf, mcap));
        IdArgs il{view(), xt_.p, skel_.p, rank_.p, rowoff_.p, U_.p, gA_.p, gnrm_.p, gsel_.p, gcand_.p, mleaf, tol2,
                  y0_.p};
        const int first = I.level_begin[MIN_ADM_LEVEL];
        if (D == 2 && stats_.max_leaf <= ID2_HELD) {
            // leaves in one launch, then the internal nodes of every level in one
            // dependency-ordered launch
            DepArgs dp{flag_.p, tickets_.p + TICKET_BASES, &info_.p->pad[1], ++epoch_};
            // few leaves: one launch of the CTAs that take any size, so that all run at once;
            // more than fill the GPU: by size, so that small leaves do not take large CTAs
            const int *none = nullptr;
            if (hleaf_ + hbig_ + hlarge_ <= ID2_ONE_LAUNCH) {
                const LeafItems all{{clist_.p, blist_.p, llist_.p}, {hlarge_, hbig_, hleaf_}};
                if (hleaf_ + hbig_ + hlarge_ > 0) id2_launch<true, 128, 2>(hleaf_ + hbig_ + hlarge_, none, all, il, dp);
            } else {
                if (hlarge_ > 0) id2_launch<true, 128, 2>(hlarge_, none, {{clist_.p, none, none}, {hlarge_, 0, 0}}, il, dp);
                if (hbig_ > 0) id2_launch<true, 128, 1>(hbig_, none, {{blist_.p, none, none}, {hbig_, 0, 0}}, il, dp);
                if (hleaf_ > 0) id2_launch<true, 64, 1>(hleaf_, none, {{llist_.p, none, none}, {hleaf_, 0, 0}}, il, dp);
            }
            mark_end(t_bases, 2);
            t_bases = mark_begin();
            near_fork_point();
            if (hint_ > 0 && id_by_level_) {
                // one launch per level, deepest first (TSNE_ID_BYLEVEL=1)
                for (int l = max_level_; l >= MIN_ADM_LEVEL; l--) {
                    const int nl = I.n_level_nodes[l];
                    if (nl <= 0) continue;
                    id2_launch<false, 128, 2>(I.level_begin[l], nullptr, LeafItems{}, il, dp, nl);
                }
            } else if (hint_ > 0) {
                DepArgs d2 = dp;
                d2.flag2 = flag2_.p;
                id2_launch<false, 128, 2>(hint_, ilist_.p, LeafItems{}, il, d2);
            }
            near_launch_side();
            mark_end(t_bases, 7);
            if (timing_) TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
            sec_end("lists+bases");
            built_ = true;
            y0_from_build_ = true;
            rank_stats_valid_ = false;
            return 0;
        }
        DepArgs dp{flag_.p, tickets_.p + TICKET_BASES, &info_.p->pad[1], ++epoch_};
        if (D == 3 && id3_) {
            // leaves by size (llist: at most ID3_TINY points; blist: at most ID3_SMALL; clist: the
            // others, up to ID3_ROWS; larger leaves, only at the depth limit, take k_id), then
            // the internal nodes in one dependency-ordered launch
            if (stats_.max_leaf <= ID3_ROWS) {
                if (hlarge_ > 0) {
                    id3_launch<true, 512, ID3_MID>(hlarge_, clist_.p, ID3_SMALL, 256, il, dp);
                    if (stats_.max_leaf > ID3_MID) id3_launch<true, 512, ID3_ROWS>(hlarge_, clist_.p, ID3_MID, 512, il, dp);
                }
                if (hbig_ > 0) id3_launch<true, 256, ID3_SMALL>(hbig_, blist_.p, ID3_TINY, 256, il, dp);
                if (hleaf_ > 0) id3_launch<true, 128, ID3_TINY>(hleaf_, llist_.p, 0, 128, il, dp);
            } else {
                launch_early(k_id<D, true>, n_node_ - first, IDG_THREADS, id_smem_bytes<D>(mleaf), st_,
                    MIN_ADM_LEVEL, il, 0, nullptr, dp);
                launches_++;
            }
            mark_end(t_bases, 2);
            t_bases = mark_begin();
            near_fork_point();
            if (hint_ > 0) {
                DepArgs d2 = dp;
                d2.flag2 = flag2_.p;
                id3_launch<false, 512, ID3_ROWS>(hint_, ilist_.p, 0, 512, il, d2);
            }
            near_launch_side();
            mark_end(t_bases, 7);
            if (timing_) TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
            sec_end("lists+bases");
            built_ = true;
            y0_from_build_ = true;
            rank_stats_valid_ = false;
            return 0;
        }
        launch_early(k_id<D, true>, n_node_ - first, IDG_THREADS, id_smem_bytes<D>(mleaf), st_, MIN_ADM_LEVEL,
            il, 0, nullptr, dp);
        launches_++;
        mark_end(t_bases, 2);
        t_bases = mark_begin();
        // internal nodes of every level in one dependency-ordered launch (their candidates are
        // the children's skeletons)
        IdArgs ia = il;
        ia.mcap = mcap;
        if (hint_ > 0) {
            launch_early(k_id<D, false>, hint_, IDG_THREADS, id_smem_bytes<D>(mcap), st_, 0, ia, hint_, ilist_.p, dp);
            launches_++;
        }
        mark_end(t_bases, 7);
        if (timing_) TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        sec_end("lists+bases");
        built_ = true;
        y0_from_build_ = true;
        rank_stats_valid_ = false;
        return 0;
    }

    // counting pass of the lists, the list pointers, the basis row offsets and the basis
    // launches' item lists
    void launch_list_counts()
    {
        DepArgs dp{flag_.p, tickets_.p + TICKET_LISTS, &info_.p->pad[1], ++epoch_};
        launch_early(k_lists<D>, std::min(148 * LIST_CTAS, ceil_div(cap_node_, LIST_WARPS)), 32 * LIST_WARPS, 0,
            st_, view(), list_out(), dp);
        const NodeScan q{far_cnt_.p, near_cnt_.p, fine_cnt_.p, far_ptr_.p, near_ptr_.p, rowoff_.p, ilist_.p, llist_.p,
                         blist_.p, clist_.p, flist_.p, rank_.p, node_blk_.p};
        const int nb = ceil_div(cap_node_, NODE_BLOCK);
        launch_early(k_node_sums<D>, nb, NODE_BLOCK, 0, st_, view(), q);
        launch_early(k_node_scan<D>, nb, NODE_BLOCK, 0, st_, view(), q);
        launches_ += 3;
    }

    void alloc_lists()
    {
        const size_t c = cap_node_;
        nset_.exact(c * nset_cap_);
        nset_cnt_.exact(c + 1);
        far_cnt_.exact(c + 1); near_cnt_.exact(c + 1); fine_cnt_.exact(c + 1);
        far_ptr_.exact(c + 2); near_ptr_.exact(c + 2);
        ilist_.exact(c + 1); llist_.exact(c + 1); blist_.exact(c + 1); clist_.exact(c + 1); flist_.exact(c + 1);
        rowoff_.exact(c + 2);
        rank_.exact(c);
        node_blk_.exact(ceil_div(c, NODE_BLOCK));
        far_slot_.exact(c * far_slots(D));
        near_slot_.exact(c * NEAR_SLOTS);
    }

    void product_force(void *F, DevScalars *sc, double *partials, int keep_rep) override
    {
        run_product();
        cudaEvent_t t_force = mark_begin();
        launch_z_force<D>(st_, n_, xt_.p, yp_.p, perm_.p, F, sc, partials, 1, keep_rep);
        launches_ += 2;
        mark_end(t_force, 6);
    }

    void product_host(std::vector<float> &s, std::vector<float> &v) override
    {
        run_product();
        std::vector<float4> yt(n_);
        std::vector<int> perm(n_);
        TSNE_CUDA_CHECK(cudaMemcpyAsync(yt.data(), yp_.p, sizeof(float4) * n_, cudaMemcpyDeviceToHost, st_));
        TSNE_CUDA_CHECK(cudaMemcpyAsync(perm.data(), perm_.p, sizeof(int) * n_, cudaMemcpyDeviceToHost, st_));
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        s.assign(n_, 0.f);
        v.assign((size_t)n_ * D, 0.f);
        for (int k = 0; k < n_; k++) {
            const int i = perm[k];
            const float *a = reinterpret_cast<const float *>(&yt[k]);   // s, v
            s[i] = a[0];
            for (int c = 0; c < D; c++) v[(size_t)c * n_ + i] = a[1 + c];
        }
    }

    void product_columns(const std::vector<float> &x_tree, std::vector<float> &y_tree) override
    {
        xin_.exact(n_);
        TSNE_CUDA_CHECK(cudaMemcpyAsync(xin_.p, x_tree.data(), sizeof(float4) * n_, cudaMemcpyHostToDevice, st_));
        run_product(xin_.p);
        y_tree.assign((size_t)n_ * 4, 0.f);
        TSNE_CUDA_CHECK(cudaMemcpyAsync(y_tree.data(), yp_.p, sizeof(float4) * n_, cudaMemcpyDeviceToHost, st_));
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
    }

    const int *perm_device() const override { return perm_.p; }

    const H2Stats &stats() const override
    {
        if (!rank_stats_valid_ && built_) {
            std::vector<int> r(n_node_);
            cudaStreamSynchronize(st_);
            cudaMemcpy(r.data(), rank_.p, sizeof(int) * n_node_, cudaMemcpyDeviceToHost);
            int mx = 0; double sum = 0; int cnt = 0;
            for (int x : r) if (x > 0) { mx = std::max(mx, x); sum += x; cnt++; }
            stats_.rank_max = mx;
            stats_.rank_mean = cnt ? sum / cnt : 0.0;
            rank_stats_valid_ = true;
        }
        return stats_;
    }

    void copy_tree(int *perm, double *corner, double *radius) override
    {
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        TSNE_CUDA_CHECK(cudaMemcpy(perm, perm_.p, sizeof(int) * n_, cudaMemcpyDeviceToHost));
        TreeInfo I;
        TSNE_CUDA_CHECK(cudaMemcpy(&I, info_.p, sizeof(TreeInfo), cudaMemcpyDeviceToHost));
        for (int k = 0; k < D; k++) corner[k] = I.corner[k];
        *radius = I.radius;
    }

    void copy_nodes(int *start, int *end, int *level, int *parent, int *fchild, int *nchild, int *leaf) override
    {
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        const size_t b = sizeof(int) * n_node_;
        TSNE_CUDA_CHECK(cudaMemcpy(start, start_.p, b, cudaMemcpyDeviceToHost));
        TSNE_CUDA_CHECK(cudaMemcpy(end, end_.p, b, cudaMemcpyDeviceToHost));
        TSNE_CUDA_CHECK(cudaMemcpy(level, level_.p, b, cudaMemcpyDeviceToHost));
        TSNE_CUDA_CHECK(cudaMemcpy(parent, parent_.p, b, cudaMemcpyDeviceToHost));
        TSNE_CUDA_CHECK(cudaMemcpy(fchild, fchild_.p, b, cudaMemcpyDeviceToHost));
        TSNE_CUDA_CHECK(cudaMemcpy(nchild, nchild_.p, b, cudaMemcpyDeviceToHost));
        TSNE_CUDA_CHECK(cudaMemcpy(leaf, leaf_.p, b, cudaMemcpyDeviceToHost));
    }

    void copy_lists(int *far_ptr, int *far_idx, int *near_ptr, int *near_idx) override
    {
        join_lists();
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        TSNE_CUDA_CHECK(cudaMemcpy(far_ptr, far_ptr_.p, sizeof(int) * (n_node_ + 1), cudaMemcpyDeviceToHost));
        TSNE_CUDA_CHECK(cudaMemcpy(near_ptr, near_ptr_.p, sizeof(int) * (n_node_ + 1), cudaMemcpyDeviceToHost));
        if (stats_.n_far) TSNE_CUDA_CHECK(cudaMemcpy(far_idx, far_idx_.p, sizeof(int) * stats_.n_far, cudaMemcpyDeviceToHost));
        if (stats_.n_near) TSNE_CUDA_CHECK(cudaMemcpy(near_idx, near_idx_.p, sizeof(int) * stats_.n_near, cudaMemcpyDeviceToHost));
    }

    void copy_ranks(int *rank) override
    {
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        if (built_) TSNE_CUDA_CHECK(cudaMemcpy(rank, rank_.p, sizeof(int) * n_node_, cudaMemcpyDeviceToHost));
        else for (int i = 0; i < n_node_; i++) rank[i] = 0;
    }

    int copy_bases(int *n_rows, int *max_rank, long long *row_off, float *U, float *skel) override
    {
        constexpr int MAXR = Dim<D>::MAXR;
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        if (!built_) return -1;
        *n_rows = (int)hrows_;
        *max_rank = MAXR;
        if (U == nullptr) return 0;
        TSNE_CUDA_CHECK(cudaMemcpy(row_off, rowoff_.p, sizeof(long long) * (n_node_ + 1), cudaMemcpyDeviceToHost));
        if (hrows_ > 0)
            TSNE_CUDA_CHECK(cudaMemcpy(U, U_.p, sizeof(float) * (size_t)hrows_ * MAXR, cudaMemcpyDeviceToHost));
        std::vector<Vec<D>> sk((size_t)n_node_ * MAXR);
        TSNE_CUDA_CHECK(cudaMemcpy(sk.data(), skel_.p, sizeof(Vec<D>) * sk.size(), cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < sk.size(); i++) {
            const float *f = reinterpret_cast<const float *>(&sk[i]);   // x, y (, z)
            for (int k = 0; k < D; k++) skel[i * D + k] = f[k];
        }
        return 0;
    }

    long long launches() const override { return launches_; }

    int probe_dependency_timeout(int polls) override
    {
        if (n_node_ <= 0) return -1;
        // an epoch that no launch has published: the wait runs out after `polls` polls
        DepArgs dp{flag_.p, tickets_.p, &info_.p->pad[1], epoch_ + (1 << 24), polls};
        launch_early(k_dep_probe, 1, 32, 0, st_, dp, 0);
        launches_++;
        return wait_failed();
    }

    int wait_failed() override
    {
        TreeInfo I;
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        TSNE_CUDA_CHECK(cudaMemcpy(&I, info_.p, sizeof(TreeInfo), cudaMemcpyDeviceToHost));
        return I.pad[1] != 0;
    }

    // TSNE_H2_TIMERS=1: device time per phase (CUDA events on the stream), summed over builds
    // and products until flush_timers() prints them
    void flush_timers() override
    {
        if (!timing_) return;
        TSNE_CUDA_CHECK(cudaStreamSynchronize(st_));
        static const char *names[N_PHASE] = {"tree", "lists", "leaf_bases", "far", "near", "down", "force",
                                             "internal_bases"};
        for (auto &m : marks_) {
            float ms = 0.f;
            TSNE_CUDA_CHECK(cudaEventElapsedTime(&ms, m.a, m.b));
            phase_ms_[m.phase] += ms;
            cudaEventDestroy(m.a);
            cudaEventDestroy(m.b);
        }
        marks_.clear();
        printf("H2TIMERS");
        for (int i = 0; i < N_PHASE; i++) printf(" %s=%.3f", names[i], phase_ms_[i] * 1e-3);
        printf(" (s)\n");
        fflush(stdout);
        for (double &x : phase_ms_) x = 0.0;
    }

private:
    static constexpr int BBOX_BLOCKS = 148 * 2;
    static constexpr int N_PHASE = 8;
    struct Mark { cudaEvent_t a, b; int phase; };
    bool timing_ = getenv("TSNE_H2_TIMERS") && atoi(getenv("TSNE_H2_TIMERS")) != 0;
    bool id_by_level_ = getenv("TSNE_ID_BYLEVEL") && atoi(getenv("TSNE_ID_BYLEVEL")) != 0;
    // 3D bases: k_id3 (default), or the stored matrix (k_id, TSNE_ID3=0)
    bool id3_ = !(getenv("TSNE_ID3") && atoi(getenv("TSNE_ID3")) == 0);
    std::vector<Mark> marks_;
    double phase_ms_[N_PHASE] = {0, 0, 0, 0, 0, 0, 0, 0};
    cudaEvent_t mark_begin(cudaStream_t st = nullptr)
    {
        cudaEvent_t e = nullptr;
        if (!timing_) return e;
        TSNE_CUDA_CHECK(cudaEventCreate(&e));
        TSNE_CUDA_CHECK(cudaEventRecord(e, st ? st : st_));
        return e;
    }
    // host wall time of one build section; sections slower than 10 ms are reported
    std::chrono::steady_clock::time_point sec_t0_;
    void sec_begin() { if (timing_) sec_t0_ = std::chrono::steady_clock::now(); }
    void sec_end(const char *name)
    {
        if (!timing_) return;
        const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - sec_t0_).count();
        if (ms > 10.0) printf("H2SLOW %s %.1f ms (n_node %d, max_leaf %d, far %d, near %d, nset_cap %d, cap_node %d)\n", name, ms,
                              n_node_, stats_.max_leaf, htot_[0], htot_[1], nset_cap_, cap_node_);
        sec_t0_ = std::chrono::steady_clock::now();
    }
    void mark_end(cudaEvent_t a, int phase, cudaStream_t st = nullptr)
    {
        if (!timing_) return;
        cudaEvent_t b;
        TSNE_CUDA_CHECK(cudaEventCreate(&b));
        TSNE_CUDA_CHECK(cudaEventRecord(b, st ? st : st_));
        marks_.push_back({a, b, phase});
    }

    template <bool LEAVES, int THREADS, int NS>
    static void id2_attr()
    {
        TSNE_CUDA_CHECK(cudaFuncSetAttribute(k_id2d<LEAVES, THREADS, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)id2_smem<THREADS, NS>()));
    }
    template <bool LEAVES, int THREADS, int NS>
    void id2_launch(int n_item, const int *items, const LeafItems &leaves, const IdArgs &a, const DepArgs &dp,
                    int ctas = 0)
    {
        launch_early(k_id2d<LEAVES, THREADS, NS>, ctas > 0 ? ctas : n_item, THREADS, id2_smem<THREADS, NS>(),
            st_, n_item, items, leaves, a, dp);
        launches_++;
    }
    template <bool LEAVES, int THREADS, int ROWS>
    static void id3_attr()
    {
        TSNE_CUDA_CHECK(cudaFuncSetAttribute(k_id3<LEAVES, THREADS, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)Id3<THREADS, ROWS>::smem()));
    }
    template <bool LEAVES, int THREADS, int ROWS>
    void id3_launch(int n_item, const int *items, int mlo, int chains, const IdArgs &a, const DepArgs &dp)
    {
        launch_early(k_id3<LEAVES, THREADS, ROWS>, n_item, THREADS, Id3<THREADS, ROWS>::smem(), st_, n_item,
            items, mlo, chains, a, dp);
        launches_++;
    }

    void alloc_nodes()
    {
        const size_t c = cap_node_;
        start_.exact(c); end_.exact(c); level_.exact(c); parent_.exact(c); fchild_.exact(c);
        nchild_.exact(c); leaf_.exact(c); ix_.exact(3 * c);
        rec_.exact(2 * c);
        bset_.exact(c * (Dim<D>::L + 1));
        flag_.exact(c);
        TSNE_CUDA_CHECK(cudaMemsetAsync(flag_.p, 0, sizeof(int) * c, st_));
        flag2_.exact(c);
        TSNE_CUDA_CHECK(cudaMemsetAsync(flag2_.p, 0, sizeof(int) * c, st_));
        nid_.exact(c * (Dim<D>::L + 1));
        alloc_lists();
    }

    TreeView view()
    {
        TreeView v;
        v.n = n_; v.L = Dim<D>::L; v.leaf_size = leaf_size_; v.cap_node = cap_node_; v.nset_cap = nset_cap_;
        v.keys = keys_.p; v.start = start_.p; v.end = end_.p; v.level = level_.p; v.parent = parent_.p;
        v.fchild = fchild_.p; v.nchild = nchild_.p; v.leaf = leaf_.p; v.ix = ix_.p; v.rec = rec_.p; v.proxies = proxies_.p;
        v.fm = fm_.p; v.blkcnt = blkcnt_.p; v.blkoff = blkoff_.p;
        v.bset = bset_.p; v.nid = nid_.p; v.btot = btot_.p; v.tickets = tickets_.p;
        v.info = info_.p;
        return v;
    }

    ListOut list_out()
    {
        ListOut lo;
        lo.far_cnt = far_cnt_.p; lo.near_cnt = near_cnt_.p;
        lo.fine_cnt = fine_cnt_.p;
        lo.far_ptr = far_ptr_.p; lo.near_ptr = near_ptr_.p;
        lo.far_idx = far_idx_.p; lo.near_idx = near_idx_.p;
        lo.nset = nset_.p; lo.nset_cnt = nset_cnt_.p;
        lo.far_slot = far_slot_.p;
        lo.near_slot = near_slot_.p;
        lo.slot_over = &info_.p->pad[2];
        return lo;
    }

    void sort_reserve(DevBuf<int> &idx, DevBuf<int> &alt, int count, const int *ptr)
    {
        if (count <= 1) return;
        alt.ensure(count);
        cub::DoubleBuffer<int> keys(idx.p, alt.p);
        size_t need = 0;
        TSNE_CUDA_CHECK(cub::DeviceSegmentedSort::SortKeys(nullptr, need, keys, count, n_node_, ptr, ptr + 1, st_));
        if (need > cub_tmp_.cap) cub_tmp_.exact(need + 256);
    }
    // ascending order inside every node's segment [ptr[t], ptr[t + 1]) of idx (count entries)
    // (sort_reserve allocates its partner buffer and scratch beforehand)
    void sort_segments(DevBuf<int> &idx, DevBuf<int> &alt, int count, const int *ptr, cudaStream_t st)
    {
        if (count <= 1) return;
        cub::DoubleBuffer<int> keys(idx.p, alt.p);
        size_t bytes = cub_tmp_.cap;
        TSNE_CUDA_CHECK(cub::DeviceSegmentedSort::SortKeys(cub_tmp_.p, bytes, keys, count, n_node_, ptr, ptr + 1, st));
        if (keys.Current() != idx.p) idx.swap(alt);
        launches_ += 2;
    }
    ProdArgs prod_args(const float4 *xin)
    {
        ProdArgs g;
        g.xin = xin;
        g.tv = view(); g.xt = xt_.p; g.skel = skel_.p; g.rank = rank_.p; g.rowoff = rowoff_.p; g.U = U_.p;
        g.y0 = y0_.p; g.y1 = y1_.p; g.yp = yp_.p;
        g.far_ptr = far_ptr_.p; g.far_idx = far_idx_.p; g.near_ptr = near_ptr_.p; g.near_idx = near_idx_.p;
        g.fine_cnt = fine_cnt_.p;
        return g;
    }
    template <int PART>
    void launch_near(const ProdArgs &g, cudaStream_t st)
    {
        if (D == 2 && g.xin == nullptr) launch_early(k_near2d<PART>, n_node_, NEAR2_THREADS, 0, st, g);
        else launch_early(k_near<D, 4, PART>, n_node_, NEAR_THREADS, PART == NEAR_BLOCKS ? near_spread() : 0, st, g);
        launches_++;
    }
    // The internal 3D bases' CTAs take a whole SM each, and where there are more of them than SMs the
    // near blocks beside them start on the first few SMs that come free. Few and large leaves
    // would all go there, up to sixteen CTAs to an SM, and the others idle: 200K points on a line, 357 leaves of
    // up to 700, took 7.8 ms that way and take 1.7 spread over the chip. So a CTA asks for as much shared
    // memory (unused) as leaves room for no more than an SM's share of the leaves; nothing from 16 to an SM on.
    size_t near_spread() const
    {
        constexpr size_t SM = 228 * 1024, RESERVED = 1024;   // an SM's shared memory, and the part per CTA
        const int share = std::max(1, ceil_div(n_node_ - hint_, 148));
        if (D == 2 || share >= 2048 / NEAR_THREADS) return 0;
        return std::min<size_t>(SM / share / 1024 * 1024 - RESERVED - NEAR_OWN, NEAR_MOST);
    }
    // k_near's own shared memory, and the most that a launch may ask for beside it (the kernel's limit is this
    // constant for every workspace: it is the process's, and threads build at the same time)
    static constexpr size_t NEAR_OWN = NEAR_THREADS * (sizeof(Vec<D>) + sizeof(float4));
    static constexpr size_t NEAR_MOST = 227 * 1024 - NEAR_OWN;
    // The near blocks of the force product ([1 | Y] columns) need only the tree, the points and
    // the near lists, so a build runs them on a side stream beside the internal bases, whose
    // dependency chain leaves SMs idle. The fork point follows the leaf bases (which fill the
    // GPU by themselves); the internal bases are queued before the near blocks, so their CTAs
    // are dispatched first. The product joins the side stream before the first kernel that
    // adds to their output (the leaves' far entries with finer sources, which read the bases,
    // then k_down_leaves).
    void near_fork_point() { TSNE_CUDA_CHECK(cudaEventRecord(fork_ev_, st_)); }
    void near_launch_side()
    {
        TSNE_CUDA_CHECK(cudaStreamWaitEvent(st2_, fork_ev_, 0));
        launch_near<NEAR_BLOCKS>(prod_args(nullptr), st2_);
        TSNE_CUDA_CHECK(cudaEventRecord(near_ev_, st2_));
        near_pending_ = true;
    }
    void join_lists()
    {
        if (!lists_pending_) return;
        TSNE_CUDA_CHECK(cudaStreamWaitEvent(st_, lists_ev_, 0));
        lists_pending_ = false;
    }
    void join_near()
    {
        join_lists();
        if (!near_pending_) return;
        TSNE_CUDA_CHECK(cudaStreamWaitEvent(st_, near_ev_, 0));
        near_pending_ = false;
    }

    void run_product(const float4 *xin = nullptr)
    {
        const bool near_done = near_pending_ && xin == nullptr;   // the side stream's near field
        if (!near_done) join_near();                              // other columns rewrite it
        else join_lists();
        const ProdArgs g = prod_args(xin);
        const TreeInfo &I = *hinfo_.p;
        if (xin != nullptr || !y0_from_build_) {
            for (int l = max_level_; l >= MIN_ADM_LEVEL; l--) {
                const int nl = I.n_level_nodes[l];
                if (nl > 0) { launch_early(k_up<D>, grid_for((long long)nl * 32, 256), 256, 0, st_, l, g);
                    launches_++; }
            }
        }
        y0_from_build_ = y0_from_build_ && xin == nullptr;
        const int first = I.level_begin[MIN_ADM_LEVEL];
        // the leaves' finer far entries read the bases and add to the near blocks' sums: they
        // follow the near blocks on the side stream, beside the far field and the downward pass
        if (near_done && hfine_ > 0) {
            TSNE_CUDA_CHECK(cudaEventRecord(fork_ev_, st_));
            TSNE_CUDA_CHECK(cudaStreamWaitEvent(st2_, fork_ev_, 0));
            launch_early(k_fine<D>, hfine_, 32 * FAR_WARPS, 0, st2_, flist_.p, g);
            TSNE_CUDA_CHECK(cudaEventRecord(near_ev_, st2_));
            launches_++;
        }
        cudaEvent_t t_far = mark_begin();
        launch_early(k_far_c<D>, grid_for((long long)(n_node_ - first) * far_halves(D), FAR_WARPS, 148 * 32), 32
            * FAR_WARPS, 0, st_, first, n_node_, g);
        mark_end(t_far, 3);
        launches_++;
        cudaEvent_t t_near = mark_begin();
        if (!near_done) launch_near<NEAR_ALL>(g, st_);
        mark_end(t_near, 4);
        cudaEvent_t t_down = mark_begin();
        if (hint_ > 0) {
            DepArgs dp{flag_.p, tickets_.p + TICKET_DOWN, &info_.p->pad[1], ++epoch_};
            launch_early(k_down_internal<D>, grid_for((long long)hint_ * 32, 256, 148 * 8), 256, 0, st_, hint_,
                ilist_.p, g, dp);
            launches_++;
        }
        if (near_done) join_near();
        launch_early(k_down_leaves<D>, grid_for((long long)(n_node_ - first) * 32, 256), 256, 0, st_, g);
        launches_++;
        mark_end(t_down, 5);
    }

    int n_;
    cudaStream_t st_;
    int leaf_size_ = 100;
    int cap_node_ = 0, nset_cap_ = 0;
    int n_node_ = 0, max_level_ = 0, last_max_level_ = 0;
    bool built_ = false;
    bool y0_from_build_ = false;   // y0 holds U^T [1 | Y] of the last build
    mutable bool rank_stats_valid_ = false;
    mutable H2Stats stats_;
    long long launches_ = 0;
    size_t sort_bytes_ = 0;
    int htot_[2] = {0, 0};
    long long hrows_ = 0;

    DevBuf<unsigned long long> keys_in_, keys_;
    DevBuf<int> idx_in_, perm_;
    DevBuf<Vec<D>> xt_;
    DevBuf<unsigned char> cub_tmp_;
    DevBuf<double> bbox_part_;
    DevBuf<TreeInfo> info_;
    HostPinned<TreeInfo> hinfo_;
    DevBuf<int> start_, end_, level_, parent_, fchild_, nchild_, leaf_, ix_;
    DevBuf<int> fm_, blkcnt_, blkoff_, bset_, nid_, btot_;
    DevBuf<int> flag_, tickets_;  // dependency-ordered launches
    DevBuf<int> done_;            // finished blocks of the bounding-box launch
    DevBuf<int> flag2_;           // second flags (bases: upward coefficients final)
    cudaStream_t st2_ = nullptr;  // side stream: the list write and the near field beside the bases
    cudaEvent_t fork_ev_ = nullptr, near_ev_ = nullptr, lists_ev_ = nullptr;
    bool near_pending_ = false, lists_pending_ = false;
    DevBuf<float4> proxies_;             // proxy table, a row per level
    DevBuf<int4> rec_;                   // node records of the list pass
    DevBuf<int> far_slot_, near_slot_;   // list entries parked by the count pass
    int epoch_ = 0;
    DevBuf<int> nset_, nset_cnt_, far_cnt_, near_cnt_, far_ptr_, near_ptr_, far_idx_, near_idx_;
    DevBuf<int> far_alt_, near_alt_;   // segmented-sort partners of the 3D lists
    DevBuf<NodeSums> node_blk_;          // block sums of the node scan
    DevBuf<int> ilist_;                  // internal nodes at level >= 2, in increasing id
    DevBuf<int> llist_;                  // leaves at level >= 2 of at most TINY_LEAF points
    DevBuf<int> blist_, clist_;          // the larger leaves at level >= 2
    DevBuf<int> flist_, fine_cnt_;       // leaves with finer far entries, and how many each node has
    int hint_ = 0, hleaf_ = 0, hbig_ = 0, hlarge_ = 0, hfine_ = 0;
    cudaEvent_t counts_ev_ = nullptr;   // end of a build's count batch (host waits on it)
    DevBuf<long long> rowoff_;
    DevBuf<int> rank_;
    DevBuf<Vec<D>> skel_;
    DevBuf<float4> y0_, y1_, yp_, xin_;
    DevBuf<float> U_;
    DevBuf<float> gA_, gnrm_;
    DevBuf<int> gsel_;
    DevBuf<Vec<D>> gcand_;
};

// The terms are the buffers of H2Impl. The nodes that a tree will have are taken from embeddings of uniform,
// normal and clustered points and of runs (30K and 200K points, leaf sizes 2 to 300): at most 4.3 n / leaf_size nodes in
// 2D and 6.5 in 3D, of them 1.13 and 0.91 internal. Tight clumps of more points than a leaf holds, each a chain
// of nodes down to the clump's size, can have more.
template <int D>
size_t h2_bytes(int n, int leaf_size)
{
    using Impl = H2Impl<D>;
    constexpr size_t V = sizeof(Vec<D>), MAXR = Dim<D>::MAXR, P = Dim<D>::NPROXY;
    const double nodes = (D == 2 ? 4.5 : 6.6) * n / leaf_size, internal = (D == 2 ? 1.2 : 0.95) * n / leaf_size;
    double cap = Impl::first_cap_node(n);
    while (cap < nodes) cap *= 2;
    const size_t point = 2 * (sizeof(unsigned long long) + sizeof(int)) + V + sizeof(float4) + sizeof(int) +
                         sizeof(unsigned long long) + sizeof(int);   // (the radix sort's scratch)
    const size_t entry = sizeof(int) * (24 + 2 * (Dim<D>::L + 1) + Dim<D>::NSET + far_slots(D) + NEAR_SLOTS) +
                         2 * sizeof(int4) + sizeof(long long);       // of the node table and the list pass
    const size_t node = MAXR * (V + 2 * sizeof(float4)) + sizeof(int) * 160;   // bases and list entries
    size_t row = sizeof(float) * MAXR;                                         // of the interpolation matrices
    if (leaf_size > (D == 2 ? Impl::id_mcap() : ID3_ROWS)) row += sizeof(float) * (P + 2) + sizeof(int) + V;
    const double rows = n + internal * (1 << D) * MAXR;
    return (size_t)((double)point * n + entry * cap + 1.25 * (node * nodes + row * rows));   // 1.25: DevBuf::ensure
}

}  // namespace

size_t h2_device_bytes(int d, int n, int leaf_size)
{
    return d == 2 ? h2_bytes<2>(n, leaf_size) : h2_bytes<3>(n, leaf_size);
}

std::unique_ptr<H2Matrix> make_h2_matrix(int d, int n, cudaStream_t st)
{
    if (d == 2) return std::unique_ptr<H2Matrix>(new H2Impl<2>(n, st));
    return std::unique_ptr<H2Matrix>(new H2Impl<3>(n, st));
}

}  // namespace tsne
