/*
 * lbvh.cu - device-built linear BVH over a snapshot's primitive boxes
 * (Karras, "Maximizing Parallelism in the Construction of BVHs, Octrees,
 * and k-d Trees", HPG 2012), emitted in the DNode layout the traversal reads.
 *
 * It replaces, on the device, the per-solve Star-3D view build of the
 * reference (src/ssol_scene.c:347-433, s3d_scene_view_create at :410-413).
 * Seven steps on one stream, without a read-back between them:
 *   1. centroid bounds of the primitive boxes (one block);
 *   2. 30-bit Morton code of each centroid in those bounds (10 bits per axis);
 *   3. stable LSD radix sort of (code, primitive) pairs, 4 passes of 8 bits,
 *      in one block of 1024 threads: per 1024-element tile each warp ranks
 *      its lanes by digit with __match_any_sync, the tile's digit offsets
 *      come from a prefix over the warps, so equal codes keep their input
 *      order and the tree is the same on every run;
 *   4. one thread per internal node finds its key range and split from the
 *      sorted codes (longest common prefix, with the sorted position breaking
 *      ties between equal codes); internal node 0 is the root; leaves are
 *      single primitives (count 1, the child field holds the primitive
 *      reference itself);
 *   5. one thread per leaf walks toward the root writing each child box into
 *      its parent's slot; the second thread to reach a node (an atomic
 *      arrival count) merges the node's two slots and goes on, the first
 *      stops, so no thread waits on another. The same walk computes each
 *      node's SAH cost, height and internal-node count;
 *   6. treelet restructuring for a lower SAH cost (Karras and Aila, HPG
 *      2013): the nodes grouped by height, lowest first, one warp per node,
 *      whose lanes share the dynamic program over the treelet's leaf subsets;
 *      one launch for each of the lower heights and one block for the rest;
 *      the root's height is the tree depth, which the host reads back to check
 *      the traversal stack bound;
 *   7. the internal nodes are renumbered depth first, slot 0 first, so that
 *      a node's first child follows it in memory; where the tree joins pairs
 *      (joins_pairs), a node of two primitives becomes one of its parent.
 * Scenes of at most SMALL_BUILD primitives go through all of them in one
 * launch.
 */
#include "kernels.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>

namespace ssolb {

namespace {

template<class R> __device__ __forceinline__ R rmax();
template<> __device__ __forceinline__ float rmax<float>() { return FLT_MAX; }
template<> __device__ __forceinline__ double rmax<double>() { return DBL_MAX; }

constexpr int SORT_THREADS = 1024;
constexpr int SORT_WARPS = SORT_THREADS / 32;

/* Spread the low 10 bits of v to every third bit */
__device__ __forceinline__ uint32_t spread3(uint32_t v)
{
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

template<class R>
__device__ __forceinline__ R centroid(const R* box, int i, int c)
{
  return (R)0.5 * (box[6 * i + c] + box[6 * i + 3 + c]);
}

/* Steps 1 to 3 run in one block of SORT_THREADS threads */

/* Step 1: bounds of the centroids */
template<class R>
__device__ __forceinline__ void lbvh_bounds(const R* box, int n, R* cb)
{
  __shared__ R red[6][SORT_WARPS];
  R lo[3], hi[3];
  for(int c = 0; c < 3; ++c) {
    lo[c] = centroid(box, 0, c);
    hi[c] = lo[c];
  }
  for(int i = threadIdx.x; i < n; i += blockDim.x)
    for(int c = 0; c < 3; ++c) {
      const R x = centroid(box, i, c);
      lo[c] = fmin(lo[c], x);
      hi[c] = fmax(hi[c], x);
    }
  for(int o = 16; o > 0; o >>= 1)
    for(int c = 0; c < 3; ++c) {
      lo[c] = fmin(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = fmax(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if(lane == 0)
    for(int c = 0; c < 3; ++c) {
      red[c][w] = lo[c];
      red[3 + c][w] = hi[c];
    }
  __syncthreads();
  if(threadIdx.x < 6) {
    const int q = threadIdx.x;
    R v = red[q][0];
    for(int k = 1; k < (int)(blockDim.x >> 5); ++k)
      v = q < 3 ? fmin(v, red[q][k]) : fmax(v, red[q][k]);
    cb[q] = v;
  }
}

/* Step 2: Morton codes; vals are the primitives' input positions */
template<class R>
__device__ __forceinline__ void lbvh_morton(const R* box, int n, const R* cb, uint32_t* keys,
                                            uint32_t* vals)
{
  for(int i = threadIdx.x; i < n; i += SORT_THREADS) {
    uint32_t q[3];
    for(int c = 0; c < 3; ++c) {
      const R ext = cb[3 + c] - cb[c];
      const R t = ext > (R)0 ? (centroid(box, i, c) - cb[c]) / ext : (R)0;
      const R s = t * (R)1024;
      q[c] = s <= (R)0 ? 0u : s >= (R)1023 ? 1023u : (uint32_t)s;
    }
    keys[i] = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
    vals[i] = (uint32_t)i;
  }
}

/* Step 3: stable radix sort; (k0, v0) in and out, (k1, v1) scratch;
 * wcnt: SORT_WARPS x 256 words of shared memory */
__device__ __forceinline__ void lbvh_sort
  (uint32_t (*wcnt)[256], uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1, int n)
{
  __shared__ uint32_t base[256];
  __shared__ uint32_t tile_total[256];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const unsigned lt = (1u << lane) - 1u;
  for(int pass = 0; pass < 4; ++pass) {
    const int shift = 8 * pass;
    const uint32_t* sk = pass & 1 ? k1 : k0;
    const uint32_t* sv = pass & 1 ? v1 : v0;
    uint32_t* dk = pass & 1 ? k0 : k1;
    uint32_t* dv = pass & 1 ? v0 : v1;
    if(tid < 256) tile_total[tid] = 0;
    __syncthreads();
    for(int i = tid; i < n; i += SORT_THREADS) atomicAdd(&tile_total[(sk[i] >> shift) & 255u], 1u);
    __syncthreads();
    if(tid < 32) {
      /* exclusive scan of the 256 digit counts by one warp, 8 per lane */
      uint32_t c[8], s = 0;
      for(int k = 0; k < 8; ++k) { c[k] = tile_total[8 * lane + k]; s += c[k]; }
      uint32_t inc = s;
      for(int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if(lane >= o) inc += y;
      }
      uint32_t run = inc - s;
      for(int k = 0; k < 8; ++k) { base[8 * lane + k] = run; run += c[k]; }
    }
    __syncthreads();
    for(int t0 = 0; t0 < n; t0 += SORT_THREADS) {
      const int i = t0 + tid;
      const bool valid = i < n;
      const uint32_t key = valid ? sk[i] : 0u, val = valid ? sv[i] : 0u;
      const uint32_t d = (key >> shift) & 255u;
      uint32_t* flat = &wcnt[0][0];
      for(int k = tid; k < SORT_WARPS * 256; k += SORT_THREADS) flat[k] = 0;
      __syncthreads();
      /* invalid lanes group under 256, which no digit takes */
      const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 256u);
      const uint32_t rank = __popc(peers & lt);
      if(valid && rank == 0) wcnt[w][d] = __popc(peers);
      __syncthreads();
      if(tid < 256) {
        uint32_t s = 0;
        for(int k = 0; k < SORT_WARPS; ++k) {
          const uint32_t c = wcnt[k][tid];
          wcnt[k][tid] = s;
          s += c;
        }
        tile_total[tid] = s;
      }
      __syncthreads();
      if(valid) {
        const uint32_t pos = base[d] + wcnt[w][d] + rank;
        dk[pos] = key;
        dv[pos] = val;
      }
      __syncthreads();
      if(tid < 256) base[tid] += tile_total[tid];
      __syncthreads();
    }
  }
}

/* Longest common prefix of sorted keys i and j (-1 outside [0, n)); equal
 * keys compare their positions, as if each key carried its position in its
 * low 32 bits */
__device__ __forceinline__ int lcp(const uint32_t* k, int n, int i, int j)
{
  if(j < 0 || j >= n) return -1;
  const uint32_t a = k[i], b = k[j];
  return a == b ? 32 + __clz(i ^ j) : __clz(a ^ b);
}

/* Step 4: internal node i of n - 1. parent[] holds (parent << 1) | slot:
 * entries [0, n - 1) for internal nodes, [n - 1, 2n - 1) for leaves. */
template<class R>
__device__ __forceinline__ void lbvh_node(const uint32_t* keys, const uint32_t* vals,
                                          const uint32_t* ref, int n, int i, DNode<R>* nodes,
                                          int32_t* parent)
{
  const int d = lcp(keys, n, i, i + 1) - lcp(keys, n, i, i - 1) > 0 ? 1 : -1;
  const int dmin = lcp(keys, n, i, i - d);
  int lmax = 2;
  while(lcp(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for(int t = lmax >> 1; t >= 1; t >>= 1)
    if(lcp(keys, n, i, i + (l + t) * d) > dmin) l += t;
  const int j = i + l * d;
  const int dnode = lcp(keys, n, i, j);
  int s = 0;
  for(int t = l;;) {
    t = (t + 1) >> 1;
    if(lcp(keys, n, i, i + (s + t) * d) > dnode) s += t;
    if(t == 1) break;
  }
  const int g = i + s * d + (d < 0 ? -1 : 0);
  const int lo = min(i, j), hi = max(i, j);
  DNode<R>& N = nodes[i];
  const int c[2] = {g, g + 1};
  const bool leaf[2] = {lo == g, hi == g + 1};
  for(int k = 0; k < 2; ++k) {
    if(leaf[k]) {
      N.child[k] = (int32_t)ref[vals[c[k]]];
      N.count[k] = 1;
      parent[(n - 1) + c[k]] = (i << 1) | k;
    } else {
      N.child[k] = c[k];
      N.count[k] = 0;
      parent[c[k]] = (i << 1) | k;
    }
  }
  if(i == 0) parent[0] = -1;
}

template<class R>
__device__ __forceinline__ void put_slot(DNode<R>& N, int k, const R lo[3], const R hi[3])
{
  for(int c = 0; c < 3; ++c) {
    N.lo[k][c] = lo[c];
    N.hi[k][c] = hi[c];
  }
}

/* Surface-area heuristic: a node costs C_NODE x its surface area (a ray
 * that reaches it tests both child boxes), a primitive C_PRIM x its box's
 * (Karras and Aila's constants; areas are half surface areas, the factor
 * cancels) */
constexpr float C_NODE = 1.2f, C_PRIM = 1.0f;
constexpr int TREELET = 6; /* leaves of a restructured treelet (7 gave a 0.2 % lower SAH
                              * cost on the field for 3x the work) */

template<class R>
__device__ __forceinline__ float half_area(const R lo[3], const R hi[3])
{
  const float dx = (float)(hi[0] - lo[0]), dy = (float)(hi[1] - lo[1]),
              dz = (float)(hi[2] - lo[2]);
  return dx * dy + dy * dz + dz * dx;
}

/* Per internal node: SAH cost, height, internal nodes in its subtree
 * (itself included) and parent link ((parent << 1) | slot; entries
 * [n - 1, 2n - 1) are the leaves') */
struct Aux {
  float* cost;
  int32_t* height;
  int32_t* ninner;
  int32_t* parent;
};

/* A treelet leaf: a slot's box, what it holds (a primitive, count 1, or a
 * subtree, count 0), and the subtree's cost, height and internal nodes */
template<class R> struct TLeaf {
  R lo[3], hi[3];
  int32_t child, count;
  float cost;
  int height, ninner;
};

/* Slot k of node N as written by other threads of this launch: read past L1 */
template<class R>
__device__ __forceinline__ void read_slot(const DNode<R>& N, int k, const Aux& A, TLeaf<R>& L)
{
  for(int c = 0; c < 3; ++c) {
    L.lo[c] = __ldcg(&N.lo[k][c]);
    L.hi[c] = __ldcg(&N.hi[k][c]);
  }
  L.child = __ldcg(&N.child[k]);
  L.count = __ldcg(&N.count[k]);
  if(L.count == 0) {
    L.cost = __ldcg(&A.cost[L.child]);
    L.height = __ldcg(&A.height[L.child]);
    L.ninner = __ldcg(&A.ninner[L.child]);
  } else {
    L.cost = C_PRIM * half_area(L.lo, L.hi);
    L.height = 0;
    L.ninner = 0;
  }
}

/* Both slots of a node by the warp, 8 lanes a slot: two loads one after the
 * other (the slot, then what is known of its subtree) instead of 22 */
template<class R>
__device__ __forceinline__ void read_slots(const DNode<R>& N, const Aux& A, TLeaf<R>& L0,
                                           TLeaf<R>& L1, int lane)
{
  const int k = lane >> 3, f = lane & 7;
  TLeaf<R>& L = k ? L1 : L0;
  if(lane < 16) {
    if(f < 3) L.lo[f] = __ldcg(&N.lo[k][f]);
    else if(f < 6) L.hi[f - 3] = __ldcg(&N.hi[k][f - 3]);
    else if(f == 6) L.child = __ldcg(&N.child[k]);
    else L.count = __ldcg(&N.count[k]);
  }
  __syncwarp();
  if(lane < 16) {
    const bool inner = L.count == 0;
    if(f == 0) L.cost = inner ? __ldcg(&A.cost[L.child]) : C_PRIM * half_area(L.lo, L.hi);
    else if(f == 1) L.height = inner ? __ldcg(&A.height[L.child]) : 0;
    else if(f == 2) L.ninner = inner ? __ldcg(&A.ninner[L.child]) : 0;
  }
  __syncwarp();
}

template<class R>
__device__ __forceinline__ void union_of(const TLeaf<R>* L, int S, R lo[3], R hi[3])
{
  for(int c = 0; c < 3; ++c) { lo[c] = rmax<R>(); hi[c] = -rmax<R>(); }
  for(int i = 0; S; ++i, S >>= 1)
    if(S & 1)
      for(int c = 0; c < 3; ++c) {
        lo[c] = fmin(lo[c], L[i].lo[c]);
        hi[c] = fmax(hi[c], L[i].hi[c]);
      }
}

/* The new internal nodes of a treelet: the leaf subset and node index of
 * each, and its two children (another of them, or -1 - leaf) */
struct Rebuilt {
  int cnt, nset[TREELET - 1], nidx[TREELET - 1], kid[TREELET - 1][2];
};

/* Rewrite the internal nodes of a treelet (root first, then inner[1..]) to
 * the binary tree over its nl leaves that part[] describes (part[S]: the
 * subset holding S's lowest leaf), and set their parent links, costs (c[]),
 * heights and internal node counts. The root keeps its index and box; the
 * leaves' subtrees are untouched. Lane 0 lays the tree out, then one lane
 * writes each slot. */
template<class R>
__device__ __forceinline__ void rebuild_treelet
  (DNode<R>* nodes, const Aux& A, const TLeaf<R>* L, int nl, const int* inner, const float* c,
   const uint8_t* part, Rebuilt& B, int lane)
{
  if(lane == 0) {
    int cnt = 1;
    B.nset[0] = (1 << nl) - 1;
    B.nidx[0] = inner[0];
    for(int q = 0; q < cnt; ++q)
      for(int k = 0; k < 2; ++k) {
        const int S = B.nset[q], T = k ? S ^ part[S] : part[S];
        if(__popc(T) == 1) {
          B.kid[q][k] = -__ffs(T);
        } else {
          B.nset[cnt] = T;
          B.nidx[cnt] = inner[cnt];
          B.kid[q][k] = cnt++;
        }
      }
    B.cnt = cnt;
  }
  __syncwarp();
  if(lane < 2 * B.cnt) {
    const int q = lane >> 1, k = lane & 1, nd = B.nidx[q], e = B.kid[q][k];
    DNode<R>& N = nodes[nd];
    if(e < 0) {
      const TLeaf<R>& leaf = L[-1 - e];
      put_slot(N, k, leaf.lo, leaf.hi);
      N.child[k] = leaf.child;
      N.count[k] = leaf.count;
      if(leaf.count == 0) A.parent[leaf.child] = (nd << 1) | k;
    } else {
      R lo[3], hi[3];
      union_of(L, B.nset[e], lo, hi);
      put_slot(N, k, lo, hi);
      N.child[k] = B.nidx[e];
      N.count[k] = 0;
      A.parent[B.nidx[e]] = (nd << 1) | k;
    }
  }
  if(lane == 0) {
    int hh[TREELET - 1], nn[TREELET - 1];
    for(int q = B.cnt - 1; q >= 0; --q) {
      int hm = 0, sum = 1;
      for(int k = 0; k < 2; ++k) {
        const int e = B.kid[q][k];
        hm = max(hm, e >= 0 ? hh[e] : L[-1 - e].height);
        sum += e >= 0 ? nn[e] : L[-1 - e].ninner;
      }
      hh[q] = 1 + hm;
      nn[q] = sum;
      A.cost[B.nidx[q]] = c[B.nset[q]];
      A.height[B.nidx[q]] = hh[q];
      A.ninner[B.nidx[q]] = nn[q];
    }
  }
}

constexpr int MAX_LEVELS = 128;

/* Internal nodes grouped by height (one block): level_first[h] .. [h + 1]
 * of level_nodes; *maxh the largest height present. Nodes of one height
 * are never ancestors of one another, so their treelets are disjoint. */
__device__ __forceinline__ void lbvh_levels
  (const int32_t* height, int m, int32_t* level_first, int32_t* level_nodes, int32_t* maxh)
{
  __shared__ uint32_t cnt[MAX_LEVELS], cur[MAX_LEVELS];
  const int tid = threadIdx.x;
  for(int h = tid; h < MAX_LEVELS; h += SORT_THREADS) cnt[h] = 0;
  __syncthreads();
  for(int i = tid; i < m; i += SORT_THREADS)
    atomicAdd(&cnt[min(max(height[i], 0), MAX_LEVELS - 1)], 1u);
  __syncthreads();
  if(tid == 0) {
    uint32_t run = 0;
    int mh = 0;
    for(int h = 0; h < MAX_LEVELS; ++h) {
      level_first[h] = (int32_t)run;
      cur[h] = run;
      run += cnt[h];
      if(cnt[h]) mh = h;
    }
    level_first[MAX_LEVELS] = (int32_t)run;
    *maxh = mh;
  }
  __syncthreads();
  for(int i = tid; i < m; i += SORT_THREADS)
    level_nodes[atomicAdd(&cur[min(max(height[i], 0), MAX_LEVELS - 1)], 1u)] = i;
}

constexpr int TREELET_WARPS = 4;

/* Shared memory of a warp's treelet */
template<class R> struct TreeletScratch {
  TLeaf<R> L[TREELET];
  float c[1 << TREELET]; /* cost of the best tree over a leaf subset */
  float area[1 << TREELET]; /* half area of its box */
  uint8_t part[1 << TREELET];
  int inner[TREELET - 1];
  Rebuilt rebuilt;
};

/* The subsets of two to five of TREELET leaves, by size, and where each size
 * starts */
__constant__ uint8_t SUBSETS[] = {
  3, 5, 6, 9, 10, 12, 17, 18, 20, 24, 33, 34, 36, 40, 48,
  7, 11, 13, 14, 19, 21, 22, 25, 26, 28, 35, 37, 38, 41, 42, 44, 49, 50, 52, 56,
  15, 23, 27, 29, 30, 39, 43, 45, 46, 51, 53, 54, 57, 58, 60,
  31, 47, 55, 59, 61, 62};
__constant__ uint8_t SUBSET_FIRST[] = {0, 15, 35, 50, 56};
static_assert(TREELET == 6, "SUBSETS lists the subsets of six leaves");

/* Treelet restructuring (Karras and Aila, "Fast Parallel Construction of
 * High-Quality Bounding Volume Hierarchies", HPG 2013) of node `root` by one
 * warp, once its subtree is final. The node's cost, height and node count are
 * refreshed from its slots (its descendants may have changed), and a treelet
 * of up to TREELET leaves grown by opening the leaf of largest area that is a
 * subtree; the lanes then find the binary tree over those leaves of lowest
 * SAH cost by dynamic programming over their subsets, all subsets of one size
 * at a time, and rewrite the treelet's internal nodes to it if it is cheaper.
 * Bound by the chain of loads and shared-memory steps of one warp, so the
 * boxes of all subsets are formed first, the lanes of a step hold one subset
 * each, and the partitions of the whole set are spread over the lanes: a
 * height of few nodes takes 12 to 19 us, and took 30 with a lane going
 * through its subsets one after the other. */
template<class R>
__device__ __forceinline__ void restructure
  (DNode<R>* nodes, const Aux& A, int root, int32_t* depth, TreeletScratch<R>& M, int lane)
{
  TLeaf<R>* L = M.L;
  float* c = M.c;
  uint8_t* part = M.part;
  read_slots(nodes[root], A, L[0], L[1], lane);
  R lo[3], hi[3];
  union_of(L, 3, lo, hi);
  const float cur = C_NODE * half_area(lo, hi) + L[0].cost + L[1].cost;
  if(lane == 0) {
    const int h = 1 + max(L[0].height, L[1].height);
    A.cost[root] = cur;
    A.height[root] = h;
    A.ninner[root] = 1 + L[0].ninner + L[1].ninner;
    if(root == 0) *depth = h;
    M.inner[0] = root;
  }
  int nl = 2, ni = 1;
  while(nl < TREELET) {
    /* the subtree of largest area, the first of equal ones */
    unsigned key = 0;
    if(lane < nl && L[lane].count == 0)
      key = __float_as_uint(half_area(L[lane].lo, L[lane].hi)) + 1u;
    const unsigned top = __reduce_max_sync(0xffffffffu, key);
    if(top == 0u) break;
    const int best = __ffs(__ballot_sync(0xffffffffu, key == top)) - 1;
    const int nd = L[best].child;
    if(lane == 0) M.inner[ni] = nd;
    ++ni;
    __syncwarp();
    read_slots(nodes[nd], A, L[best], L[nl], lane);
    ++nl;
  }
  __syncwarp();
  if(nl >= 3) {
    const int full = (1 << nl) - 1;
    for(int S = lane + 1; S <= full; S += 32) {
      for(int k = 0; k < 3; ++k) { lo[k] = rmax<R>(); hi[k] = -rmax<R>(); }
#pragma unroll
      for(int i = 0; i < TREELET; ++i)
        if((S >> i) & 1)
          for(int k = 0; k < 3; ++k) {
            lo[k] = fmin(lo[k], L[i].lo[k]);
            hi[k] = fmax(hi[k], L[i].hi[k]);
          }
      M.area[S] = half_area(lo, hi);
      if((S & (S - 1)) == 0) c[S] = L[__ffs(S) - 1].cost;
    }
    __syncwarp();
    for(int k = 0; k < 4; ++k) {
      const int i = SUBSET_FIRST[k] + lane;
      const int S = i < SUBSET_FIRST[k + 1] ? SUBSETS[i] : full;
      if(S < full) {
        /* each partition once: the part holding S's lowest leaf */
        const int low = S & -S, others = S ^ low;
        float bc = 3.4e38f;
        int bp = low;
        for(int Q = others;;) {
          Q = (Q - 1) & others;
          const int P = Q | low;
          const float v = c[P] + c[S ^ P];
          if(v < bc) { bc = v; bp = P; }
          if(Q == 0) break;
        }
        c[S] = C_NODE * M.area[S] + bc;
        part[S] = (uint8_t)bp;
      }
      __syncwarp();
    }
    /* The whole set: one of its partitions per lane. A lane without one must
     * not win, also where the costs of all partitions overflow: it stands for
     * the first partition, at an infinite cost. */
    {
      const int P = 2 * lane + 1;
      float v = P < full ? c[P] + c[full ^ P] : INFINITY;
      int bp = P < full ? P : 1;
      for(int o = 16; o > 0; o >>= 1) {
        const float u = __shfl_xor_sync(0xffffffffu, v, o);
        const int q = __shfl_xor_sync(0xffffffffu, bp, o);
        if(u < v || (u == v && q > bp)) { v = u; bp = q; }
      }
      if(lane == 0) {
        c[full] = C_NODE * M.area[full] + v;
        part[full] = (uint8_t)bp;
      }
      __syncwarp();
    }
    if(c[full] < cur * (1.f - 1e-5f)) {
      rebuild_treelet(nodes, A, L, nl, M.inner, c, part, M.rebuilt, lane);
      if(lane == 0 && root == 0) *depth = A.height[0];
    }
  }
  __syncwarp();
}

/* The nodes of one height, one warp per node: heights in increasing order,
 * so that a node's subtree is final when its treelet is formed. Trees of
 * MAX_LEVELS heights or more are left as they are. */
template<class R>
__global__ void __launch_bounds__(32 * TREELET_WARPS) lbvh_treelets
  (DNode<R>* nodes, const Aux A, const int32_t* level_first, const int32_t* level_nodes,
   int level, int32_t* depth)
{
  __shared__ TreeletScratch<R> scratch[TREELET_WARPS];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int maxh = level_first[MAX_LEVELS + 1];
  if(level > maxh || maxh >= MAX_LEVELS - 1) return;
  const int first = level_first[level], count = level_first[level + 1] - first;
  for(int t = blockIdx.x * TREELET_WARPS + w; t < count; t += gridDim.x * TREELET_WARPS)
    restructure(nodes, A, level_nodes[first + t], depth, scratch[w], lane);
}

/* The remaining heights, whose nodes are few, in one block of `warps` warps */
template<class R>
__device__ __forceinline__ void treelets_from
  (DNode<R>* nodes, const Aux& A, const int32_t* level_first, const int32_t* level_nodes,
   int level, int32_t* depth, TreeletScratch<R>* scratch)
{
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int maxh = level_first[MAX_LEVELS + 1];
  if(maxh >= MAX_LEVELS - 1) return;
  for(; level <= maxh; ++level) {
    const int first = level_first[level], count = level_first[level + 1] - first;
    for(int t = w; t < count; t += warps)
      restructure(nodes, A, level_nodes[first + t], depth, scratch[w], lane);
    __syncthreads();
  }
}

/* Step 5: boxes, SAH costs, heights and internal node counts, one thread
 * per leaf; flags start at zero */
template<class R>
__device__ __forceinline__ void lbvh_box(const R* box, const uint32_t* vals, int n, int j,
                                         DNode<R>* nodes, const Aux& A, uint32_t* flags,
                                         int32_t* depth)
{
  const int src = (int)vals[j];
  R lo[3], hi[3];
  for(int c = 0; c < 3; ++c) {
    lo[c] = box[6 * src + c];
    hi[c] = box[6 * src + 3 + c];
  }
  int p = A.parent[(n - 1) + j];
  int node = p >> 1, slot = p & 1, h = 0, nin = 0;
  float my_cost = C_PRIM * half_area(lo, hi);
  put_slot(nodes[node], slot, lo, hi);
  for(;;) {
    /* publish this slot (and what is known below it) before arriving */
    __threadfence();
    if(atomicAdd(&flags[node], 1u) == 0u) return;
    __threadfence();
    /* both slots are final: the sibling's box, cost and height were written
     * by the thread that arrived first, read past L1 */
    DNode<R>& N = nodes[node];
    TLeaf<R> sib;
    read_slot(N, 1 - slot, A, sib);
    for(int c = 0; c < 3; ++c) {
      lo[c] = fmin(lo[c], sib.lo[c]);
      hi[c] = fmax(hi[c], sib.hi[c]);
    }
    h = 1 + max(h, sib.height);
    nin = 1 + nin + sib.ninner;
    my_cost = C_NODE * half_area(lo, hi) + my_cost + sib.cost;
    A.cost[node] = my_cost;
    A.height[node] = h;
    A.ninner[node] = nin;
    if(node == 0) {
      *depth = h;
      return;
    }
    p = A.parent[node];
    node = p >> 1;
    slot = p & 1;
    put_slot(nodes[node], slot, lo, hi);
  }
}

/* Step 7: depth-first order of the internal nodes (slot 0 first), as the
 * host builder numbers them, so that a node's first child follows it in
 * memory: a node's index is the sum, over the path from the root, of one
 * per step plus, where the path takes slot 1, the internal nodes of the
 * slot-0 subtree it passes by */
template<class R>
__device__ __forceinline__ int lbvh_index(const DNode<R>* nodes, const int32_t* parent,
                                          const int32_t* ninner, int i)
{
  int x = 0, node = i;
  while(node != 0) {
    const int p = parent[node];
    const int par = p >> 1;
    x += 1;
    if(p & 1) {
      const DNode<R>& P = nodes[par];
      if(P.count[0] == 0) x += ninner[P.child[0]];
    }
    node = par;
  }
  return x;
}

/* With `pairs`, a node of two primitives becomes a pair in its parent, whose
 * references are listed at the node's index (its place stays, unread), as in
 * the host's tree (joins_pairs). */
template<class R>
__device__ __forceinline__ void lbvh_permute(const DNode<R>* src, DNode<R>* dst,
                                             const int32_t* newidx, uint32_t* pairs, int i)
{
  DNode<R> N = src[i];
  for(int k = 0; k < 2; ++k) {
    if(N.count[k] != 0) continue;
    const DNode<R>& C = src[N.child[k]];
    const int at = newidx[N.child[k]];
    if(pairs && C.count[0] == 1 && C.count[1] == 1) {
      pairs[2 * at] = (uint32_t)C.child[0];
      pairs[2 * at + 1] = (uint32_t)C.child[1];
      N.child[k] = PAIR_LEAF | (2 * at);
    } else {
      N.child[k] = at;
    }
  }
  dst[newidx[i]] = N;
}

/* The arguments of a build, typed: the tree is built in `work` and written
 * depth first to `nodes` */
template<class R> struct Build {
  int n;
  const R* box;
  const uint32_t* ref;
  R* cb;
  DNode<R>* work;
  DNode<R>* nodes;
  uint32_t* pairs;
  uint32_t *k0, *k1, *v0, *v1, *flags;
  int32_t *depth, *newidx, *level_first, *level_nodes;
  Aux aux;
};

template<class R>
__global__ void __launch_bounds__(SORT_THREADS) lbvh_sorted(const Build<R> B)
{
  __shared__ uint32_t wcnt[SORT_WARPS][256];
  lbvh_bounds(B.box, B.n, B.cb);
  __syncthreads();
  lbvh_morton(B.box, B.n, B.cb, B.k0, B.v0);
  __syncthreads();
  lbvh_sort(wcnt, B.k0, B.v0, B.k1, B.v1, B.n);
}
template<class R>
__global__ void lbvh_hierarchy(const Build<R> B)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= B.n - 1) return;
  B.flags[i] = 0;
  lbvh_node(B.k0, B.v0, B.ref, B.n, i, B.work, B.aux.parent);
}
template<class R>
__global__ void lbvh_boxes(const Build<R> B)
{
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if(j < B.n) lbvh_box(B.box, B.v0, B.n, j, B.work, B.aux, B.flags, B.depth);
}
template<class R>
__global__ void __launch_bounds__(SORT_THREADS) lbvh_heights(const Build<R> B)
{
  lbvh_levels(B.aux.height, B.n - 1, B.level_first, B.level_nodes,
              B.level_first + MAX_LEVELS + 1);
}
template<class R>
__global__ void __launch_bounds__(SORT_THREADS) lbvh_treelets_top(const Build<R> B, int level)
{
  __shared__ TreeletScratch<R> scratch[SORT_WARPS];
  treelets_from(B.work, B.aux, B.level_first, B.level_nodes, level, B.depth, scratch);
}
template<class R>
__global__ void lbvh_order(const Build<R> B)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i < B.n - 1) B.newidx[i] = lbvh_index(B.work, B.aux.parent, B.aux.ninner, i);
}
template<class R>
__global__ void lbvh_write(const Build<R> B)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i < B.n - 1) lbvh_permute(B.work, B.nodes, B.newidx, B.pairs, i);
}

/* Every step in one block, for scenes so small that the launches and the gaps
 * between them are the build: four triangles take 112 us of plan creation
 * with a launch per step, and 65 so; the block keeps up with the
 * launches up to a few hundred primitives */
constexpr int SMALL_BUILD = 512;
template<class R>
__global__ void __launch_bounds__(SORT_THREADS) lbvh_small(const Build<R> B, int optimize)
{
  /* the sort's counts, then the treelets */
  __shared__ union Shared {
    uint32_t wcnt[SORT_WARPS][256];
    TreeletScratch<R> treelets[SORT_WARPS];
  } shared;
  const int tid = threadIdx.x, n = B.n;
  lbvh_bounds(B.box, n, B.cb);
  __syncthreads();
  lbvh_morton(B.box, n, B.cb, B.k0, B.v0);
  __syncthreads();
  lbvh_sort(shared.wcnt, B.k0, B.v0, B.k1, B.v1, n);
  __syncthreads();
  if(tid < n - 1) {
    B.flags[tid] = 0;
    lbvh_node(B.k0, B.v0, B.ref, n, tid, B.work, B.aux.parent);
  }
  __syncthreads();
  if(tid < n) lbvh_box(B.box, B.v0, n, tid, B.work, B.aux, B.flags, B.depth);
  __syncthreads();
  if(optimize) {
    lbvh_levels(B.aux.height, n - 1, B.level_first, B.level_nodes,
                B.level_first + MAX_LEVELS + 1);
    __syncthreads();
    treelets_from(B.work, B.aux, B.level_first, B.level_nodes, 2, B.depth,
                  shared.treelets);
    __syncthreads();
  }
  if(tid < n - 1) B.newidx[tid] = lbvh_index(B.work, B.aux.parent, B.aux.ninner, tid);
  __syncthreads();
  if(tid < n - 1) lbvh_permute(B.work, B.nodes, B.newidx, B.pairs, tid);
}

/* Heights whose nodes get a launch of their own, lowest first; a few dozen
 * nodes are left above them (3152 primitives have 664, 368, 240, 196 and 116
 * nodes of heights 2 to 6, and 64 of height 7). The counts stay on the
 * device: each launch is sized by a bound and strides over what there is. */
static int wide_levels(int n)
{
  int last = 6;
  for(long long m = 3000; m < n; m *= 2) last += (last & 1) ? 2 : 1;
  return std::min(last, MAX_LEVELS - 1);
}

template<class R>
int launch_lbvh(const LbvhArgs& A, void* stream)
{
  const cudaStream_t s = (cudaStream_t)stream;
  const int n = A.n;
  if(n < 2) return (int)cudaErrorInvalidValue;
  Build<R> B;
  B.n = n;
  B.box = (const R*)A.box;
  B.ref = A.ref;
  B.cb = (R*)A.cbounds;
  B.work = (DNode<R>*)A.tmp_nodes;
  B.nodes = (DNode<R>*)A.nodes;
  B.pairs = A.pairs;
  B.k0 = A.keys;
  B.k1 = A.keys + n;
  B.v0 = A.vals;
  B.v1 = A.vals + n;
  B.flags = A.flags;
  B.depth = A.depth;
  B.newidx = A.newidx;
  B.level_first = A.level_first;
  B.level_nodes = A.level_nodes;
  B.aux = {A.cost, A.height, A.ninner, A.parent};
  const bool optimize = A.optimize && n >= 3;
  if(n <= SMALL_BUILD) {
    lbvh_small<R><<<1, SORT_THREADS, 0, s>>>(B, optimize ? 1 : 0);
    return (int)cudaGetLastError();
  }
  const unsigned g = (unsigned)((n + 255) / 256);
  lbvh_sorted<R><<<1, SORT_THREADS, 0, s>>>(B);
  lbvh_hierarchy<R><<<g, 256, 0, s>>>(B);
  lbvh_boxes<R><<<g, 256, 0, s>>>(B);
  if(optimize) {
    lbvh_heights<R><<<1, SORT_THREADS, 0, s>>>(B);
    const int wide = wide_levels(n);
    for(int h = 2; h <= wide; ++h) {
      const unsigned blocks = (unsigned)std::min(n / (2 * h * TREELET_WARPS) + 1, 148 * 8);
      lbvh_treelets<R><<<blocks, 32 * TREELET_WARPS, 0, s>>>(B.work, B.aux, B.level_first,
                                                             B.level_nodes, h, B.depth);
    }
    lbvh_treelets_top<R><<<1, SORT_THREADS, 0, s>>>(B, wide + 1);
  }
  lbvh_order<R><<<g, 256, 0, s>>>(B);
  lbvh_write<R><<<g, 256, 0, s>>>(B);
  return (int)cudaGetLastError();
}

} /* namespace */

size_t lbvh_scratch_bytes(int n)
{
  const size_t m = n > 0 ? (size_t)n : 0;
  /* centroid bounds (6 doubles), depth (one int, padded), a copy of the
   * nodes (sized for FP64), keys and vals (2n each), parent (2n), flags,
   * heights, costs, internal node counts, new indices and nodes by level (n
   * each), level offsets and the largest height */
  return 6 * sizeof(double) + 16 + sizeof(DNode<double>) * m
    + sizeof(uint32_t) * (2 * m + 2 * m + 2 * m + 6 * m) + sizeof(int32_t) * (MAX_LEVELS + 2);
}

void lbvh_bind_scratch(LbvhArgs& A, void* scratch)
{
  const size_t m = A.n > 0 ? (size_t)A.n : 0;
  /* the doubles first, so that they are 8-byte aligned */
  unsigned char* p = (unsigned char*)scratch;
  A.cbounds = p;
  p += 6 * sizeof(double);
  A.depth = (int32_t*)p;
  p += 16;
  A.tmp_nodes = p;
  p += sizeof(DNode<double>) * m;
  A.keys = (uint32_t*)p;
  p += sizeof(uint32_t) * 2 * m;
  A.vals = (uint32_t*)p;
  p += sizeof(uint32_t) * 2 * m;
  A.parent = (int32_t*)p;
  p += sizeof(int32_t) * 2 * m;
  A.flags = (uint32_t*)p;
  p += sizeof(uint32_t) * m;
  A.height = (int32_t*)p;
  p += sizeof(int32_t) * m;
  A.cost = (float*)p;
  p += sizeof(float) * m;
  A.ninner = (int32_t*)p;
  p += sizeof(int32_t) * m;
  A.newidx = (int32_t*)p;
  p += sizeof(int32_t) * m;
  A.level_nodes = (int32_t*)p;
  p += sizeof(int32_t) * m;
  A.level_first = (int32_t*)p;
}

int launch_lbvh_f32(const LbvhArgs& A, void* stream) { return launch_lbvh<float>(A, stream); }
int launch_lbvh_f64(const LbvhArgs& A, void* stream) { return launch_lbvh<double>(A, stream); }

} /* namespace ssolb */
