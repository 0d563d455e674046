// chainmesh.cu -- the chain-mesh cell sort on the device.
//
// Reference: chainmesh_create -> sort (src/chainmesh.cpp:139-213) ->
// particles_sort (src/particles.cpp:414-444).  The reference bisects the
// chain box recursively (split dim = the LAST dim with span > 1, mid =
// begin + span/2) and partitions the particle range in place at each node
// with a two-pointer (Hoare) pass on x[dim] >= fixed32(mid * (1.0/C)).
//
// Device design (no recursion, no per-node launches):
//  1. keys:   each particle's chain cell from the reference's own split
//             thresholds thr[m] = fixed32(m * (1.0/C)), so "x < thr[mid]" and
//             "cell < mid" are the same predicate bit for bit;
//  2. counts: per-cell histogram (warp-aggregated atomics) + exclusive scan
//             gives the cell offsets, which the recursion leaves in
//             (z, y, x)-lexicographic order;
//  3. PARITY order: every node of the recursion tree owns a contiguous
//             position range that the offsets already determine, so all nodes
//             of one depth are partitioned together.  A two-pointer pass swaps
//             the i-th misplaced element of the left part (ascending) with the
//             i-th misplaced element of the right part (descending): one
//             level is a flag scan that restarts at every node and writes the
//             misplaced positions, and a pairwise swap.  Nodes that fit a
//             block's shared memory are finished there, all their remaining
//             levels in one launch.
//     FAST order: a stable counting sort (input order inside each cell).
//  4. gather: the accumulated permutation is applied once to x, y, z, vx, vy,
//             vz and rung, and positions are packed as int4 for the PP kernel.
#include "tpm_internal.cuh"

#include <algorithm>
#include <cstring>

namespace tpm {
namespace {

constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kSwapBlock = 1024;  // positions per block of a swap pass
static_assert(kScanTile % kSwapBlock == 0 && kSwapBlock % kScanItems == 0, "swap blocks begin at a scan thread's first position");
// Positions and cells of a unit that one block sorts in shared memory
constexpr int kUnit = 8192;
constexpr int kUnitCells = 2048;
constexpr int64_t kRecordsFrom = 1 << 22;  // particles from which k_gather may read records
constexpr int kFinishThreads = 1024;
constexpr int kFinishPer = kUnit / kFinishThreads;  // positions per thread
static_assert(kUnit <= 8192 && kUnitCells <= 65536, "13-bit positions in a node word, 16-bit cells");
constexpr size_t kFinishSmem = 6 * (size_t)kUnit + 4 * (2 * (kUnit / 32)) + 8 * kUnitCells + 2 * (kUnitCells + 2);
static_assert(kScanTile == kScanTileElems, "scan tiles must match the status and block-sum arrays");

// Cell coordinate of raw position r along one axis: the largest m with
// r >= thr[m] (thr[0] = 0).  The integer estimate floor(r*C/2^32) is within
// one of it; the threshold table settles the boundary exactly.
__device__ __forceinline__ int cell_coord(uint32_t r, int C, const uint32_t* __restrict__ thr) {
  int c = (int)(((uint64_t)r * (uint64_t)C) >> 32);
  if (c + 1 < C && r >= __ldg(thr + c + 1)) c++;
  else if (c > 0 && r < __ldg(thr + c)) c--;
  return c;
}

__global__ void k_cell_keys(int64_t n, const uint32_t* __restrict__ x, const uint32_t* __restrict__ y,
                            const uint32_t* __restrict__ z, const uint32_t* __restrict__ thr, int C,
                            uint32_t* __restrict__ key, int32_t* __restrict__ idx,
                            int32_t* __restrict__ count) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool live = i < n;
  uint32_t k = 0xffffffffu;
  if (live) {
    const int cx = cell_coord(x[i], C, thr);
    const int cy = cell_coord(y[i], C, thr);
    const int cz = cell_coord(z[i], C, thr);
    k = ((uint32_t)cz * (uint32_t)C + (uint32_t)cy) * (uint32_t)C + (uint32_t)cx;
    key[i] = k;
    idx[i] = (int32_t)i;
  }
  // warp-aggregated histogram: one atomic per distinct key in the warp
  const unsigned live_mask = __ballot_sync(0xffffffffu, live);
  if (live) {
    const unsigned peers = __match_any_sync(live_mask, k);
    const int leader = __ffs(peers) - 1;
    if ((int)(threadIdx.x & 31) == leader) atomicAdd(count + k, __popc(peers));
  }
}

// Block-wide exclusive scan of one int per thread (kScanThreads threads).
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_tot, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < (kScanThreads / 32) ? warp_tot[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < (kScanThreads / 32)) warp_tot[lane] = wi - w;
    if (lane == (kScanThreads / 32) - 1) *total = wi;
  }
  __syncthreads();
  const int r = warp_tot[warp] + incl - v;
  return r;
}

// Exclusive scan of in[0..n) into out[0..n], out[n] = total, in ONE block
// (used for per-block sums and cell counts of modest size).
__global__ void __launch_bounds__(kScanThreads) k_scan_single(const int32_t* __restrict__ in, int64_t n,
                                                              int32_t* __restrict__ out) {
  __shared__ int warp_tot[32];
  __shared__ int total;
  int carry = 0;
  for (int64_t base = 0; base < n; base += kScanTile) {
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      const int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
      v[k] = i < n ? in[i] : 0;
      s += v[k];
    }
    int off = block_exclusive_scan(s, warp_tot, &total) + carry;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      const int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
      if (i < n) out[i] = off;
      off += v[k];
    }
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry;
}

// Multi-block exclusive scan, pass 1: per-block totals.
__global__ void __launch_bounds__(kScanThreads) k_scan_blocksum(const int32_t* __restrict__ in, int64_t n,
                                                                int32_t* __restrict__ bsum) {
  __shared__ int warp_tot[32];
  __shared__ int total;
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
    s += i < n ? in[i] : 0;
  }
  block_exclusive_scan(s, warp_tot, &total);
  if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// pass 3: block-local exclusive scan plus the scanned block offset.
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const int32_t* __restrict__ in, int64_t n,
                                                             const int32_t* __restrict__ boff,
                                                             int32_t* __restrict__ out) {
  __shared__ int warp_tot[32];
  __shared__ int total;
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
    v[k] = i < n ? in[i] : 0;
    s += v[k];
  }
  int off = block_exclusive_scan(s, warp_tot, &total) + boff[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
    if (i < n) out[i] = off;
    off += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = boff[gridDim.x];
}

// cellof[p] = the cell whose final range holds position p (one warp per cell).
__global__ void k_cellof(int64_t ncell, const int32_t* __restrict__ begin, int32_t* __restrict__ cellof) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= ncell) return;
  const int32_t b = begin[w], e = begin[w + 1];
  for (int32_t p = b + lane; p < e; p += 32) cellof[p] = (int32_t)w;
}

// One level of the partition: dimension dim (2 = z, 1 = y, 0 = x; all levels
// of z come first, then y, then x, and nodes of one tree level are
// independent of each other) at depth `level` of its 1-D bisection.  A unit
// is a node of dimension udim at depth ulevel: k_finish sorts the units of
// at most kUnit positions in shared memory, so the levels from there on
// (big_only) take the positions of larger units only, and nothing at all
// unless *nbig says that there are such units.
struct LevelArgs {
  int64_t n;
  int C;
  int dim, level;
  int udim, ulevel;
  int big_only;
  const int* __restrict__ nbig;
  const int32_t* __restrict__ cellof;
  const uint32_t* __restrict__ key;
  const int32_t* __restrict__ begin;
  const TreeNode* __restrict__ tree;
  const int* __restrict__ depth;
};

// A recursion node: its position range [b, e), the split point pm (first
// position of the right child) and the first cell of the right child.  The
// keys of its elements lie in its own cell range, so an element belongs to the
// left child exactly when its key is below that cell (its coordinate along
// the split dimension is below mid, i.e. x < xmid).
struct Node {
  int32_t b, pm, e;
  uint32_t mid;
  bool live;
};

// The interval of coordinate c at depth l of the 1-D bisection (lo, mid, hi);
// mid = hi where the bisection has ended.
__device__ __forceinline__ TreeNode interval(const TreeNode* __restrict__ tree, const int* __restrict__ depth, int c, int l) {
  if (l < __ldg(depth + c)) return tree[c * kMaxTreeDepth + l];
  return TreeNode{c, c + 1, c + 1, 0};
}

// Positions of the cells [lo, hi) of dimension dim's coordinate around cell
// (cx, cy, cz): dimensions below dim whole, those above fixed.
__device__ __forceinline__ int64_t cell_at(int dim, int64_t C, int cy, int cz, int c) {
  return dim == 2 ? c * C * C : dim == 1 ? (cz * C + c) * C : (cz * C + cy) * C + c;
}

// The node that owns the positions of final cell `cell` at this level; not
// live when the cell's bisection has ended or the level leaves its unit out.
__device__ __forceinline__ Node node_of_cell(const LevelArgs& a, int cell) {
  Node nd;
  const int C = a.C;
  const int cx = cell % C, cy = (cell / C) % C, cz = cell / (C * C);
  const TreeNode t = interval(a.tree, a.depth, a.dim == 2 ? cz : a.dim == 1 ? cy : cx, a.level);
  const int64_t m = cell_at(a.dim, C, cy, cz, t.mid);
  nd.b = __ldg(a.begin + cell_at(a.dim, C, cy, cz, t.lo));
  nd.pm = __ldg(a.begin + m);
  nd.e = __ldg(a.begin + cell_at(a.dim, C, cy, cz, t.hi));
  nd.mid = (uint32_t)m;
  nd.live = t.mid < t.hi;
  if (a.big_only) {
    const TreeNode u = interval(a.tree, a.depth, a.udim == 2 ? cz : a.udim == 1 ? cy : cx, a.ulevel);
    nd.live = nd.live && __ldg(a.begin + cell_at(a.udim, C, cy, cz, u.hi)) -
                                 __ldg(a.begin + cell_at(a.udim, C, cy, cz, u.lo)) > kUnit;
  }
  return nd;
}

// Four consecutive int32 entries from position p (a multiple of 4, so the
// 16-byte load is aligned) when all four are below n; else one by one.
__device__ __forceinline__ int4 load4(const int32_t* __restrict__ a, unsigned p, unsigned n) {
  if (p + 4 <= n) return *reinterpret_cast<const int4*>(a + p);
  int4 r = make_int4(0, 0, 0, 0);
  if (p < n) r.x = a[p];
  if (p + 1 < n) r.y = a[p + 1];
  if (p + 2 < n) r.z = a[p + 2];
  return r;
}

// Decoupled look-back scan status word: stamp (30 bits) | flag (2 bits) | value (32 bits).
constexpr unsigned long long kFlagAgg = 1ull, kFlagIncl = 2ull;
__device__ __forceinline__ unsigned long long pack_status(unsigned stamp, unsigned long long flag, int value) {
  return ((unsigned long long)stamp << 34) | (flag << 32) | (unsigned long long)(unsigned)value;
}

// One partition level, part 1: the left-child flags of every position,
// counted from the start of its node, in a single pass, and the misplaced
// positions: the k-th of the left part (ascending) goes to slot[b + k], the
// k-th of the right part from its end to slot[pm + k], their number to
// misplaced[b].  The count restarts at every node, so a tile's predecessors
// matter only to the node that runs into it (chained scan with decoupled
// look-back; tiles are taken in launch order through an atomic counter, so
// every predecessor a tile waits on is already running).  The look-back is
// done by one warp, 32 predecessor tiles at a time; its polls are bounded: at
// the limit the tile records kErrTimeout, sets *gave_up and uses what it has
// summed.  Counts and slots are then wrong (though in range), so no level
// swaps from there on and the units keep their order: the result is still a
// permutation of the particles.
//
// Bound by latency and issue (36 us per level of 7.65e6 particles, 31 MB read):
// 4 bytes of key read per position, 4 written per misplaced one.  Nodes come
// from the tile's first position; only positions outside that node look
// their cell up.  A level's scan and swap take 63 us; as a flag scan with a
// prefix array, a slot pass and a swap pass they took 145 us.
__global__ void __launch_bounds__(kScanThreads, 4)
    k_level_scan(LevelArgs a, unsigned stamp, int* __restrict__ counter, unsigned long long* __restrict__ status,
                 int32_t* __restrict__ slot, int32_t* __restrict__ misplaced, int4* __restrict__ heads, int polls,
                 int* __restrict__ gave_up, int* __restrict__ err) {
  __shared__ int warp_tot[32];
  __shared__ int total;
  __shared__ unsigned tile_s;
  __shared__ int carry_s;
  __shared__ int before[kScanThreads + 1];            // flags before each thread's positions
  __shared__ unsigned char bits[kScanThreads];        // its kScanItems flags
  static_assert(kScanItems == 8, "one byte of flags per thread");
  if (a.big_only && *a.nbig == 0) return;
  const unsigned n = (unsigned)a.n, tiles = (n + kScanTile - 1) / kScanTile;
  while (true) {
    if (threadIdx.x == 0) tile_s = (unsigned)atomicAdd(counter, 1);
    __syncthreads();
    const unsigned tile = tile_s;
    if (tile >= tiles) return;
    const unsigned base = tile * kScanTile, first = base + threadIdx.x * kScanItems;
    const unsigned end = min(base + kScanTile, n);
    int4 keys[kScanItems / 4];
#pragma unroll
    for (int k = 0; k < kScanItems; k += 4) keys[k / 4] = load4(reinterpret_cast<const int32_t*>(a.key), first + k, n);
    const Node head = node_of_cell(a, __ldg(a.cellof + base));
    Node nd = head;
    unsigned m = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k += 4) {
      const int4 q = keys[k / 4];
      const uint32_t ky[4] = {(uint32_t)q.x, (uint32_t)q.y, (uint32_t)q.z, (uint32_t)q.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const unsigned p = first + k + i;
        if (p >= n) continue;
        if (p >= (unsigned)nd.e) nd = node_of_cell(a, __ldg(a.cellof + p));
        if (nd.live && ky[i] < nd.mid) m |= 1u << (k + i);
      }
    }
    const int off = block_exclusive_scan(__popc(m), warp_tot, &total);
    before[threadIdx.x] = off;
    bits[threadIdx.x] = (unsigned char)m;
    if (threadIdx.x == kScanThreads - 1) before[kScanThreads] = total;
    __syncthreads();
    // flags of the tile before position base + i
    auto count = [&](unsigned i) {
      return i >= kScanTile ? before[kScanThreads]
                            : before[i / kScanItems] + __popc(bits[i / kScanItems] & ((1u << (i % kScanItems)) - 1u));
    };
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      // The count to hand on: from the start of the node of the tile's last
      // position.  It is complete when that node starts in this tile.
      const unsigned last = end - 1;
      const Node tail = last < (unsigned)head.e ? head : node_of_cell(a, __ldg(a.cellof + last));
      const bool whole = (unsigned)tail.b < base;
      const int mine = total - (whole ? 0 : count((unsigned)tail.b - base));
      if (lane == 0) atomicExch(status + tile, pack_status(stamp, whole ? kFlagAgg : kFlagIncl, mine));
      int carry = 0;
      if ((unsigned)head.b < base) {
        // warp-parallel look-back: lane l reads the status of tile (top - l);
        // once all 32 are published, the values up to the closest complete one
        // are summed, else the window moves 32 tiles back
        int top = (int)tile - 1;
        int spins = 0;
        bool late = polls == 0;
        while (!late) {
          const int j = top - lane;
          unsigned long long f = kFlagIncl;  // before tile 0: a complete zero
          int v = 0;
          if (j >= 0) {
            const unsigned long long w = *reinterpret_cast<volatile unsigned long long*>(status + j);
            f = (unsigned)(w >> 34) == stamp ? (w >> 32) & 3ull : 0ull;
            v = (int)(unsigned)(w & 0xffffffffull);
          }
          if (__any_sync(0xffffffffu, f == 0)) {
            late = ++spins > polls;
            continue;
          }
          const unsigned incl = __ballot_sync(0xffffffffu, f == kFlagIncl);
          const int nearest = incl ? __ffs(incl) - 1 : 32;
          int sum = lane <= nearest ? v : 0;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
          carry += sum;
          if (incl) break;
          top -= 32;
        }
        if (late && lane == 0) {
          atomicExch(gave_up, 1);
          atomicOr(err, kErrTimeout);
        }
        if (whole && lane == 0) atomicExch(status + tile, pack_status(stamp, kFlagIncl, carry + mine));
      }
      if (lane == 0) carry_s = carry;
    }
    __syncthreads();
    nd = head;
    // flags of the tile before the node, less those of the node before the tile
    int from = (unsigned)head.b < base ? -carry_s : count((unsigned)head.b - base);
    int run = off;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      const unsigned p = first + k;
      if (p >= n) break;
      if (p >= (unsigned)nd.e) {
        nd = node_of_cell(a, __ldg(a.cellof + p));
        from = (unsigned)nd.b < base ? -carry_s : count((unsigned)nd.b - base);
      }
      // the swap's blocks begin at these positions
      if (k == 0 && p % kSwapBlock == 0) heads[p / kSwapBlock] = make_int4(nd.b, nd.pm, nd.live ? nd.e : -nd.e, 0);
      const int flag = (m >> k) & 1;
      const int in_node = run - from;  // flags in [b, p)
      run += flag;
      if (!nd.live) continue;
      // the range checks only matter after a look-back gave up
      if (p < (unsigned)nd.pm) {
        const int wrong = (int)(p - nd.b) - in_node;
        if (!flag && wrong >= 0 && nd.b + wrong < nd.pm) slot[nd.b + wrong] = (int32_t)p;
        if (p == (unsigned)nd.pm - 1) misplaced[nd.b] = wrong + (flag ? 0 : 1);
      } else if (flag) {
        const int back = (nd.pm - nd.b) - in_node - 1;  // flags in (p, e)
        if (back >= 0 && nd.pm + back < nd.e) slot[nd.pm + back] = (int32_t)p;
      }
    }
    if (tiles <= gridDim.x) return;  // a tile for every block: no other ticket
    __syncthreads();                 // the tile's shared values are read before the next one's
  }
}

// Part 2: the k-th misplaced element of the left part swaps with the k-th of
// the right part from its end.  A block takes kSwapBlock positions as slots
// (the slots of a node are its first misplaced[b] positions); its first
// node's range comes from the scan, which saves the four dependent loads of a
// lookup.
__global__ void __launch_bounds__(256) k_level_swap(LevelArgs a, const int32_t* __restrict__ misplaced,
                                                    const int32_t* __restrict__ slot, const int4* __restrict__ heads,
                                                    const int* __restrict__ gave_up, uint32_t* __restrict__ key,
                                                    int32_t* __restrict__ idx) {
  if (a.big_only && *a.nbig == 0) return;
  const int none = __ldg(gave_up);
  const unsigned n = (unsigned)a.n;
  for (unsigned blk = blockIdx.x; blk < (n + kSwapBlock - 1) / kSwapBlock; blk += gridDim.x) {
    const int4 h = __ldg(heads + blk);
    Node nd{h.x, h.y, h.z < 0 ? -h.z : h.z, 0, h.z > 0};
    int32_t wrong = -1;  // misplaced[nd.b], read once it is needed
#pragma unroll
    for (int k = 0; k < kSwapBlock / 256; k++) {
      const unsigned p = blk * kSwapBlock + k * 256 + threadIdx.x;
      if (p >= n) break;
      if (p >= (unsigned)nd.e) {
        nd = node_of_cell(a, __ldg(a.cellof + p));
        wrong = -1;
      }
      if (!nd.live || p >= (unsigned)nd.pm) continue;
      if (wrong < 0) wrong = __ldg(misplaced + nd.b);
      const int32_t i = (int32_t)(p - nd.b);
      if (i >= wrong) continue;
      const int32_t u = __ldg(slot + p), v = __ldg(slot + nd.pm + i);
      // no swap after a give-up; tested here, with the slots, and not before
      // their loads (the swaps of 8e6 particles: 356 against 402 us)
      if ((unsigned)u >= n || (unsigned)v >= n || none) continue;
      const uint32_t ku = key[u], kv = key[v];
      const int32_t iu = idx[u], iv = idx[v];
      key[u] = kv;
      key[v] = ku;
      idx[u] = iv;
      idx[v] = iu;
    }
  }
}

// The units of a partition: the 1-D bisection's intervals of dimension udim at
// depth ulevel (first[i] .. first[i + 1] in `cuts`), for every combination of
// the dimensions above it.
struct UnitArgs {
  int C;
  int udim, ulevel;
  int cuts_n;                      // intervals
  const int* __restrict__ cuts;    // their first coordinates, cuts_n + 1 entries
  const int32_t* __restrict__ begin;
  const TreeNode* __restrict__ tree;
  const int* __restrict__ depth;
  int max_depth;
  const uint32_t* __restrict__ key;
  const int32_t* __restrict__ idx;
  int32_t* __restrict__ out;
  int* __restrict__ nbig;
  int* __restrict__ njump;
  const int* __restrict__ gave_up;
};

__device__ __forceinline__ void unit_cells(const UnitArgs& a, int u, int64_t& c0, int64_t& c1) {
  const int64_t above = u / a.cuts_n;  // cz for y, cz * C + cy for x
  const int i = u - (int)above * a.cuts_n;
  const int64_t C = a.C;
  const int64_t span = a.udim == 2 ? C * C : a.udim == 1 ? C : 1;
  c0 = above * C * span + a.cuts[i] * span;
  c1 = above * C * span + a.cuts[i + 1] * span;
}

// Counts the units that k_finish leaves to the level kernels.
__global__ void k_big_units(UnitArgs a, int units) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= units) return;
  int64_t c0, c1;
  unit_cells(a, u, c0, c1);
  if (__ldg(a.begin + c1) - __ldg(a.begin + c0) > kUnit) atomicAdd(a.nbig, 1);
}

// All remaining levels of one unit, in shared memory; out = the unit's
// original particle indices in their final order.  An element is one word,
// its cell relative to the unit's first and its position at the start; its
// cell also names the node that it is in at each level, since every level
// leaves it inside its node.  Per level: the flags as one ballot word per 32
// positions with a scan of the words' counts, the misplaced positions of the
// right parts as a slot list, and the swaps (the same pairing as the level
// kernels').  Four barriers per level against two launches and 30 bytes of
// HBM traffic per position.  Bound by instruction issue (161 per element and
// level when each element looked its node up in the bisection's intervals), so
// the nodes of a level come from a table by cell, which the warps that have no
// part in the scan fill for the next level: 7 levels of 7.65e6 particles 230 us
// (370 before; the level kernels take 65 us each).
__global__ void __launch_bounds__(kFinishThreads, 2) k_finish(UnitArgs a) {
  extern __shared__ __align__(16) unsigned char fin[];
  uint32_t* el = reinterpret_cast<uint32_t*>(fin);                          // kUnit elements
  uint16_t* slot = reinterpret_cast<uint16_t*>(el + kUnit);                 // kUnit
  uint32_t* word = reinterpret_cast<uint32_t*>(slot + kUnit);               // kUnit / 32 flag words
  uint32_t* pre = word + kUnit / 32;                                        // flags before each word
  uint32_t* tab = pre + kUnit / 32;                                         // nodes by cell, this level
  uint32_t* tab2 = tab + kUnitCells;                                        // and the next
  uint16_t* off = reinterpret_cast<uint16_t*>(tab2 + kUnitCells);           // cell offsets, kUnitCells + 1
  __shared__ int jumps;
  const int none = __ldg(a.gave_up);
  int64_t c0, c1;
  unit_cells(a, blockIdx.x, c0, c1);
  const int32_t b0 = __ldg(a.begin + c0);
  const int n = __ldg(a.begin + c1) - b0;
  const int cells = (int)(c1 - c0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Left as it is: a unit that the level kernels sort, and every unit once a
  // look-back gave up (its elements may then belong to any cell, and the tables
  // below are read by the element's cell).
  if (n > kUnit || none) {
    for (int i = tid; i < n; i += kFinishThreads) a.out[b0 + i] = a.idx[b0 + i];
    return;
  }
  if (n == 0) return;
  const int C = a.C;
  const int first = a.cuts[blockIdx.x % a.cuts_n];  // the unit's first coordinate of dimension udim
  // The node of each cell at a level: first position (bits 0-12), live (14),
  // the cell is the left child's (15), first position of the right child
  // (16-29).
  auto fill = [&](uint32_t* t, int dim, int level, int from, int step) {
    const int per = dim == 2 ? C * C : dim == 1 ? C : 1;  // cells per coordinate
    for (int cell = from; cell < cells; cell += step) {
      int c = cell / per, base;  // base: the cell of coordinate 0
      if (dim == a.udim) {
        c += first;
        base = -first * per;
      } else {
        base = c / C * C * per;
        c %= C;
      }
      const TreeNode g = interval(a.tree, a.depth, c, level);
      const int mid = base + g.mid * per;
      t[cell] = off[base + g.lo * per] | (g.mid < g.hi ? 1u << 14 : 0u) | (cell < mid ? 1u << 15 : 0u) |
                ((uint32_t)off[mid] << 16);
    }
  };
  if (tid == 0) jumps = 0;
  for (int i = tid; i <= cells; i += kFinishThreads) off[i] = (uint16_t)(__ldg(a.begin + c0 + i) - b0);
  for (int i = tid; i < n; i += kFinishThreads)
    el[i] = ((__ldg(a.key + b0 + i) - (uint32_t)c0) << 16) | (uint32_t)i;
  __syncthreads();
  fill(tab, a.udim, a.ulevel, tid, kFinishThreads);
  __syncthreads();
  const int words = (n + 31) >> 5;
  auto flags_before = [&](int p) {  // p < n
    return (int)pre[p >> 5] + __popc(word[p >> 5] & ((1u << (p & 31)) - 1u));
  };
  for (int dim = a.udim, level = a.ulevel; dim >= 0;) {
    const int dim2 = level + 1 < a.max_depth ? dim : dim - 1, level2 = level + 1 < a.max_depth ? level + 1 : 0;
    // Each thread keeps its elements and, where one is misplaced, its node in
    // registers through the level.
    uint32_t e[kFinishPer], node[kFinishPer];
#pragma unroll
    for (int k = 0; k < kFinishPer; k++) {
      const int p = k * kFinishThreads + tid;
      node[k] = 0;
      if (k * kFinishThreads + (tid & ~31) >= n) continue;  // whole warps
      uint32_t t = 0;
      if (p < n) {
        e[k] = el[p];
        t = tab[e[k] >> 16];
        const bool right = p >= (int)(t >> 16);
        if ((t >> 14 & 1) && right == (bool)(t >> 15 & 1)) node[k] = t;
      }
      const unsigned m = __ballot_sync(0xffffffffu, (t >> 14 & 3) == 3);
      if (lane == 0) word[k * (kFinishThreads / 32) + warp] = m;
    }
    __syncthreads();
    if (warp == 0) {
      // flags before each word: kUnit / 1024 consecutive words per lane
      constexpr int kW = kUnit / 1024;
      uint32_t w[kW];
      int sum = 0;
#pragma unroll
      for (int i = 0; i < kW; i++) {
        w[i] = lane * kW + i < words ? __popc(word[lane * kW + i]) : 0;
        sum += w[i];
      }
      int incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      int run = incl - sum;
#pragma unroll
      for (int i = 0; i < kW; i++) {
        pre[lane * kW + i] = run;
        run += w[i];
      }
    } else if (dim2 >= 0) {
      fill(tab2, dim2, level2, tid - 32, kFinishThreads - 32);
    }
    __syncthreads();
    // misplaced elements of the right parts: the k-th from its node's end to
    // slot[pm + k]
#pragma unroll
    for (int k = 0; k < kFinishPer; k++) {
      if (!(node[k] >> 15 & 1)) continue;
      const int p = k * kFinishThreads + tid, b = (int)(node[k] & 0x1fffu), pm = (int)(node[k] >> 16);
      slot[pm + (pm - b) - (flags_before(p) - flags_before(b)) - 1] = (uint16_t)p;
    }
    __syncthreads();
    // the k-th misplaced element of a left part swaps with slot[pm + k]
#pragma unroll
    for (int k = 0; k < kFinishPer; k++) {
      if ((node[k] >> 14 & 3) != 1) continue;
      const int p = k * kFinishThreads + tid, b = (int)(node[k] & 0x1fffu), pm = (int)(node[k] >> 16);
      const int q = slot[pm + (p - b) - (flags_before(p) - flags_before(b))];
      el[p] = el[q];
      el[q] = e[k];
    }
    __syncthreads();
    uint32_t* t = tab;
    tab = tab2;
    tab2 = t;
    dim = dim2;
    level = level2;
  }
  // the final order; a jump: a source outside the previous one's 8 particles
  int mine = 0;
  for (int p0 = 0; p0 < n; p0 += kFinishThreads) {
    const int p = p0 + tid;
    if (p0 + (tid & ~31) >= n) break;
    const int32_t v = p < n ? __ldg(a.idx + b0 + (el[p] & 0xffffu)) : 0;
    const int32_t u = __shfl_up_sync(0xffffffffu, v, 1);
    if (p < n) {
      a.out[b0 + p] = v;
      mine += lane == 0 || (u >> 3) != (v >> 3);
    }
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0) atomicAdd(&jumps, mine);
  __syncthreads();
  if (tid == 0) atomicAdd(a.njump, jumps);
}

// FAST order: stable counting sort.  rank-in-cell of particle i = number of
// earlier particles with the same key; computed by a scatter with atomics
// followed by a per-cell sort of the original indices.
__global__ void k_fast_scatter(int64_t n, const uint32_t* __restrict__ key, const int32_t* __restrict__ begin,
                               int32_t* __restrict__ fill, int32_t* __restrict__ idx_out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t k = key[i];
  const int32_t pos = begin[k] + atomicAdd(fill + k, 1);
  idx_out[pos] = (int32_t)i;
}

// One warp per cell: insertion-merge of the cell's original indices into
// ascending order (cells are small; large cells fall back to a shared-memory
// odd-even transposition loop with a bounded trip count).
__global__ void k_fast_cellsort(int64_t ncell, const int32_t* __restrict__ begin, int32_t* __restrict__ idx) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= ncell) return;
  const int32_t b = begin[w], e = begin[w + 1];
  const int32_t len = e - b;
  // odd-even transposition sort: len phases, each lane handles pairs
  for (int32_t phase = 0; phase < len; phase++) {
    for (int32_t j = b + (phase & 1) + 2 * lane; j + 1 < e; j += 64) {
      const int32_t u = idx[j], v = idx[j + 1];
      if (u > v) {
        idx[j] = v;
        idx[j + 1] = u;
      }
    }
    __syncwarp();
  }
}

// Particles as two 16-byte records each, for k_gather: (x, y, z, rung) and
// (vx, vy, vz, -).  A gather of particles in no order reads a whole 32-byte
// sector (64 bytes of HBM) for each of seven arrays' values; from the records
// it reads two.  It pays only for such an order: *njump, counted over the
// final order by k_finish, says how many sources lie outside the previous
// one's sector (nearly n in random order, n / 8 in a sorted set).
__device__ __forceinline__ bool records_pay(const int* njump, int64_t n) { return njump && *njump > n / 2; }

__global__ void k_records(int64_t n, const int* __restrict__ njump, const uint32_t* __restrict__ x,
                          const uint32_t* __restrict__ y, const uint32_t* __restrict__ z, const float* __restrict__ vx,
                          const float* __restrict__ vy, const float* __restrict__ vz, const int8_t* __restrict__ rung,
                          int4* __restrict__ pr, float4* __restrict__ vr) {
  if (!records_pay(njump, n)) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    pr[i] = make_int4((int)x[i], (int)y[i], (int)z[i], rung[i]);
    vr[i] = make_float4(vx[i], vy[i], vz[i], 0.f);
  }
}

// The permutation applied to every array, from the records (njump given and
// large) or from the arrays; pos4 is written where it is not the records.
__global__ void k_gather(int64_t n, const int32_t* __restrict__ idx, const int* __restrict__ njump,
                         const int4* __restrict__ pr, const float4* __restrict__ vr, const uint32_t* __restrict__ x,
                         const uint32_t* __restrict__ y, const uint32_t* __restrict__ z,
                         const float* __restrict__ vx, const float* __restrict__ vy,
                         const float* __restrict__ vz, const int8_t* __restrict__ rung,
                         uint32_t* __restrict__ x2, uint32_t* __restrict__ y2, uint32_t* __restrict__ z2,
                         float* __restrict__ vx2, float* __restrict__ vy2, float* __restrict__ vz2,
                         int8_t* __restrict__ rung2, int4* __restrict__ pos4) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int32_t i = idx[p];
  if (records_pay(njump, n)) {
    const int4 a = __ldg(pr + i);
    const float4 v = __ldg(vr + i);
    x2[p] = (uint32_t)a.x;
    y2[p] = (uint32_t)a.y;
    z2[p] = (uint32_t)a.z;
    rung2[p] = (int8_t)a.w;
    vx2[p] = v.x;
    vy2[p] = v.y;
    vz2[p] = v.z;
    return;
  }
  const uint32_t a = x[i], b = y[i], c = z[i];
  x2[p] = a;
  y2[p] = b;
  z2[p] = c;
  vx2[p] = vx[i];
  vy2[p] = vy[i];
  vz2[p] = vz[i];
  rung2[p] = rung[i];
  pos4[p] = make_int4((int)a, (int)b, (int)c, 0);
}

// pos4 from the sorted positions, once the records have been read.
__global__ void k_pack_positions(int64_t n, const int* __restrict__ njump, const uint32_t* __restrict__ x,
                                 const uint32_t* __restrict__ y, const uint32_t* __restrict__ z, int4* __restrict__ pos4) {
  if (!records_pay(njump, n)) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    pos4[i] = make_int4((int)x[i], (int)y[i], (int)z[i], 0);
}

// The sorted set back into the current arrays (batch members keep fixed
// device addresses across steps).
__global__ void k_copy_back(int64_t n, const uint32_t* __restrict__ x2, const uint32_t* __restrict__ y2,
                            const uint32_t* __restrict__ z2, const float* __restrict__ vx2,
                            const float* __restrict__ vy2, const float* __restrict__ vz2,
                            const int8_t* __restrict__ rung2, uint32_t* __restrict__ x, uint32_t* __restrict__ y,
                            uint32_t* __restrict__ z, float* __restrict__ vx, float* __restrict__ vy,
                            float* __restrict__ vz, int8_t* __restrict__ rung) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= n) return;
  x[p] = x2[p];
  y[p] = y2[p];
  z[p] = z2[p];
  vx[p] = vx2[p];
  vy[p] = vy2[p];
  vz[p] = vz2[p];
  rung[p] = rung2[p];
}

// One block for up to four tiles; above that, block sums + one-block scan of
// them + apply (three launches of a few microseconds each against 0.22 ms
// for one block walking the 262,144 cells of a 64^3 chain mesh).
int scan_exclusive(tpm_ctx* c, const int32_t* in, int64_t n, int32_t* out) {
  if (n <= (int64_t)kScanTile * 4) {
    k_scan_single<<<1, kScanThreads, 0, c->stream>>>(in, n, out);
    c->launches++;
  } else {
    const int nb = ceil_div(n, kScanTile);
    k_scan_blocksum<<<nb, kScanThreads, 0, c->stream>>>(in, n, c->blocksum);
    k_scan_single<<<1, kScanThreads, 0, c->stream>>>(c->blocksum, nb, c->blocksum + nb + 1);
    k_scan_apply<<<nb, kScanThreads, 0, c->stream>>>(in, n, c->blocksum + nb + 1, out);
    c->launches += 3;
  }
  TPM_CUDA_TRY(cudaGetLastError());
  return TPM_OK;
}

// Where k_finish takes over: the first node level whose nodes are expected to
// fit its shared memory (0.8 of kUnit positions at the mean density, for the
// widest node) with few enough cells.  udim < 0: no level does, or the level
// kernels are faster.
//
// A wave of units (two blocks on each of 148 SMs) takes 4.7 us per level
// however few particles they hold, since each fills a table of its cells'
// nodes; the level kernels take 18 us up to 5e5 particles and 22 us per 1e6
// particles above (deep levels of fine meshes, where every position looks its
// node up).  Hence units are taken up to four waves, or with at least 700
// particles each; empty ones cost a block's start.  Sort with and without
// them: 0.65 / 0.78 ms (8,000 particles, 128^3 cells, 1,024 units), 1.26 / 0.96
// (200,003, 160^3, 2,560), 1.92 / 2.25 (4e6, 160^3), 2.86 / 2.65 (4e6, 200^3,
// 6,400), 5.00 / 2.11 (200,003, 260^3, 16,640).
constexpr int64_t kUnitsFew = 4 * 2 * 148, kUnitMean = 700;

struct FinishStart {
  int udim = -1, ulevel = 0;
};

FinishStart finish_start(const tpm_ctx* c, int64_t n) {
  const int64_t C = c->C;
  for (int dim = 2; dim >= 0; dim--)
    for (int level = 0; level < c->max_depth1d; level++) {
      const int64_t row = dim == 2 ? C * C : dim == 1 ? C : 1;
      const int64_t cells = c->unit_levels[level].widest * row;
      const double mean = (double)n * (double)cells / ((double)C * C * C);
      if (cells > kUnitCells || (n > kUnit && mean > 0.8 * kUnit)) continue;
      const int64_t units = C * C / row * c->unit_levels[level].count;
      if (std::min(units, n) + units / 128 > std::max(kUnitsFew, n / kUnitMean)) return {};
      return {dim, level};
    }
  return {};
}

// The partition levels over c->key / c->idx (cell offsets and cellof are in
// place); the final order goes to c->prefix.  Launches: two per level above
// the units, one for all the rest.  The levels below the units are launched
// only where a unit may exceed kUnit (n > kUnit); they return at once unless
// one does.
int partition(tpm_ctx* c, int64_t n) {
  const int C = c->C;
  cudaStream_t s = c->stream;
  const int nb = ceil_div(n, kScanTile), depth = c->max_depth1d;
  const FinishStart f = finish_start(c, n);
  // look-back words, then a tile counter per level and the sort's other counters
  unsigned long long* status = c->scan_status;
  int* counters = reinterpret_cast<int*>(status + nb);
  TPM_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(unsigned long long) * nb + sizeof(int) * kSortCounters, s));
  int* nbig = counters + kSortBig;
  const UnitLevel ul = f.udim < 0 ? UnitLevel{} : c->unit_levels[f.ulevel];
  UnitArgs u{C, f.udim, f.ulevel, ul.count, c->unit_cuts + ul.at, c->cell_begin, c->tree, c->depth1d, depth, c->key,
             c->idx, c->prefix, nbig, counters + kSortJumps, counters + kSortGaveUp};
  const int64_t units = f.udim < 0 ? 0 : (f.udim == 2 ? 1 : f.udim == 1 ? (int64_t)C : (int64_t)C * C) * u.cuts_n;
  if (n > kUnit && units > 0) {
    k_big_units<<<ceil_div(units, 256), 256, 0, s>>>(u, (int)units);
    c->launches++;
  }
  // resident blocks at most, which take tiles in turn: a launch with nothing
  // to do (below the units) is then short
  const int scan_blocks = std::min(nb, 148 * 4), swap_blocks = std::min(ceil_div(n, kSwapBlock), 148 * 8);
  int4* heads = reinterpret_cast<int4*>(c->blocksum);  // free once the cell counts are scanned
  int l = 0;
  for (int dim = 2; dim >= 0; dim--)
    for (int level = 0; level < depth; level++, l++) {
      const bool below = dim < f.udim || (dim == f.udim && level >= f.ulevel);
      if (below && n <= kUnit) continue;
      LevelArgs a{n, C, dim, level, f.udim, f.ulevel, below ? 1 : 0, nbig, c->cellof, c->key, c->cell_begin, c->tree,
                  c->depth1d};
      k_level_scan<<<scan_blocks, kScanThreads, 0, s>>>(a, (unsigned)(l + 1), counters + l, status, c->slot, c->prefix,
                                                         heads, c->wait_polls, counters + kSortGaveUp, c->d_err);
      k_level_swap<<<swap_blocks, 256, 0, s>>>(a, c->prefix, c->slot, heads, counters + kSortGaveUp, c->key, c->idx);
      c->launches += 2;
    }
  if (units > 0) {
    k_finish<<<(unsigned)units, kFinishThreads, kFinishSmem, s>>>(u);
    c->launches++;
  } else {
    TPM_CUDA_TRY(cudaMemcpyAsync(c->prefix, c->idx, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s));
  }
  TPM_CUDA_TRY(cudaGetLastError());
  return TPM_OK;
}

}  // namespace

// Host tables: split thresholds and the 1-D bisection tree.
int sort_init(tpm_ctx* c) {
  const int C = c->C;
  std::vector<uint32_t> thr(C + 1);
  // mid_x = mid_box * Ninv with Ninv = 1.0 / N; xmid = fixed32(mid_x)
  // (src/chainmesh.cpp:171,198-199; src/particles.cpp:417; tigerpm/fixed.hpp:73-75).
  const double Cinv = 1.0 / C;
  for (int m = 0; m < C; m++) thr[m] = (uint32_t)(4294967296.0 * (m * Cinv));
  thr[C] = 0xffffffffu;
  std::vector<TreeNode> tree((size_t)C * kMaxTreeDepth, TreeNode{0, 0, 0, 0});
  std::vector<int> depth(C);
  int maxd = 0;
  for (int v = 0; v < C; v++) {
    int lo = 0, hi = C, k = 0;
    while (hi - lo > 1) {
      if (k >= kMaxTreeDepth) return fail(TPM_ERR_INVALID, "chain_dim too large");
      const int mid = lo + (hi - lo) / 2;
      tree[(size_t)v * kMaxTreeDepth + k] = TreeNode{lo, mid, hi, 0};
      if (v < mid) hi = mid;
      else lo = mid;
      k++;
    }
    depth[v] = k;
    maxd = std::max(maxd, k);
  }
  c->max_depth1d = maxd;
  TPM_CUDA_TRY(cudaMemcpy(c->thr, thr.data(), sizeof(uint32_t) * (C + 1), cudaMemcpyHostToDevice));
  TPM_CUDA_TRY(cudaMemcpy(c->tree, tree.data(), sizeof(TreeNode) * tree.size(), cudaMemcpyHostToDevice));
  TPM_CUDA_TRY(cudaMemcpy(c->depth1d, depth.data(), sizeof(int) * C, cudaMemcpyHostToDevice));
  // the intervals of each depth of the bisection, as their first coordinates
  std::vector<int> cuts, at{0, C};
  for (int l = 0; l < maxd; l++) {
    UnitLevel u{(int)cuts.size(), (int)at.size() - 1, 0};
    for (size_t i = 0; i + 1 < at.size(); i++) u.widest = std::max<int64_t>(u.widest, at[i + 1] - at[i]);
    c->unit_levels.push_back(u);
    cuts.insert(cuts.end(), at.begin(), at.end());
    std::vector<int> next;
    for (size_t i = 0; i + 1 < at.size(); i++) {
      next.push_back(at[i]);
      if (at[i + 1] - at[i] > 1) next.push_back(at[i] + (at[i + 1] - at[i]) / 2);
    }
    next.push_back(C);
    at = next;
  }
  if ((int64_t)cuts.size() > unit_cuts_entries(C)) return fail(TPM_ERR_INVALID, "chain_dim too large");
  TPM_CUDA_TRY(cudaMemcpy(c->unit_cuts, cuts.data(), sizeof(int) * cuts.size(), cudaMemcpyHostToDevice));
  TPM_CUDA_TRY(cudaFuncSetAttribute(k_finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFinishSmem));
  return TPM_OK;
}

int chainmesh_sort(tpm_ctx* c) {
  const int64_t n = c->n;
  const int C = c->C;
  const int64_t ncell = (int64_t)C * C * C;
  cudaStream_t s = c->stream;
  stage_begin(c, kStSort);
  TPM_CUDA_TRY(cudaMemsetAsync(c->cell_count, 0, sizeof(int32_t) * (ncell + 1), s));
  if (n > 0) {
    k_cell_keys<<<ceil_div(n, 256), 256, 0, s>>>(n, c->x, c->y, c->z, c->thr, C, c->key, c->idx,
                                                  c->cell_count);
    c->launches++;
  }
  int rc = scan_exclusive(c, c->cell_count, ncell, c->cell_begin);
  if (rc) return rc;
  if (n > 0) {
    const int32_t* order = c->prefix;  // original index of the particle at each sorted position
    if (c->opt.sort_mode == TPM_SORT_FAST) {
      TPM_CUDA_TRY(cudaMemsetAsync(c->cell_count, 0, sizeof(int32_t) * (ncell + 1), s));
      k_fast_scatter<<<ceil_div(n, 256), 256, 0, s>>>(n, c->key, c->cell_begin, c->cell_count, c->prefix);
      k_fast_cellsort<<<ceil_div(ncell * 32, 256), 256, 0, s>>>(ncell, c->cell_begin, c->prefix);
      c->launches += 2;
    } else {
      k_cellof<<<ceil_div(ncell * 32, 256), 256, 0, s>>>(ncell, c->cell_begin, c->cellof);
      c->launches++;
      const int rc2 = partition(c, n);
      if (rc2) return rc2;
    }
    // Records pay once the arrays outgrow the 126 MB L2 (7.65e6 particles in
    // random order: gather 654 -> 366 us with its two helpers; 2.1e6: 30 us
    // slower): pos4 and the key / idx / cellof / slot block hold them.
    const int* njump = nullptr;
    if (c->opt.sort_mode != TPM_SORT_FAST && n >= kRecordsFrom) {
      njump = reinterpret_cast<const int*>(c->scan_status + ceil_div(n, kScanTile)) + kSortJumps;
      const int blocks = (int)std::min<int64_t>(ceil_div(n, 256), 148 * 16);
      k_records<<<blocks, 256, 0, s>>>(n, njump, c->x, c->y, c->z, c->vx, c->vy, c->vz, c->rung, c->pos4,
                                       reinterpret_cast<float4*>(c->sort4));
      c->launches++;
    }
    k_gather<<<ceil_div(n, 256), 256, 0, s>>>(n, order, njump, c->pos4, reinterpret_cast<const float4*>(c->sort4), c->x, c->y,
                                               c->z, c->vx, c->vy, c->vz, c->rung, c->x2, c->y2, c->z2, c->vx2, c->vy2,
                                               c->vz2, c->rung2, c->pos4);
    c->launches++;
    if (njump) {
      const int blocks = (int)std::min<int64_t>(ceil_div(n, 256), 148 * 16);
      k_pack_positions<<<blocks, 256, 0, s>>>(n, njump, c->x2, c->y2, c->z2, c->pos4);
      c->launches++;
    }
    TPM_CUDA_TRY(cudaGetLastError());
    if (c->stable_buffers) {
      k_copy_back<<<ceil_div(n, 256), 256, 0, s>>>(n, c->x2, c->y2, c->z2, c->vx2, c->vy2, c->vz2, c->rung2, c->x,
                                                   c->y, c->z, c->vx, c->vy, c->vz, c->rung);
      c->launches++;
      TPM_CUDA_TRY(cudaGetLastError());
    } else {
      std::swap(c->x, c->x2);
      std::swap(c->y, c->y2);
      std::swap(c->z, c->z2);
      std::swap(c->vx, c->vx2);
      std::swap(c->vy, c->vy2);
      std::swap(c->vz, c->vz2);
      std::swap(c->rung, c->rung2);
    }
  }
  stage_end(c, kStSort);
  c->sorted = true;
  c->pot_valid = false;  // forces and potentials are not permuted with the particles
  c->host_cells_valid = false;
  return TPM_OK;
}

}  // namespace tpm
