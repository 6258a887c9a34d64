// fcdem_count.cu -- the cell counting-sort pipeline of fcdemUpdate.
//
// The reference re-sorts all particles by cell hash every step
// (thrust::sort_by_key, particleSystem.cu:265-270) and then scatters the
// cell ranges (reorderDataAndFindCellStartD).  Inside fcdemUpdate the same
// result comes from a counting sort over the cells:
//
//   count   the kernel that computes a particle's cell hash h (the fused
//           collide+integrate of the previous step, or kIntegrateHashCount)
//           also takes r = atomicAdd(&cnt[h], 1) and counts h's 4096-cell
//           tile in tileCnt;
//   scan    up to 4,608 tiles kScanCellsOwn, whose CTAs sum the tile counts
//           before their own; above that kScanTiles (one CTA) or
//           kScanTileBlocks and kAddTileBlocks scan the tile counts and
//           kScanCellsMany the tiles' cells -- no inter-CTA waits; a
//           tile without particles writes its constant offsets and skips
//           reading cnt.  off = exclusive prefix sum of cnt over C + 1 cells,
//           cnt and tileCnt are cleared for the next step; off[c] .. off[c+1]
//           is cell c's range, empty or not;
//   scatter kScatterCells: slot off[h] + r receives (h, particle, ...);
//   fix-up  kFixupGather: the atomic ranks order a cell's members
//           arbitrarily, so each slot re-ranks its particle among the
//           members of its cell by particle index (the order of the
//           reference's stable sort), then writes hash/index in sorted order
//           and gathers pos/vel into sortedPos/sortedVel (the reorder).
//
// The collide kernel reads `off` instead of cellStart/cellEnd.  At the end of
// fcdemUpdate kCellTables writes cellStart/cellEnd from `off`, so every array
// holds what the reference's stages leave.  A cell with more than
// kFixupMaxCell members is left out of the per-slot re-rank (its cost grows
// with the square of the cell) and listed instead; kFixupLarge then gives each
// listed cell one CTA that ranks its members by particle index, whatever the
// cell's size: with a bitmap of their indices when the indices are dense
// enough, else with a stable block radix sort.
#include <algorithm>

#include "fcdem_dem.cuh"

namespace fcdem {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;  // 4096 cells
constexpr int kTileShift = 12;  // log2(kScanTile)
constexpr unsigned kEmpty = 0xffffffffu;
static_assert((1 << kTileShift) == kScanTile, "tile shift");

// The fix-up lists this step's large cells afresh, and collide its crowded
// groups (crowdCount: two counters, or none).
__device__ __forceinline__ void resetLists(unsigned *largeCount, unsigned *crowdCount) {
  *largeCount = 0u;
  if (crowdCount) crowdCount[0] = crowdCount[1] = 0u;
}

// Exclusive prefix sums of the per-tile counts (one tile = kScanTile cells):
// tileOff[t] = sum of tileCnt[0..t), tileOff[tiles] = the total; tileCnt is
// cleared for the next step.  One CTA of 1024 threads, tiles in chunks.
__global__ void __launch_bounds__(1024)
kScanTiles(unsigned *tileCnt, unsigned *tileOff, unsigned tiles,
           unsigned *largeCount, unsigned *crowdCount) {
  chainTrigger();
  chainWait();
  __shared__ unsigned sWarp[32];
  __shared__ unsigned sCarry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    sCarry = 0;
    resetLists(largeCount, crowdCount);
  }
  __syncthreads();
  for (unsigned base = 0; base < tiles; base += 1024) {
    const unsigned t = base + tid;
    const unsigned v = t < tiles ? tileCnt[t] : 0u;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sWarp[warp] = x;
    __syncthreads();
    if (warp == 0) {
      unsigned w = sWarp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      sWarp[lane] = w;
    }
    __syncthreads();
    const unsigned carry = sCarry;
    if (t < tiles) {
      tileOff[t] = carry + (warp ? sWarp[warp - 1] : 0u) + x - v;
      tileCnt[t] = 0u;
    }
    __syncthreads();
    if (tid == 0) sCarry = carry + sWarp[31];
    __syncthreads();
  }
  if (tid == 0) tileOff[tiles] = sCarry;
}

// The same prefix over many tiles (batches of many scenes: tens of
// thousands of tiles), in two short launches instead of one CTA walking them
// all: kScanTileBlocks scans each block of 1024 tile counts and writes its
// total, kAddTileBlocks adds the totals of the blocks before.
constexpr unsigned kTileBlock = 1024;
constexpr unsigned kTilesOneCta = 8192;  // up to this many tiles kScanTiles runs alone
constexpr unsigned kTilesOwnPrefix = 4608;  // up to this many tiles kScanCellsOwn

__global__ void __launch_bounds__(kTileBlock)
kScanTileBlocks(unsigned *tileCnt, unsigned *tileOff, unsigned tiles,
                unsigned *blockSum, unsigned *largeCount,
                unsigned *crowdCount) {
  chainTrigger();
  chainWait();
  __shared__ unsigned sWarp[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (blockIdx.x == 0 && tid == 0) resetLists(largeCount, crowdCount);
  const unsigned t = blockIdx.x * kTileBlock + tid;
  const unsigned v = t < tiles ? tileCnt[t] : 0u;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sWarp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    unsigned w = sWarp[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    sWarp[lane] = w;
  }
  __syncthreads();
  if (t < tiles) {
    tileOff[t] = (warp ? sWarp[warp - 1] : 0u) + x - v;
    tileCnt[t] = 0u;
  }
  if (tid == 0) blockSum[blockIdx.x] = sWarp[31];
}

__global__ void __launch_bounds__(kTileBlock)
kAddTileBlocks(unsigned *tileOff, unsigned tiles,
               const unsigned *blockSum) {
  chainTrigger();
  chainWait();
  __shared__ unsigned sPart[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned part = 0;
  for (unsigned b = tid; b < blockIdx.x; b += kTileBlock) part += blockSum[b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) sPart[warp] = part;
  __syncthreads();
  unsigned carry = 0;
  for (int w = 0; w < (int)(kTileBlock / 32); ++w) carry += sPart[w];
  const unsigned t = blockIdx.x * kTileBlock + tid;
  if (t < tiles) tileOff[t] += carry;
  if (blockIdx.x == gridDim.x - 1 && tid == 0)
    tileOff[tiles] = carry + blockSum[blockIdx.x];
}

// One tile of the cell scan: off[c] = t0 + exclusive prefix of cnt within the
// tile, cnt cleared.  A tile without particles (t0 == t1) only writes its
// constant offsets; tileOffPrev[tile] records the constant a tile's offsets
// were last written with (0xffffffff after a tile with particles, whose
// offsets vary), and a tile that stays empty with the same prefix -- the
// common case in sparse grids: the cells above and below a pile -- is left as
// it is by the callers.
// Round q of a tile covers cells q*1024 .. +1024, thread t the four at 4t
// (16-byte accesses, coalesced).  All threads of the CTA, which have met at a
// barrier since tileOffPrev was read and sWarp was used.
__device__ __forceinline__ void scanTile(unsigned tile, unsigned t0, unsigned t1, unsigned *cnt,
                                         unsigned *off, unsigned m, unsigned *tileOffPrev,
                                         unsigned *sWarp) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kRounds = kScanItems / 4;
  const size_t tbase = (size_t)tile * kScanTile;
  if (tid == 0) tileOffPrev[tile] = t0 == t1 ? t0 : 0xffffffffu;
  if (t0 == t1) {  // every cell starts (and ends) at t0
#pragma unroll
    for (int q = 0; q < kRounds; ++q) {
      const size_t c0 = tbase + (size_t)q * (kScanThreads * 4) + (size_t)tid * 4;
      if (c0 + 4 <= m) {
        reinterpret_cast<uint4 *>(off + c0)[0] = make_uint4(t0, t0, t0, t0);
      } else {
        for (int k = 0; k < 4; ++k)
          if (c0 + k < m) off[c0 + k] = t0;
      }
    }
    return;
  }
  uint4 v[kRounds];
  unsigned excl[kRounds];
#pragma unroll
  for (int q = 0; q < kRounds; ++q) {  // all loads in flight before the scans
    const size_t c0 = tbase + (size_t)q * (kScanThreads * 4) + (size_t)tid * 4;
    if (c0 + 4 <= m) {
      v[q] = reinterpret_cast<const uint4 *>(cnt + c0)[0];
    } else {
      v[q].x = c0 < m ? cnt[c0] : 0u;
      v[q].y = c0 + 1 < m ? cnt[c0 + 1] : 0u;
      v[q].z = c0 + 2 < m ? cnt[c0 + 2] : 0u;
      v[q].w = c0 + 3 < m ? cnt[c0 + 3] : 0u;
    }
  }
  unsigned carry = 0;
#pragma unroll
  for (int q = 0; q < kRounds; ++q) {
    const unsigned sum = v[q].x + v[q].y + v[q].z + v[q].w;
    unsigned x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sWarp[warp] = x;
    __syncthreads();
    if (warp == 0) {
      unsigned w = lane < kScanThreads / 32 ? sWarp[lane] : 0u;
#pragma unroll
      for (int o = 1; o < kScanThreads / 32; o <<= 1) {
        unsigned y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      if (lane < kScanThreads / 32) sWarp[lane] = w;
    }
    __syncthreads();
    excl[q] = carry + (warp ? sWarp[warp - 1] : 0u) + x - sum;
    carry += sWarp[kScanThreads / 32 - 1];
    __syncthreads();  // sWarp is reused by the next round
  }
#pragma unroll
  for (int q = 0; q < kRounds; ++q) {
    const size_t c0 = tbase + (size_t)q * (kScanThreads * 4) + (size_t)tid * 4;
    uint4 o;
    o.x = t0 + excl[q];
    o.y = o.x + v[q].x;
    o.z = o.y + v[q].y;
    o.w = o.z + v[q].z;
    if (c0 + 4 <= m) {
      reinterpret_cast<uint4 *>(off + c0)[0] = o;
      reinterpret_cast<uint4 *>(cnt + c0)[0] = make_uint4(0u, 0u, 0u, 0u);
    } else {
      const unsigned ov[4] = {o.x, o.y, o.z, o.w};
      for (int k = 0; k < 4; ++k)
        if (c0 + k < m) {
          off[c0 + k] = ov[k];
          cnt[c0 + k] = 0u;
        }
    }
  }
}

// Few tiles (kTilesOwnPrefix): one CTA per tile, which sums the tile counts
// before its own itself; the scatter clears them.  Saves the launch of
// kScanTiles and its single CTA's latency (4 to 7 us per step).
__global__ void __launch_bounds__(kScanThreads)
kScanCellsOwn(unsigned *cnt, unsigned *off, unsigned m, const unsigned *tileCnt,
              unsigned *tileOffPrev, unsigned *largeCount, unsigned *crowdCount) {
  __shared__ unsigned sWarp[kScanThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned tile = blockIdx.x;
  chainTrigger();
  chainWait();
  if (tile == 0 && tid == 0) resetLists(largeCount, crowdCount);
  const unsigned held = tileOffPrev[tile], mine = tileCnt[tile];
  unsigned part = 0;
  for (unsigned k = tid; k < tile; k += kScanThreads) part += tileCnt[k];
  part = __reduce_add_sync(0xffffffffu, part);
  if (lane == 0) sWarp[warp] = part;
  __syncthreads();
  unsigned t0 = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) t0 += sWarp[w];
  if (mine == 0u && held == t0) return;
  __syncthreads();  // sWarp is used again
  scanTile(tile, t0, t0 + mine, cnt, off, m, tileOffPrev, sWarp);
}

// Many tiles: a CTA takes tiles blockIdx, blockIdx + grid, ... (at most 32).
// Neighbouring tiles, which are full or empty together, go to different CTAs,
// and an empty one that stays as it is costs a lane's three loads instead of
// a CTA (20,481 tiles of 40 obstacle scenes: 25 -> 11 us; with 4,097 tiles a
// CTA each is as fast).
constexpr unsigned kScanCtas = 8 * 152;
__global__ void __launch_bounds__(kScanThreads)
kScanCellsMany(unsigned *cnt, unsigned *off, unsigned m, unsigned tiles, const unsigned *tileOff,
               unsigned *tileOffPrev) {
  __shared__ unsigned sWarp[kScanThreads / 32];
  const unsigned lane = threadIdx.x & 31u;
  chainTrigger();
  chainWait();
  // lane k: the CTA's tile k, its first slot, its end and what off holds there
  const unsigned mine = blockIdx.x + lane * gridDim.x;
  const unsigned first = mine < tiles ? tileOff[mine] : 0u;
  const unsigned end = mine < tiles ? tileOff[mine + 1] : 0u;
  const unsigned held = mine < tiles ? tileOffPrev[mine] : 0u;
  unsigned todo = __ballot_sync(0xffffffffu, mine < tiles && (first != end || held != first));
  __syncthreads();  // every warp has read tileOffPrev
  while (todo) {
    const int k = __ffs((int)todo) - 1;
    todo &= todo - 1u;
    scanTile(blockIdx.x + (unsigned)k * gridDim.x, __shfl_sync(0xffffffffu, first, k),
             __shfl_sync(0xffffffffu, end, k), cnt, off, m, tileOffPrev, sWarp);
  }
}

// Entry i (a slot of the previous order, or the particle itself on the first
// step) holds the particle's new cell hash h and its count rank r; slot
// off[h] + r receives (h, the particle's index, the entry i, off[h]) as one
// 16-byte word: the scatter is bound by the sectors it touches, and three
// 4-byte arrays touched three (4.2M spheres, four steps, the first from random
// order: 40 us a step against 50; 2M in box scenes 16.7 against 19.1).
__global__ void __launch_bounds__(256)
kScatterCells(const unsigned *hashN, const unsigned *rankN, const unsigned *origOf,
              const unsigned *off, uint4 *slots, unsigned n, unsigned numCells, unsigned *tileCnt,
              unsigned tiles, DeviceStatus *status) {
  chainTrigger();
  chainWait();
  unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  // (tiles == 0 when kScanTiles has cleared the tile counts)
  for (unsigned k = i; k < tiles; k += gridDim.x * blockDim.x) tileCnt[k] = 0u;
  if (i >= n) return;
  unsigned h = hashN[i];
  if (h >= numCells) {
    report(status, kStatusKeyRange);
    return;
  }
  const unsigned a = off[h], s = a + rankN[i];
  if (s >= n) {
    report(status, kStatusKeyRange);
    return;
  }
  slots[s] = make_uint4(h, origOf ? origOf[i] : i, i, a);
}

// Largest cell that the per-slot re-rank handles (each slot reads every
// member of its cell).
constexpr unsigned kFixupMaxCell = 1024;
// Up to this many particles it handles any cell, and kFixupLarge is not
// launched: one launch of nine of a small scene's update (2,000 spheres: 28 ->
// 25.7 us); a cell of all 4,096 costs some 50 us then.
constexpr unsigned kFixupAllCells = 4096;
inline unsigned fixupMaxCell(unsigned n) { return n <= kFixupAllCells ? n : kFixupMaxCell; }

// Capacity of the large-cell list: a listed cell has more than kFixupMaxCell
// of the n particles, so at most n / (kFixupMaxCell + 1) cells are listed.
inline unsigned largeCapacity(unsigned n) { return n / (kFixupMaxCell + 1) + 1; }
// CTAs of kFixupLarge: one per SM at most.
inline unsigned largeCtas(unsigned n) { return std::min(largeCapacity(n), numSms()); }

// Stable order inside each cell + the reorder gather.  The particle of slot
// s is re-ranked among its cell's members by particle index; its position and
// velocity are gathered from its entry of the previous order.  A cell above
// maxCell members is appended to large[1..] (large[0] counts) by its
// first slot and left to kFixupLarge.
__global__ void __launch_bounds__(256)
kFixupGather(const uint4 *slots, const unsigned *off, unsigned *hashOut, unsigned *indexOut,
             float4 *sortedPos, float4 *sortedVel, const float4 *prevPos, const float4 *prevVel,
             unsigned n, unsigned numCells, unsigned maxCell, unsigned *large, unsigned largeCap,
             DeviceStatus *status) {
  chainTrigger();
  chainWait();
  unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint4 w = slots[s];
  const unsigned h = w.x, me = w.y, prev = w.z, a = w.w;
  if (h >= numCells || me >= n || prev >= n || a > s) return;  // unfilled slot (reported)
  const float4 p4 = prevPos[prev], v4 = prevVel[prev];
  const unsigned b = min(off[h + 1], n);
  if (b - a > maxCell) {
    if (s == a) {
      const unsigned k = atomicAdd(large, 1u);
      if (k < largeCap)
        large[1 + k] = h;
      else
        report(status, kStatusCellOverflow);
    }
    return;
  }
  unsigned r = 0;
  for (unsigned t = a; t < b; ++t) r += slots[t].y < me ? 1u : 0u;
  const unsigned dst = a + r;
  if (dst >= n) return;
  hashOut[dst] = h;
  indexOut[dst] = me;
  sortedPos[dst] = p4;
  sortedVel[dst] = v4;
}

// --- sortParticles as a counting sort (countSortPairs) -----------------------
// The same passes over (key, value) pairs: the key is the cell (its low `bits`
// bits), the position in the arrays takes the particle index's place, and the
// value travels in the slot, so the sort is stable and in place.
//
// Crowded cells.  A cell of at least `least` pairs (a giant: at most 256 of them)
// would keep one CTA busy for long.  Its pairs are not ranked by slot but taken
// in the order of the arrays: kScatterPairs leaves each one's slot in rank
// (kGiantSlot set) and counts them per giant and part of the arrays, and
// kFixupLarge scatters each part from there, one CTA each.  Sorts with giants /
// before there were any / with the radix sort: 2M pairs of one key 139 / 5,936 /
// 104 us, of four keys 140 / 1,500 / 104, 100,003 pairs of one key 35 / 305 / 58;
// it costs a sort without giants about 1 us.  Cells between 1,025 pairs and a giant
// stay with one CTA each, smaller ones with the ranking by slot: 2M pairs in cells
// of 500, 1,000 and 20,000 take 241, 412 and 473 us (radix 110).
constexpr unsigned kGiants = 256, kGiantSlot = 1u << 31;
struct Giants {
  unsigned *count;  // [giant][part]
  unsigned *first;  // [giant]: first slot, or 0xffffffff; [kGiants]: whether there are any
  unsigned least;   // pairs in a giant
  unsigned parts, part;  // parts of the arrays and their size
  // giants begin at least `least` slots apart
  __device__ __forceinline__ unsigned id(unsigned firstSlot) const { return firstSlot / least; }
};

template <bool kTiles>
__global__ void __launch_bounds__(256)
kCountKeys(const unsigned *keys, unsigned n, unsigned mask, unsigned *rank, unsigned *cnt,
           unsigned *tileCnt, Giants giants, DeviceStatus *status) {
  chainTrigger();
  chainWait();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned k = i < n ? keys[i] : 0u, h = k & mask;
  for (unsigned c = i; c < kGiants * giants.parts; c += gridDim.x * blockDim.x) {
    giants.count[c] = 0u;
    if (c < kGiants) giants.first[c] = 0xffffffffu;
    if (c == 0u) giants.first[kGiants] = 0u;
  }
  const unsigned live = __ballot_sync(0xffffffffu, i < n), lane = threadIdx.x & 31u;
  if (i >= n) return;
  if (k != h) report(status, kStatusKeyRange);
  // Where two lanes in a row share a cell, one atomic for the members of the warp
  // that do: the pairs of a crowded cell would queue on its counter (2M pairs of
  // one key: 5.8 ms the sort, with plain atomics and without giants; always
  // looking for the members costs a sort of 1M pairs of many keys 4 us).
  const unsigned up = __shfl_down_sync(live, h, 1);
  if (__any_sync(live, lane < 31u && ((live >> (lane + 1u)) & 1u) && up == h)) {
    const unsigned peers = __match_any_sync(live, h);
    const int leader = __ffs((int)peers) - 1;
    unsigned first = 0u;
    if ((int)lane == leader) first = atomicAdd(cnt + h, (unsigned)__popc(peers));
    rank[i] = __shfl_sync(live, first, leader) + __popc(peers & ((1u << lane) - 1u));
  } else {
    rank[i] = atomicAdd(cnt + h, 1u);
  }
  if (kTiles) countTile(tileCnt, h >> kTileShift);
}

__global__ void __launch_bounds__(256)
kScatterPairs(const unsigned *keys, const unsigned *vals, unsigned *rankN, const unsigned *off,
              uint4 *slots, unsigned n, unsigned mask, unsigned *tileCnt, unsigned tiles,
              Giants giants) {
  chainTrigger();
  chainWait();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  for (unsigned k = i; k < tiles; k += gridDim.x * blockDim.x) tileCnt[k] = 0u;
  const unsigned live = __ballot_sync(0xffffffffu, i < n), lane = threadIdx.x & 31u;
  if (i >= n) return;
  const unsigned k = keys[i], a = off[k & mask], b = off[(k & mask) + 1u], r = rankN[i], s = a + r;
  if (s < n) slots[s] = make_uint4(k, i, vals[i], a);
  const bool giant = b - a >= giants.least;
  const unsigned inGiants = __ballot_sync(live, giant);
  if (!giant) return;
  const unsigned id = giants.id(a), part = i / giants.part;
  rankN[i] = kGiantSlot | s;
  if (r == 0u) {
    giants.first[id] = a;
    giants.first[kGiants] = 1u;
  }
  // (a warp may lie in two parts)
  const unsigned peers = __match_any_sync(inGiants, id * giants.parts + part);
  if ((int)lane == __ffs((int)peers) - 1)
    atomicAdd(giants.count + id * giants.parts + part, (unsigned)__popc(peers));
}

__global__ void __launch_bounds__(256)
kFixupPairs(const uint4 *slots, const unsigned *off, unsigned *keys, unsigned *vals, unsigned n,
            unsigned mask, unsigned maxCell, unsigned least, unsigned *large, unsigned largeCap,
            DeviceStatus *status) {
  chainTrigger();
  chainWait();
  const unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint4 w = slots[s];
  const unsigned h = w.x & mask, a = w.w, b = min(off[h + 1], n);
  if (a > s) return;
  if (b - a > maxCell) {  // for kFixupLarge
    if (s == a && b - a < least) {
      const unsigned k = atomicAdd(large, 1u);
      if (k < largeCap)
        large[1 + k] = h;
      else
        report(status, kStatusCellOverflow);
    }
    return;
  }
  unsigned r = 0;
  if (b - a < 32u) {
#pragma unroll 4
    for (unsigned t = a; t < b; ++t) r += slots[t].y < w.y ? 1u : 0u;
  } else {
#pragma unroll 32  // eight slots a line: several lines on their way
    for (unsigned t = a; t < b; ++t) r += slots[t].y < w.y ? 1u : 0u;
  }
  if (a + r >= n) return;
  keys[a + r] = w.x;
  vals[a + r] = w.z;
}

constexpr int kLargeThreads = 1024;
constexpr int kLargeWarps = kLargeThreads / 32;
constexpr int kBitmapSlots = 16;  // CTAs of kFixupLarge that own a bitmap

// Words of one bitmap slot: a presence bit per particle index.
__host__ __device__ inline size_t bitmapWords(unsigned n) { return (size_t)n / 32 + 1; }

struct LargeSmem {
  unsigned bin[256];                  // running base of each digit
  unsigned total[256];                // a chunk's count of each digit
  unsigned part[8];                   // warp totals of the digit scan
  unsigned warpCnt[kLargeWarps][256]; // per-warp digit counts of a chunk
  unsigned warpSum[kLargeWarps];      // bitmap path: popcount of each warp's run
  unsigned lo, hi;                    // bitmap path: smallest / largest member index
};

// Bitmap rank of a large cell's members (the members' particle indices are
// distinct): bit i of `bits` is set for member index i; pre[w] is the number
// of set bits in words w0 .. w-1; the rank of member i among the cell's
// members is pre[i / 32] + the set bits below i in its word.  Words w0..w1
// (the members' index span) are cleared, filled, counted and scanned: the
// work grows with the span, not with the member count, so the caller takes
// this path when the span is at most kBitmapSpan words per member.
constexpr unsigned kBitmapSpan = 16;

__device__ void bitmapRanks(const uint4 *slots, unsigned a, unsigned c, unsigned n,
                            unsigned w0, unsigned w1, unsigned *bits, unsigned *pre,
                            LargeSmem &sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (unsigned w = w0 + tid; w <= w1; w += kLargeThreads) bits[w] = 0u;
  __syncthreads();
  for (unsigned t = tid; t < c; t += kLargeThreads) {
    const unsigned me = slots[a + t].y;
    if (me < n) atomicOr(bits + (me >> 5), 1u << (me & 31u));
  }
  __syncthreads();
  // each warp owns a contiguous run of words: its total, then the scan
  const unsigned span = w1 - w0 + 1u;
  const unsigned run = ((span + kLargeWarps - 1u) / kLargeWarps + 31u) & ~31u;
  const unsigned ws = w0 + (unsigned)warp * run;
  const unsigned we = min(ws + run, w1 + 1u);
  unsigned sum = 0;
  for (unsigned w = ws + lane; w < we; w += 32) sum += __popc(bits[w]);
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) sm.warpSum[warp] = sum;
  __syncthreads();
  if (warp == 0) {
    const unsigned v = sm.warpSum[lane];
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    sm.warpSum[lane] = x - v;
  }
  __syncthreads();
  unsigned carry = sm.warpSum[warp];
  for (unsigned base = ws; base < we; base += 32) {
    const unsigned w = base + lane;
    const unsigned v = w < we ? __popc(bits[w]) : 0u;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (w < we) pre[w] = carry + x - v;
    carry += __shfl_sync(0xffffffffu, x, 31);
  }
  __syncthreads();
}

// Exclusive prefix sums of 256 counts (thread d < 256: digit d's).
__device__ __forceinline__ unsigned digitScan(unsigned v, LargeSmem &sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned x = v;
  if (tid < 256) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sm.part[warp] = x;
  }
  __syncthreads();
  unsigned before = 0;
  if (tid < 256)
    for (int w = 0; w < warp; ++w) before += sm.part[w];
  __syncthreads();
  return before + x - v;
}

// Entries 0 .. c-1 in order, each to the next free place of its digit (sm.bin[d]
// on entry).  load(t, e) returns the digit of entry t (256: leave it out) and the
// entry in e.  Chunks of kLargeThreads entries go in order; inside a chunk an entry's place is its
// digit's running base + the count of that digit in earlier warps + its rank
// among its warp's peers.
template <class Load, class Store>
__device__ __forceinline__ void stableScatter(unsigned c, LargeSmem &sm, Load load, Store store) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (unsigned base = 0; base < c; base += kLargeThreads) {
    for (int q = tid; q < kLargeWarps * 256; q += kLargeThreads) (&sm.warpCnt[0][0])[q] = 0u;
    __syncthreads();
    const unsigned t = base + tid;
    unsigned long long e = 0ull;
    const unsigned d = t < c ? load(t, e) : 256u;
    const bool valid = d < 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const unsigned rank = __popc(peers & lt);
    if (valid && rank == 0) sm.warpCnt[warp][d] = __popc(peers);
    __syncthreads();
    if (tid < 256) {  // per digit: exclusive prefix over the warps
      unsigned run = 0;
      for (int w = 0; w < kLargeWarps; ++w) {
        const unsigned k = sm.warpCnt[w][tid];
        sm.warpCnt[w][tid] = run;
        run += k;
      }
      sm.total[tid] = run;
    }
    __syncthreads();
    if (valid) store(sm.bin[d] + sm.warpCnt[warp][d] + rank, e);
    __syncthreads();
    if (tid < 256) sm.bin[tid] += sm.total[tid];
    __syncthreads();
  }
}

// One stable pass of a block-wide LSD radix sort: src[0..c) -> dst[0..c)
// by the 8-bit digit at bit `shift`.
__device__ void largeRadixPass(const unsigned long long *src, unsigned long long *dst,
                               unsigned c, int shift, LargeSmem &sm) {
  const int tid = threadIdx.x;
  if (tid < 256) sm.bin[tid] = 0u;
  __syncthreads();
  for (unsigned t = tid; t < c; t += kLargeThreads)
    atomicAdd(&sm.bin[(unsigned)(src[t] >> shift) & 255u], 1u);
  __syncthreads();
  const unsigned first = digitScan(tid < 256 ? sm.bin[tid] : 0u, sm);
  if (tid < 256) sm.bin[tid] = first;
  __syncthreads();
  stableScatter(
      c, sm,
      [&](unsigned t, unsigned long long &e) {
        e = src[t];
        return (unsigned)(e >> shift) & 255u;
      },
      [&](unsigned at, unsigned long long e) { dst[at] = e; });
}

// The large cells listed by kFixupGather, one CTA per cell at a time.  A
// CTA with a bitmap slot (blockIdx < kBitmapSlots) ranks a cell whose
// members' index span is at most kBitmapSpan words per member with
// bitmapRanks and gathers each member straight to its ranked place.
// Otherwise the members (particle index, previous entry) are sorted by
// particle index in the cell's own range of sortedPos (16 bytes per member:
// two 8-byte arrays of the cell's size), written back to their slots,
// then gathered as in kFixupGather.  idBits = bits of the largest particle
// index; bitmaps = kBitmapSlots slots of 2 * bitmapWords(n) words (the bits,
// then the word prefix), or nullptr for the sort only.  kPairs: the members
// of countSortPairs -- position and value in the slot; the keys, which may
// have bits above the cell number, are found again by the position's `rank` in
// the cell; sortedPos is then 16 bytes of work space per pair.
template <bool kPairs>
__global__ void __launch_bounds__(kLargeThreads)
kFixupLarge(uint4 *slots, const unsigned *off, const unsigned *large,
            unsigned largeCap, unsigned *hashOut, unsigned *indexOut,
            float4 *sortedPos, float4 *sortedVel,
            const float4 *prevPos, const float4 *prevVel, unsigned n,
            int idBits, unsigned *bitmaps, const unsigned *rank, Giants giants) {
  chainTrigger();
  chainWait();
  __shared__ LargeSmem sm;
  const unsigned count = min(large[0], largeCap);
  if (kPairs) {
    // this CTA's part of the arrays: the pairs in giants
    if (giants.first[kGiants]) {
      if (threadIdx.x < kGiants) {
        const unsigned first = giants.first[threadIdx.x];
        unsigned before = 0;
        if (first != 0xffffffffu)
          for (unsigned p = 0; p < blockIdx.x; ++p)
            before += giants.count[threadIdx.x * giants.parts + p];
        sm.bin[threadIdx.x] = first + before;
      }
      __syncthreads();
      const unsigned lo = min(n, blockIdx.x * giants.part), c = min(n, lo + giants.part) - lo;
      stableScatter(
          c, sm,
          [&](unsigned t, unsigned long long &e) {
            const unsigned r = rank[lo + t];
            if (!(r & kGiantSlot)) return 256u;
            const uint4 w = slots[r & ~kGiantSlot];
            e = ((unsigned long long)w.x << 32) | w.z;
            return giants.id(w.w);
          },
          [&](unsigned at, unsigned long long e) {
            if (at >= n) return;
            hashOut[at] = (unsigned)(e >> 32);
            indexOut[at] = (unsigned)e;
          });
    }
  }
  const int tid = threadIdx.x;
  const size_t words = bitmapWords(n);
  unsigned *bits = blockIdx.x < (unsigned)kBitmapSlots && bitmaps
                       ? bitmaps + (size_t)blockIdx.x * 2u * words
                       : nullptr;
  for (unsigned k = blockIdx.x; k < count; k += gridDim.x) {
    const unsigned h = large[1 + k];
    const unsigned a = off[h], b = off[h + 1];
    if (b > n || a >= b) continue;  // cannot happen for a listed cell
    const unsigned c = b - a;
    if (bits) {
      // the members' index span decides between the bitmap and the sort
      if (tid == 0) {
        sm.lo = 0xffffffffu;
        sm.hi = 0u;
      }
      __syncthreads();
      unsigned lo = 0xffffffffu, hi = 0u;
      for (unsigned t = tid; t < c; t += kLargeThreads) {
        const unsigned me = slots[a + t].y;
        if (me < n) {
          lo = min(lo, me);
          hi = max(hi, me);
        }
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      if ((tid & 31) == 0) {
        atomicMin(&sm.lo, lo);
        atomicMax(&sm.hi, hi);
      }
      __syncthreads();
      const unsigned mlo = sm.lo, mhi = sm.hi;
      const unsigned w0 = mlo >> 5, w1 = mhi >> 5;
      if (mlo <= mhi && w1 - w0 + 1u <= kBitmapSpan * c) {
        unsigned *pre = bits + words;
        bitmapRanks(slots, a, c, n, w0, w1, bits, pre, sm);
        for (unsigned t = tid; t < c; t += kLargeThreads) {
          const unsigned me = slots[a + t].y, prev = slots[a + t].z;
          if (me >= n || (!kPairs && prev >= n)) continue;  // unfilled slot (reported)
          const unsigned wd = me >> 5;
          const unsigned dst = a + pre[wd] + __popc(bits[wd] & ((1u << (me & 31u)) - 1u));
          if (dst >= n) continue;
          if (kPairs) {
            hashOut[dst] = slots[a + t].x;
            indexOut[dst] = prev;
          } else {
            hashOut[dst] = h;
            indexOut[dst] = me;
            sortedPos[dst] = prevPos[prev];
            sortedVel[dst] = prevVel[prev];
          }
        }
        __syncthreads();  // the bitmap is reused by the next cell
        continue;
      }
    }
    unsigned long long *A = reinterpret_cast<unsigned long long *>(sortedPos + a);
    unsigned long long *B = A + c;
    for (unsigned t = tid; t < c; t += kLargeThreads)
      A[t] = ((unsigned long long)slots[a + t].y << 32) | slots[a + t].z;
    __syncthreads();
    for (int shift = 0; shift < idBits; shift += 8) {
      largeRadixPass(A, B, c, 32 + shift, sm);
      unsigned long long *tmp = A;
      A = B;
      B = tmp;
    }
    if (kPairs) {
      for (unsigned t = tid; t < c; t += kLargeThreads) {
        const unsigned long long e = A[t];
        hashOut[a + t] = slots[a + rank[(unsigned)(e >> 32)]].x;
        indexOut[a + t] = (unsigned)e;
      }
    } else {
      for (unsigned t = tid; t < c; t += kLargeThreads) {
        const unsigned long long e = A[t];
        slots[a + t].y = (unsigned)(e >> 32);
        slots[a + t].z = (unsigned)e;
      }
      __syncthreads();
      for (unsigned t = tid; t < c; t += kLargeThreads) {
        const unsigned me = slots[a + t].y, prev = slots[a + t].z;
        if (me >= n || prev >= n) continue;  // unfilled slot (reported by the scatter)
        hashOut[a + t] = h;
        indexOut[a + t] = me;
        sortedPos[a + t] = prevPos[prev];
        sortedVel[a + t] = prevVel[prev];
      }
    }
    __syncthreads();
  }
}

// cellStart/cellEnd from the prefix table (cellEnd of empty cells untouched,
// as the reference leaves it).  Bound by HBM (8 bytes per cell): four cells per
// thread, 16-byte accesses where the caller's cellStart allows (kVec); 16.7M
// cells in 19 us, one cell per thread 34 (23 with read-only loads).
template <bool kVec>
__global__ void __launch_bounds__(256)
kCellTables(const unsigned *off, unsigned *cellStart, unsigned *cellEnd, unsigned numCells) {
  chainTrigger();
  chainWait();
  const size_t stride = (size_t)gridDim.x * blockDim.x * 4;
  for (size_t c = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; c < numCells; c += stride) {
    if (c + 4 <= numCells) {
      const uint4 o = *reinterpret_cast<const uint4 *>(off + c);
      const unsigned v[5] = {o.x, o.y, o.z, o.w, off[c + 4]};
      unsigned st[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool some = v[k] < v[k + 1];
        st[k] = some ? v[k] : kEmpty;
        if (some) cellEnd[c + k] = v[k + 1];
      }
      if (kVec) {
        *reinterpret_cast<uint4 *>(cellStart + c) = make_uint4(st[0], st[1], st[2], st[3]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) cellStart[c + k] = st[k];
      }
    } else {
      for (size_t k = c; k < numCells; ++k) {
        const unsigned a = off[k], b = off[k + 1];
        cellStart[k] = a < b ? a : kEmpty;
        if (a < b) cellEnd[k] = b;
      }
    }
  }
}

// First step of fcdemUpdate: integrate + calcHash + count.  kTiles: the tile
// counts too; otherwise they follow in kTileReduce.
template <bool kTiles>
__global__ void __launch_bounds__(256)
kIntegrateHashCount(float4 *pos, float4 *vel, float dt,
                    unsigned *hash, unsigned *rank,
                    unsigned *cnt, unsigned *tileCnt, unsigned n,
                    KParams kp) {
  chainTrigger();
  chainWait();
  unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 p4 = pos[i], v4 = vel[i];
  float3 p = make_float3(p4.x, p4.y, p4.z), v = make_float3(v4.x, v4.y, v4.z);
  float r = kp.radiusFromW ? p4.w : kp.p.particleRadius;
  integrateOne(p, v, dt, r, kp.p);
  pos[i] = make_float4(p.x, p.y, p.z, p4.w);
  vel[i] = make_float4(v.x, v.y, v.z, v4.w);
  int3 g = gridPos(p.x, p.y, p.z, kp.p);
  unsigned h = gridHash(g.x, g.y, g.z, kp.p);
  hash[i] = h;
  rank[i] = atomicAdd(cnt + h, 1u);
  if (kTiles) countTile(tileCnt, h >> kTileShift);
}

// tileCnt[t] = sum of cnt over tile t (after kIntegrateHashCount, whose
// particle-order cells are scattered over the tiles: summing the counts once
// is cheaper than one atomic per particle on the few tile counters).
__global__ void __launch_bounds__(kScanThreads)
kTileReduce(const unsigned *cnt, unsigned *tileCnt, unsigned m) {
  chainTrigger();
  chainWait();
  __shared__ unsigned sWarp[kScanThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t tbase = (size_t)blockIdx.x * kScanTile;
  unsigned sum = 0;
#pragma unroll
  for (int q = 0; q < kScanItems / 4; ++q) {
    const size_t c0 = tbase + (size_t)q * (kScanThreads * 4) + (size_t)tid * 4;
    if (c0 + 4 <= m) {
      uint4 v = reinterpret_cast<const uint4 *>(cnt + c0)[0];
      sum += v.x + v.y + v.z + v.w;
    } else {
      for (int k = 0; k < 4; ++k)
        if (c0 + k < m) sum += cnt[c0 + k];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) sWarp[warp] = sum;
  __syncthreads();
  if (tid == 0) {
    unsigned t = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) t += sWarp[w];
    tileCnt[blockIdx.x] = t;
  }
}

}  // namespace

// First step of a batch: scene of particle i from sceneOf, integrate in the
// scene's box, global cell id = the scene's cellBase + local hash.
template <bool kRadiusFromW>
__global__ void __launch_bounds__(256)
kBatchIntegrateHashCount(const BatchScene *scenes,
                         const unsigned *sceneOf, float4 *pos,
                         float4 *vel, float dt, unsigned *hash,
                         unsigned *rank, unsigned *cnt, unsigned n) {
  chainTrigger();
  chainWait();
  unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const BatchScene &S = scenes[sceneOf[i]];
  const SimParams &P = S.p;
  float4 p4 = pos[i], v4 = vel[i];
  float3 p = make_float3(p4.x, p4.y, p4.z), v = make_float3(v4.x, v4.y, v4.z);
  float r = kRadiusFromW ? p4.w : P.particleRadius;
  integrateOneBox(p, v, dt, r, P, S.lo, S.hi);
  pos[i] = make_float4(p.x, p.y, p.z, p4.w);
  vel[i] = make_float4(v.x, v.y, v.z, v4.w);
  int3 g = gridPos(p.x, p.y, p.z, P);
  unsigned h = S.cellBase + gridHash(g.x, g.y, g.z, P);
  hash[i] = h;
  rank[i] = atomicAdd(cnt + h, 1u);
}

// Buffers of the pipeline, kept in the context between calls: cnt (all zero
// between calls) and off over numCells + 1 cells, ranks and slots over the
// particles, and the scan's look-back words.
static bool countBuffers(Context &c, unsigned n, unsigned numCells, CountBuffers &b) {
  return countBuffersIn(c.countBuf, c.countBytes, c.countCells, n, numCells, b);
}

bool countBuffersIn(void *&buf, size_t &bytes, unsigned &cells, unsigned n, unsigned numCells,
                    CountBuffers &b) {
  const size_t m = (size_t)numCells + 1;
  const unsigned tiles = (unsigned)((m + kScanTile - 1) / kScanTile);
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const unsigned largeCap = largeCapacity(n);
  const unsigned tileBlocks = (tiles + kTileBlock - 1) / kTileBlock;
  const size_t need = 2 * al(m * 4) + al((size_t)n * 4) + al((size_t)n * 16) + 3 * al((size_t)(tiles + 1) * 4) +
                      al(((size_t)largeCap + 1) * 4) + al((size_t)tileBlocks * 4) +
                      al((size_t)kBitmapSlots * 2 * bitmapWords(n) * 4);
  if (buf == nullptr || bytes < need || cells != numCells) {
    if (!cudaOk(cudaDeviceSynchronize())) return false;
    if (buf) cudaFree(buf);
    buf = nullptr;
    bytes = 0;
    if (cudaMalloc(&buf, need) != cudaSuccess) {
      cudaGetLastError();
      buf = nullptr;
      setError(FCDEM_ERR_ALLOC);
      return false;
    }
    // cnt starts at zero, and no tile's offsets are known yet (see scanTile);
    // done when this returns, so that any stream may use the buffer next
    const size_t prevAt = 2 * al(m * 4) + 2 * al((size_t)(tiles + 1) * 4);
    if (!clearNow(buf, 0, need) ||
        !clearNow((char *)buf + prevAt, 0xff, (size_t)(tiles + 1) * 4))
      return false;
    bytes = need;  // the buffer counts from here on
    cells = numCells;
  }
  // The arrays that must stay zero between calls (cnt, tileCnt) sit first,
  // at offsets that depend on the cell count only, so that a call with
  // another particle count reuses them in place.
  char *p = (char *)buf;
  b.cnt = (unsigned *)p;
  p += al(m * 4);
  b.tileCnt = (unsigned *)p;
  p += al((size_t)(tiles + 1) * 4);
  b.off = (unsigned *)p;
  p += al(m * 4);
  b.tileOff = (unsigned *)p;
  p += al((size_t)(tiles + 1) * 4);
  b.tileOffPrev = (unsigned *)p;
  p += al((size_t)(tiles + 1) * 4);
  b.rank = (unsigned *)p;
  p += al((size_t)n * 4);
  b.slots = (uint4 *)p;
  p += al((size_t)n * 16);
  b.large = (unsigned *)p;
  b.largeCap = largeCap;
  p += al(((size_t)largeCap + 1) * 4);
  b.tileBlockSum = (unsigned *)p;
  p += al((size_t)tileBlocks * 4);
  b.bitmaps = (unsigned *)p;  // cleared where used (kFixupLarge)
  b.work = nullptr;
  b.scanTiles = tiles;
  return true;
}

// Up to this many particles tiles are counted with atomics (one per distinct
// tile of a warp) instead of a pass over all cells.  The pass reads the cells
// (14 us for 16.7M); the atomics of particles in random order queue on the tile
// counters.  One staged step, atomics / pass: 262,144 spheres in lattice order
// 72 / 88 us, 400,000 in random order 159 / 142.
constexpr unsigned kTileAtomicsMax = 1u << 18;

bool countPipelineBegin(Context &c, float4 *pos, float4 *vel, float dt, unsigned *hash,
                        unsigned n, unsigned numCells, const KParams &kp, CountBuffers &b) {
  if (!countBuffers(c, n, numCells, b)) return false;
  const bool tiles = n <= kTileAtomicsMax;
  launchChained(true, tiles ? kIntegrateHashCount<true> : kIntegrateHashCount<false>,
                (n + 255) / 256, 256, 0, pos, vel, dt, hash, b.rank, b.cnt, b.tileCnt, n, kp);
  if (!launchOk()) return false;
  if (tiles) return true;
  launchChained(true, kTileReduce, b.scanTiles, kScanThreads, 0, b.cnt, b.tileCnt, numCells + 1);
  return launchOk();
}

bool countPipelineBeginBatch(const BatchScene *scenes, const unsigned *sceneOf, bool radiusFromW,
                             float4 *pos, float4 *vel, float dt, unsigned *hash, unsigned n,
                             unsigned numCells, const CountBuffers &b) {
  launchChained(true, radiusFromW ? kBatchIntegrateHashCount<true> : kBatchIntegrateHashCount<false>,
                (n + 255) / 256, 256, 0, scenes, sceneOf, pos, vel, dt, hash, b.rank, b.cnt, n);
  if (!launchOk()) return false;
  launchChained(true, kTileReduce, b.scanTiles, kScanThreads, 0, b.cnt, b.tileCnt, numCells + 1);
  return launchOk();
}

// scan + scatter + fix-up/gather for one step (the counts are in place).
// hashN/rankN/origOf/prevPos/prevVel are indexed by the previous order's
// entries (origOf == nullptr: entry i is particle i, the first step).
// crowdCount (optional): collide's two group counters, cleared on the way.
bool countPipelineSort(Context &c, const CountBuffers &b, const unsigned *origOf,
                       const float4 *prevPos, const float4 *prevVel, unsigned *hash,
                       unsigned *index, float4 *sortedPos, float4 *sortedVel, unsigned n,
                       unsigned numCells, unsigned *crowdCount) {
  const unsigned m = numCells + 1;
  const bool own = b.scanTiles <= kTilesOwnPrefix;
  if (own) {
    launchChained(true, kScanCellsOwn, b.scanTiles, kScanThreads, 0, b.cnt, b.off, m, b.tileCnt,
                  b.tileOffPrev, b.large, crowdCount);
    if (!launchOk()) return false;
  } else {
    if (b.scanTiles <= kTilesOneCta) {
      launchChained(true, kScanTiles, 1, 1024, 0, b.tileCnt, b.tileOff, b.scanTiles, b.large,
                    crowdCount);
      if (!launchOk()) return false;
    } else {
      const unsigned blocks = (b.scanTiles + kTileBlock - 1) / kTileBlock;
      launchChained(true, kScanTileBlocks, blocks, kTileBlock, 0, b.tileCnt, b.tileOff, b.scanTiles,
                    b.tileBlockSum, b.large, crowdCount);
      if (!launchOk()) return false;
      launchChained(true, kAddTileBlocks, blocks, kTileBlock, 0, b.tileOff, b.scanTiles,
                    b.tileBlockSum);
      if (!launchOk()) return false;
    }
    const unsigned ctas = std::min(b.scanTiles, std::max(kScanCtas, (b.scanTiles + 31u) / 32u));
    launchChained(true, kScanCellsMany, ctas, kScanThreads, 0, b.cnt, b.off, m, b.scanTiles, b.tileOff,
                  b.tileOffPrev);
    if (!launchOk()) return false;
  }
  // hash holds the new hashes in entry order until the fix-up overwrites it
  launchChained(true, kScatterCells, (n + 255) / 256, 256, 0, hash, b.rank, origOf, b.off, b.slots, n,
                numCells, b.tileCnt, own ? b.scanTiles : 0u, c.dStatus);
  if (!launchOk()) return false;
  launchChained(true, kFixupGather, (n + 255) / 256, 256, 0, b.slots, b.off, hash, index,
                 sortedPos, sortedVel, prevPos, prevVel, n, numCells,
                fixupMaxCell(n), b.large,
                b.largeCap, c.dStatus);
  if (!launchOk()) return false;
  if (n <= kFixupAllCells) return true;  // no cell is left
  // Returns at once when the fix-up listed no cell (the common case).
  launchChained(true, kFixupLarge<false>, largeCtas(n), kLargeThreads, 0, b.slots, b.off, b.large,
                b.largeCap, hash, index, sortedPos, sortedVel, prevPos, prevVel, n,
                keyBits(n), b.bitmaps, nullptr, Giants{});
  return launchOk();
}

static_assert(((1u << kCountSortBits) >> kTileShift) + 1 <= kTilesOwnPrefix, "tiles of a key width");
constexpr unsigned kCountSortMax = 1u << 21;  // pairs
// Pairs per cell.  Fuller tables are left to the radix sort, whatever the keys: 2M
// pairs over 512 cells 484 us here, 85 there, 100,003 (195 a cell) 48 each.
constexpr unsigned kCountSortFill = 64;

// Buffers of countSortPairs.  A recorded graph may hold their addresses, so
// they live as long as those of the radix sort: each key width has its own
// cell tables (8 * 2^bits bytes: 134 MB at 24 bits, twice that over all
// widths), which are got once and never moved, and what belongs to the pairs is
// in the scratch block, which only grows with the number of pairs.  That block
// is taken large enough for the radix sort too, which can then step in while a
// graph is captured at a key width that has no tables yet.  False, without an
// error: nothing to be had (or to be got during a capture).
static bool sortBuffers(Context &c, unsigned n, int bits, CountBuffers &b) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t m = ((size_t)1 << bits) + 1;
  const unsigned tiles = (unsigned)((m + kScanTile - 1) / kScanTile);
  const unsigned largeCap = largeCapacity(n);
  const size_t cellBytes = al(m * 4), tileBytes = al((size_t)tiles * 4);
  const size_t rankBytes = al((size_t)n * 4), slotBytes = al((size_t)n * 16),
               largeBytes = al(((size_t)largeCap + 1) * 4),
               giantBytes = al(((size_t)kGiants * (largeCtas(n) + 1) + 1) * 4);
  const size_t pairBytes = std::max(rankBytes + 2 * slotBytes + largeBytes + giantBytes +
                                        (size_t)kBitmapSlots * 2 * bitmapWords(n) * 4,
                                    radixScratchBytes(n));
  void *&tables = c.sortTables[bits];
  if (!tables || c.scratchBytes < pairBytes) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(curStream(), &cap) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (cap != cudaStreamCaptureStatusNone) return false;
  }
  if (!tables) {
    void *got = nullptr;
    if (cudaMalloc(&got, 2 * (cellBytes + tileBytes)) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    // the counts start at zero, and no tile's offsets are known yet (scanTile)
    if (!clearNow(got, 0, 2 * cellBytes + tileBytes) ||
        !clearNow((char *)got + 2 * cellBytes + tileBytes, 0xff, tileBytes)) {
      cudaFree(got);
      return false;
    }
    tables = got;
  }
  char *p = (char *)scratch(c, pairBytes, true);
  if (!p) return false;
  char *t = (char *)tables;
  b = CountBuffers{};
  b.cnt = (unsigned *)t;
  b.off = (unsigned *)(t + cellBytes);
  b.tileCnt = (unsigned *)(t + 2 * cellBytes);
  b.tileOffPrev = (unsigned *)(t + 2 * cellBytes + tileBytes);
  b.scanTiles = tiles;
  b.slots = (uint4 *)p;
  b.work = p + slotBytes;
  b.rank = (unsigned *)(p + 2 * slotBytes);
  b.large = (unsigned *)(p + 2 * slotBytes + rankBytes);
  b.largeCap = largeCap;
  b.giants = (unsigned *)(p + 2 * slotBytes + rankBytes + largeBytes);
  b.bitmaps = (unsigned *)(p + 2 * slotBytes + rankBytes + largeBytes + giantBytes);
  return true;
}

// sortParticles' stable sort of n (key, value) pairs by the low `bits` bits as
// a counting sort over 2^bits cells, in place; keys with higher bits raise
// kStatusKeyRange.  False (nothing done): more than kCountSortBits bits,
// kCountSortMax pairs or kCountSortFill pairs per cell, or no buffers -- the radix
// sort then takes the pairs.
// Five short passes instead of a histogram and three look-back passes of eight
// bits, whose chain over the tiles is what they wait for.  A staged step with
// it / with the radix sort: 3,000 spheres in a 64^3 grid 59 / 73 us, 100,003 packed
// in a 128^3 grid 87 / 106, 1M falling in a 256^3 grid 188 / 210 (shuffled 198 /
// 204), 2M packed there 427 / 437 (shuffled 449 / 448), 4.2M 901 / 892 (hence the
// bound).  Spheres all over a 256^3 grid touch all of its 4,097 tiles: 300,000 take
// 187 / 171 us, 1M 293 / 260; in a 128^3 grid 105 / 126 and 213 / 234.  The fused
// step's buffers are others: it may run on another stream.
bool countSortPairs(Context &c, unsigned *keys, unsigned *vals, unsigned n, int bits) {
  if (bits > kCountSortBits || n > kCountSortMax || (n >> bits) > kCountSortFill) return false;
  const unsigned cells = 1u << bits, mask = cells - 1u;
  CountBuffers b;
  if (!sortBuffers(c, n, bits, b)) return false;
  const unsigned blocks = (n + 255) / 256;
  const bool tiles = n <= kTileAtomicsMax, large = n > kFixupAllCells;
  Giants giants{};
  giants.least = ~0u;
  if (large) {
    giants.parts = largeCtas(n);
    giants.part = (n + giants.parts - 1) / giants.parts;
    giants.count = b.giants;
    giants.first = b.giants + kGiants * giants.parts;
    giants.least = std::max((n + kGiants - 1) / kGiants, kFixupMaxCell + 1);
  }
  launchChained(true, tiles ? kCountKeys<true> : kCountKeys<false>, blocks, 256, 0, keys, n, mask,
                b.rank, b.cnt, b.tileCnt, giants, c.dStatus);
  if (!launchOk()) return true;  // recorded
  if (!tiles) {
    launchChained(true, kTileReduce, b.scanTiles, kScanThreads, 0, b.cnt, b.tileCnt, cells + 1);
    if (!launchOk()) return true;
  }
  launchChained(true, kScanCellsOwn, b.scanTiles, kScanThreads, 0, b.cnt, b.off, cells + 1, b.tileCnt,
                b.tileOffPrev, b.large, nullptr);
  if (!launchOk()) return true;
  launchChained(true, kScatterPairs, blocks, 256, 0, keys, vals, b.rank, b.off, b.slots, n, mask,
                b.tileCnt, b.scanTiles, giants);
  if (!launchOk()) return true;
  launchChained(true, kFixupPairs, blocks, 256, 0, b.slots, b.off, keys, vals, n, mask,
                fixupMaxCell(n), giants.least, b.large, b.largeCap, c.dStatus);
  if (!launchOk() || !large) return true;
  launchChained(true, kFixupLarge<true>, largeCtas(n), kLargeThreads, 0, b.slots, b.off, b.large,
                b.largeCap, keys, vals, (float4 *)b.work, nullptr, nullptr, nullptr, n, keyBits(n),
                b.bitmaps, b.rank, giants);
  launchOk();
  return true;
}

bool countPipelineTables(const CountBuffers &b, unsigned *cellStart, unsigned *cellEnd,
                         unsigned numCells) {
  unsigned blocks = numCells / 1024 + 1;
  if (blocks > numSms() * 16u) blocks = numSms() * 16u;
  const bool vec = ((uintptr_t)cellStart & 15u) == 0;
  launchChained(true, vec ? kCellTables<true> : kCellTables<false>, blocks, 256, 0, b.off, cellStart, cellEnd, numCells);
  return launchOk();
}

}  // namespace fcdem
