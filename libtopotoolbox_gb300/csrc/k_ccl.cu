// gwdt_computecosts (src/gwdt.c:167-278) on the GPU.
//
// Flat pixels are labelled into 8-connected components with a lock-free
// union-find: every label points at a smaller or equal linear index, and a
// union links the larger root under the smaller one with atomicMin, retrying
// when another thread relinked it first.  The maximum depth
// (filled - original) of each component is an order-independent maximum,
// taken with atomicMax on an order-preserving integer image of the float, so
// the costs
//
//     cost = (float)((double)(float)(maxdepth - depth) + 0.1)
//
// are bit-identical to the reference (the difference is taken in float and
// the 0.1 offset added in double, src/gwdt.c:247-277).  The label stored in
// `conncomps` is the smallest linear index among the component's pixels of
// maximal depth; the reference picks one of those pixels by its scan-order
// union-find (src/gwdt.c:141-153), which can differ when depths tie.
//
// Work decomposition: one block per 32 x 32 tile labels the tile's internal
// edges in shared memory (with path halving) and reduces each tile-local
// component to its maximum depth and the smallest pixel attaining it; only
// edges that cross tile borders touch the global union-find, and the global
// maximum / argmax take one atomic per (tile, component), not per pixel.
#include <algorithm>
#include <climits>

#include "tt_internal.cuh"

namespace tt {
namespace {

__device__ __forceinline__ int ordered_key(float x) {
  int b = __float_as_int(x);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float key_to_float(int k) {
  return __int_as_float(k >= 0 ? k : k ^ 0x7fffffff);
}

// Root of x; labels always point at smaller or equal indices.  Path halving
// only ever lowers a label (atomicMin), so it is safe under concurrent unions.
__device__ __forceinline__ int uf_find(int *L, int x) {
  volatile int *vL = L;
  int p = vL[x];
  while (p != x) {
    int gp = vL[p];
    if (gp < p) atomicMin(&L[x], gp);
    x = p;
    p = gp;
  }
  return x;
}

// Unites the components of a and b.  The greater label, where it is a root,
// goes under the other one wherever that stands in its tree, so a row of tiles
// that lie in one flat is linked up without a walk (the borders of a row or
// column of 2^20 pixels 4 us; 1.6 to 2.1 ms when each union looked for both
// roots first, up a chain of thousands of tiles); only where the greater one has
// been linked before are the roots looked for.
__device__ void uf_union(int *L, int a, int b) {
  volatile int *vL = L;
  a = vL[a];
  b = vL[b];
  for (int it = 0; it < (1 << 30) && a != b; it++) {
    const int hi = max(a, b), lo = min(a, b);
    if (vL[hi] == hi) {
      const int old = atomicMin(&L[hi], lo);
      if (old == hi) return;
      a = old;
      b = lo;
    } else {
      a = uf_find(L, a);
      b = uf_find(L, b);
    }
  }
}

constexpr int kCclThreads = 128;
constexpr int kSlots = kTile * kTile / 2;          // run slots of a tile (see CclTile)
constexpr int kSlotsPer = kSlots / kCclThreads;    // 4 a thread
constexpr int kMaxRoots = (kTile / 2) * (kTile / 2);  // 8-connected components of a tile

// Shared-memory union-find over run slots (see ccl_tile_kernel).
__device__ __forceinline__ int sfind(int *lab, int x) {
  volatile int *v = lab;
  int p = v[x];
  while (p != x) {
    const int gp = v[p];
    if (gp < p) atomicMin(&lab[x], gp);
    x = p;
    p = gp;
  }
  return x;
}

// Roots first: a link at the raw label, as across tiles, deepens the trees, on
// which a small grid's slowest tile waits (300^2 of noise 14.6 -> 16.8 us, 1024^2
// of metre steps 20 -> 23; 4096^2 196 -> 184).
__device__ void sunion(int *lab, int a, int b) {
  for (int it = 0; it < 4096; it++) {
    a = sfind(lab, a);
    b = sfind(lab, b);
    if (a == b) return;
    if (a < b) {
      const int old = atomicMin(&lab[b], a);
      if (old == b) return;
      b = old;
    } else {
      const int old = atomicMin(&lab[a], b);
      if (old == a) return;
      a = old;
    }
  }
}

// Bits s.. of the run of set bits that starts at bit s of m.
__device__ __forceinline__ uint32_t run_mask(uint32_t m, int s) {
  const uint32_t tail = ~(m >> s);
  const int len = tail ? __ffs(tail) - 1 : 32 - s;
  return len >= 32 ? 0xffffffffu : (((1u << len) - 1u) << s);
}

// Start bit of the run containing bit b (b set in m, starts = run starts).
__device__ __forceinline__ int run_start(uint32_t starts, int b) {
  const uint32_t below = starts & (b == 31 ? 0xffffffffu : ((2u << b) - 1u));
  return 31 - __clz(below);
}

// A component's maximum depth key and the smallest tile index attaining it,
// packed so that one 64-bit maximum reduces both: the key (sign flipped to
// order as unsigned) above, 1023 - index below.  0 means no key.
__device__ __forceinline__ unsigned long long pack_best(int key, int loc) {
  return ((unsigned long long)((unsigned)key ^ 0x80000000u) << 32) | (unsigned)(1023 - loc);
}

// Two run starts of a column are at least two rows apart, so column * 16 +
// (first row) / 2 numbers the runs of a tile: 512 slots.
struct CclTile {
  uint32_t mask[kTile];               // flat mask of each column (bit = row)
  int lab[kSlots];                    // union-find over run slots
  int key[kTile * kTile];             // per pixel: depth key (INT_MIN: none)
  unsigned long long best[kSlots];    // per root slot: the component's pack_best
  int warp_roots[kCclThreads / 32];
  int base;
};

// A tile-local component: its root pixel (the first pixel of its first run),
// its largest depth key and the smallest pixel attaining it (INT_MAX: none).
struct __align__(16) LocalRoot {
  int pixel, key, arg, pad;
};

// The component of root pixel gp in the tile at (i0, j0), v its pack_best.
__device__ __forceinline__ LocalRoot local_root(int gp, unsigned long long v, int64_t i0,
                                                int64_t j0, int64_t m) {
  const int a = 1023 - (int)(v & 1023u);
  return LocalRoot{gp, v ? (int)((unsigned)(v >> 32) ^ 0x80000000u) : INT_MIN,
                   v ? (int)((j0 + a / kTile) * m + (i0 + a % kTile)) : INT_MAX, 0};
}

__device__ __forceinline__ uint32_t run_starts(uint32_t m) { return m & ~(m << 1); }
// First row of the run in slot k of a column with run starts s, -1 without one.
__device__ __forceinline__ int slot_row(uint32_t s, int k) {
  const uint32_t two = (s >> (2 * k)) & 3u;
  return two ? 2 * k + (int)(two >> 1) : -1;
}

// One block of four warps per tile.  A vertical run of flats is connected by
// construction, so the union-find only runs over runs, uniting each run with
// the runs of the column before that touch it (8-connectivity = its extent
// grown by one row).  Threads take run slots, four each, so that the serial
// parts -- unions, and a run's best pixel -- are at most four runs a thread;
// a warp per tile with a lane per column stepped through up to sixteen, half
// of its lanes idle (14.7 of 32 active), and took 39 us for any grid, however
// small.  (512^2 39 -> 17 us, 4096^2 191 -> 174 us, 16384^2 2.64 -> 2.31 ms, and
// 1.97 with the tiles inside a flat taken as a whole; ten blocks an SM: 2.45 ms
// with eight, 2.25 with fourteen, which is slower on the smaller grids.)
// Each tile-local component is reduced to its maximum depth and the smallest
// pixel attaining it, and every flat pixel takes its component's root.
__global__ void __launch_bounds__(kCclThreads, 10)
ccl_tile_kernel(int *__restrict__ L, unsigned long long *__restrict__ best,
                LocalRoot *__restrict__ roots, int *__restrict__ nroots,
                uint4 *__restrict__ edges, const int32_t *__restrict__ flats,
                const float *__restrict__ orig, const float *__restrict__ filled, int64_t m,
                int64_t n, int tm) {
  __shared__ CclTile t;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = blockIdx.x;
  const int64_t i0 = (int64_t)(tile % tm) * kTile, j0 = (int64_t)(tile / tm) * kTile;
  const int64_t i = i0 + lane;  // pixels: lane = row, eight columns a warp
  constexpr int kCols = kTile / (kCclThreads / 32);
  bool some = false;
  {
    // every load of the thread in flight at once, from a clamped, always
    // valid address
    const int64_t icl = i < m ? i : m - 1;
    int fv[kCols];
    float fl[kCols], og[kCols];
#pragma unroll
    for (int u = 0; u < kCols; u++) {
      const int64_t j = j0 + warp * kCols + u;
      const int64_t p = (j < n ? j : n - 1) * m + icl;
      fv[u] = flats[p];
      fl[u] = filled[p];
      og[u] = orig[p];
    }
#pragma unroll
    for (int q = 0; q < kSlotsPer; q++) t.lab[tid + q * kCclThreads] = tid + q * kCclThreads;
#pragma unroll
    for (int u = 0; u < kCols; u++) {
      const int jj = warp * kCols + u;
      const bool f = i < m && j0 + jj < n && (fv[u] & 1);
      int k = INT_MIN;
      if (f) {
        const float d = __fsub_rn(fl[u], og[u]);
        if (!isnan(d)) k = ordered_key(d);
      }
      t.key[jj * kTile + lane] = k;
      const uint32_t b = __ballot_sync(0xffffffffu, f);
      if (lane == 0) t.mask[jj] = b;
      some |= f;
    }
  }
  some = __syncthreads_or(some);
  if (warp == 0) {  // the tile's edge flat masks for the border pass: top and
                    // bottom row (bit = column), left and right column (bit = row)
    const uint32_t mk = t.mask[lane];
    const uint32_t top = __ballot_sync(0xffffffffu, mk & 1u);
    const uint32_t bottom = __ballot_sync(0xffffffffu, (mk >> 31) & 1u);
    if (lane == 0) edges[tile] = make_uint4(top, bottom, t.mask[0], t.mask[kTile - 1]);
  }
  if (!some) return;  // no labels: L is only ever read at flat pixels

  // A tile inside a flat is one component, of runs as long as they get, each of
  // which one thread would scan: 4096^2 pixels of one flat 226 -> 55 us, a row
  // of 2^20 262 -> 85 us, 16384^2 of metre steps 3.37 -> 2.86 ms.
  const uint32_t all_rows = m - i0 >= kTile ? 0xffffffffu : (1u << (m - i0)) - 1u;
  if (__all_sync(0xffffffffu, j0 + lane >= n || t.mask[lane] == all_rows)) {
    const int first = (int)(j0 * m + i0);  // the root
    int km = INT_MIN, kl = 0;
#pragma unroll
    for (int u = 0; u < kCols; u++) {
      const int jj = warp * kCols + u, k = t.key[jj * kTile + lane];
      if (i < m && j0 + jj < n) L[(j0 + jj) * m + i] = first;
      if (k > km) {
        km = k;
        kl = jj * kTile + lane;
      }
    }
    const int most = __reduce_max_sync(0xffffffffu, km);
    const int at = __reduce_min_sync(0xffffffffu, km == most ? kl : INT_MAX);
    if (lane == 0) t.best[warp] = most == INT_MIN ? 0ULL : pack_best(most, at);
    __syncthreads();
    if (tid == 0) {
      unsigned long long v = t.best[0];
      for (int w = 1; w < kCclThreads / 32; w++) v = max(v, t.best[w]);
      roots[atomicAdd(nroots, 1)] = local_root(first, v, i0, j0, m);
      best[first] = 0ULL;
    }
    return;
  }

#pragma unroll
  for (int q = 0; q < kSlotsPer; q++) {  // unions with the column before
    const int slot = tid + q * kCclThreads, c = slot >> 4;
    const uint32_t M = t.mask[c];
    const int s0 = slot_row(run_starts(M), slot & 15);
    if (s0 < 0 || c == 0) continue;
    const uint32_t M1 = t.mask[c - 1], S1 = run_starts(M1);
    const uint32_t rm = run_mask(M, s0);
    uint32_t ov = M1 & (rm | (rm << 1) | (rm >> 1));
    while (ov) {
      const int s1 = run_start(S1, __ffs(ov) - 1);
      sunion(t.lab, (c - 1) * 16 + (s1 >> 1), slot);
      ov &= ~run_mask(M1, s1);
    }
  }
  __syncthreads();

  // Every run finds its root and its best (largest key, first pixel attaining
  // it); roots start the reduction with their own.
  unsigned long long mine[kSlotsPer];
  int root[kSlotsPer], nroot = 0;
#pragma unroll
  for (int q = 0; q < kSlotsPer; q++) {
    const int slot = tid + q * kCclThreads, c = slot >> 4;
    const uint32_t M = t.mask[c];
    const int s0 = slot_row(run_starts(M), slot & 15);
    root[q] = -1;
    mine[q] = 0ULL;
    if (s0 < 0) continue;
    root[q] = sfind(t.lab, slot);
    int km = INT_MIN, kl = 0;
    for (uint32_t b = run_mask(M, s0); b; b &= b - 1) {
      const int loc = c * kTile + __ffs(b) - 1;
      const int k = t.key[loc];
      if (k > km) {  // strictly: the first (smallest) pixel keeps a tie
        km = k;
        kl = loc;
      }
    }
    if (km != INT_MIN) mine[q] = pack_best(km, kl);
    if (root[q] == slot) {
      t.best[slot] = mine[q];
      nroot++;
    }
  }
  int incl = nroot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) t.warp_roots[warp] = incl;
  __syncthreads();
  if (tid == 0) {  // one reservation per tile in the list of local roots
    int total = 0;
    for (int w = 0; w < kCclThreads / 32; w++) total += t.warp_roots[w];
    t.base = atomicAdd(nroots, total);
  }
#pragma unroll
  for (int q = 0; q < kSlotsPer; q++) {
    const int slot = tid + q * kCclThreads;
    if (root[q] < 0) continue;
    if (root[q] != slot) {
      t.lab[slot] = root[q];  // for the pixels below
      if (mine[q]) atomicMax(&t.best[root[q]], mine[q]);
    }
  }
  __syncthreads();

  int at = t.base + incl - nroot;
  for (int w = 0; w < warp; w++) at += t.warp_roots[w];
#pragma unroll
  for (int q = 0; q < kSlotsPer; q++) {
    const int slot = tid + q * kCclThreads, c = slot >> 4;
    if (root[q] != slot) continue;
    const int gp = (int)((j0 + c) * m + i0 + slot_row(run_starts(t.mask[c]), slot & 15));
    roots[at++] = local_root(gp, t.best[slot], i0, j0, m);
    best[gp] = 0ULL;
  }
#pragma unroll
  for (int u = 0; u < kCols; u++) {  // labels, coalesced per column
    const int jj = warp * kCols + u;
    const uint32_t M = t.mask[jj];
    if (!((M >> lane) & 1u)) continue;  // L is only ever read at flat pixels
    const int r = t.lab[jj * 16 + (run_start(run_starts(M), lane) >> 1)];
    const int rc = r >> 4;
    L[(j0 + jj) * m + i] =
        (int)((j0 + rc) * m + i0 + slot_row(run_starts(t.mask[rc]), r & 15));
  }
}

// Edges that cross tile borders, from the tiles' edge masks (bit k of a row
// mask is column k, of a column mask row k).  Flat pixels next to each other
// along one tile edge are already connected inside the tile, so a border
// needs one union per pair of touching runs (8-connectivity: a run on one
// side touches the other side's pixels from one position before its start to
// one after its end), not one per pixel.
// Per tile: the border with the tile below (its bottom row against their
// top row), the border with the tile to the right (right column against
// their left column), and the two corners: (31, 31) against (0, 0) of the
// tile below-right, (31, 0) against (0, 31) of the tile below-left.
//
// A warp takes `per` tiles and a lane a run at a time of all their borders.  A
// union is a chain of dependent accesses, so on small grids the pass takes as
// long as the most unions in one thread (512^2 9 us with a tile a warp, 17 with
// four, 65 with 32), and on large ones, where most tiles have few runs or none,
// as long as the warps that find few: 16384^2 of metre steps 358, 264, 225, 250
// and 317 us with 1, 2, 4, 8 and 32 tiles a warp, of noise 219, 148, 103, 88 and
// 117.  So a tile a warp until the SMs hold 48 warps each, then up to four.
constexpr int kBorderWarps = 8;
constexpr int kBorderTiles = 4;           // most tiles a warp
constexpr int kBorderItems = 2 * 16 + 2;  // runs of two borders and two corners

struct BorderWarp {
  uint4 mask[kBorderTiles];  // bottom row, top row below, right column, left column beside
  uint16_t item[kBorderTiles * kBorderItems];  // tile << 7 | kind << 5 | first bit
};

__device__ __forceinline__ void unite_run(int *L, uint32_t a, uint32_t b, int s0, int64_t pa0,
                                          int64_t pa_step, int64_t pb0, int64_t pb_step) {
  const uint32_t sb = b & ~(b << 1);  // run starts of b
  const uint32_t rm = run_mask(a, s0);
  uint32_t ov = b & (rm | (rm << 1) | (rm >> 1));
  while (ov) {
    const int t0 = run_start(sb, __ffs(ov) - 1);
    uf_union(L, (int)(pa0 + s0 * pa_step), (int)(pb0 + t0 * pb_step));
    ov &= ~run_mask(b, t0);
  }
}

__global__ void __launch_bounds__(kBorderWarps * 32)
ccl_border_kernel(int *L, const uint4 *edges, int64_t m, int tm, int tn, int per) {
  __shared__ BorderWarp warps[kBorderWarps];
  start_after_previous();
  BorderWarp &w = warps[threadIdx.x >> 5];
  const int T = tm * tn;
  const int lane = threadIdx.x & 31;
  const int64_t first = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * per;
  if (first >= T) return;
  uint4 e = {};                              // top, bottom, left, right of this lane's tile
  uint32_t d = 0, r = 0, below = 0, above = 0;
  if (lane < per && first + lane < T) {
    const int tile = (int)first + lane, ti = tile % tm, tj = tile / tm;
    // the five tiles' masks in one round trip
    e = edges[tile];
    if (ti + 1 < tm) {
      d = edges[tile + 1].x;
      if (tj + 1 < tn) below = edges[tile + 1 + tm].x & 1u;
      if (tj > 0) above = edges[tile + 1 - tm].x >> 31;
    }
    if (tj + 1 < tn) r = edges[tile + tm].z;
  }
  if (lane < per) w.mask[lane] = make_uint4(e.y, d, e.w, r);
  const uint32_t down = d ? run_starts(e.y) : 0u, right = r ? run_starts(e.w) : 0u;
  below &= e.y >> 31;
  above &= e.y & 1u;
  const int mine = __popc(down) + __popc(right) + (int)below + (int)above;
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  int at = incl - mine;
  for (uint32_t s = down; s; s &= s - 1) w.item[at++] = (uint16_t)(lane << 7 | (__ffs(s) - 1));
  for (uint32_t s = right; s; s &= s - 1)
    w.item[at++] = (uint16_t)(lane << 7 | 1 << 5 | (__ffs(s) - 1));
  if (below) w.item[at++] = (uint16_t)(lane << 7 | 2 << 5);
  if (above) w.item[at++] = (uint16_t)(lane << 7 | 3 << 5);
  __syncwarp();
  for (int k = lane; k < total; k += 32) {
    const int item = w.item[k], s0 = item & 31;
    const int tile = (int)first + (item >> 7), ti = tile % tm, tj = tile / tm;
    const int64_t i0 = (int64_t)ti * kTile, j0 = (int64_t)tj * kTile;
    const uint4 b = w.mask[item >> 7];
    switch ((item >> 5) & 3) {
      case 0:  // bottom row (i0 + 31, j0 + k) against row i0 + 32
        unite_run(L, b.x, b.y, s0, j0 * m + i0 + kTile - 1, m, j0 * m + i0 + kTile, m);
        break;
      case 1:  // right column (i0 + k, j0 + 31) against column j0 + 32
        unite_run(L, b.z, b.w, s0, (j0 + kTile - 1) * m + i0, 1, (j0 + kTile) * m + i0, 1);
        break;
      case 2:
        uf_union(L, (int)((j0 + kTile - 1) * m + i0 + kTile - 1),
                 (int)((j0 + kTile) * m + i0 + kTile));
        break;
      default:
        uf_union(L, (int)(j0 * m + i0 + kTile - 1), (int)((j0 - 1) * m + i0 + kTile));
    }
  }
}

// A component's maximum depth key and the smallest pixel attaining it,
// packed so that one 64-bit maximum over its local roots reduces both: the
// key (sign flipped to order as unsigned) above, 2^31 - 1 - pixel below.
// 0 means no key.
__device__ __forceinline__ unsigned long long pack_root(int key, int pixel) {
  return ((unsigned long long)((unsigned)key ^ 0x80000000u) << 32) |
         (unsigned)(0x7fffffff - pixel);
}
__device__ __forceinline__ int root_key(unsigned long long v) {
  return v ? (int)((unsigned)(v >> 32) ^ 0x80000000u) : INT_MIN;
}
__device__ __forceinline__ int root_arg(unsigned long long v) {
  return v ? 0x7fffffff - (int)(unsigned)(v & 0xffffffffu) : INT_MAX;
}

// Local roots (a compact list) fold their maximum and its first pixel into
// their global root with one 64-bit maximum, and then point straight at it,
// so any flat pixel p reaches its root in two steps: L[L[p]] (every label
// above a pixel is a local root).  The roots are final here (every union
// is done), and a label only ever moves down to the root, so pointing a
// local root at it while other threads still walk through it is safe.
__global__ void ccl_root_kernel(int *L, const LocalRoot *roots,
                                const int *nroots,
                                unsigned long long *best) {
  start_after_previous();
  const int K = *nroots;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
    const int4 r = *reinterpret_cast<const int4 *>(roots + k);  // pixel, key, arg
    const int R = uf_find(L, r.x);
    if (r.y != INT_MIN) atomicMax(&best[R], pack_root(r.y, r.z));
    atomicMin(&L[r.x], R);
  }
}

// Several pixels per thread: each level of the dependent gather (a pixel's
// local root, its global root, the root's maximum and argmax) is issued for all
// before any result is used.  Two where the gwdt start is written: 16384^2
// takes 1.52 ms so, 1.65 with four and 1.93 with one; 4096^2 112, 129 and 135
// us.  Four for the costs and labels alone: 16384^2 1.41 ms, 1.53 with two (of
// metre steps 1.51 and 1.58), 512^2 4.2 and 4.9 us.  Tiles instead of runs of
// pixels (2.04 ms), 16-byte vectors of four (1.57) and roots that carry their
// component's maximum, one level less (1.96 + 0.10), were slower.  Labels are
// read at flat pixels only (the labelling writes none elsewhere); `conncomps`
// may be null (the pipeline needs the costs alone).
template <bool SEED>
__global__ void costs_kernel(float *costs,
                             ptrdiff_t *conncomps, int *L,
                             const unsigned long long *best,
                             const int32_t *flats,
                             const float *orig,
                             const float *filled, int64_t N,
                             GwdtSeed seed, int64_t m, int64_t n, int tm) {
  start_after_previous();
  constexpr int kCostPer = SEED ? 2 : 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p0 < N;
       p0 += kCostPer * stride) {
    int fv[kCostPer], l1[kCostPer], R[kCostPer], mk[kCostPer], am[kCostPer];
    float fl[kCostPer], og[kCostPer];
#pragma unroll
    for (int u = 0; u < kCostPer; u++) {
      const int64_t p = p0 + u * stride;
      fv[u] = p < N ? flats[p] : 0;
    }
    // the depths are read with the labels, at flat pixels only: the same
    // dependent level, two thirds fewer bytes where flats are a third
#pragma unroll
    for (int u = 0; u < kCostPer; u++) {
      const int64_t p = p0 + u * stride;
      const bool f = fv[u] & 1;
      l1[u] = f ? L[p] : -1;
      fl[u] = f ? filled[p] : 0.f;
      og[u] = f ? orig[p] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kCostPer; u++) R[u] = l1[u] >= 0 ? L[l1[u]] : -1;
#pragma unroll
    for (int u = 0; u < kCostPer; u++) {
      const unsigned long long v = R[u] >= 0 ? best[R[u]] : 0ULL;
      mk[u] = root_key(v);
      am[u] = root_arg(v);
    }
#pragma unroll
    for (int u = 0; u < kCostPer; u++) {
      const int64_t p = p0 + u * stride;
      if (p >= N) continue;
      float c = 0.0f;
      ptrdiff_t lab = 0;
      if (R[u] >= 0) {
        const float maxd = key_to_float(mk[u]);
        const float depth = __fsub_rn(fl[u], og[u]);
        const float diff = __fsub_rn(maxd, depth);
        c = __double2float_rn(__dadd_rn((double)diff, 0.1));
        lab = (am[u] == INT_MAX) ? R[u] : am[u];
      }
      if (SEED) {  // the gwdt start (src/gwdt.c:296-308) instead of plain costs
        const int32_t f = fv[u];
        costs[p] = (f & 1) ? c * 0.5f : NAN;  // halved: c >= 0.1, exact
        seed.dist[p] = (f & 5) == 5 ? 1.0f : (f & 1) ? INFINITY : 0.0f;
        if ((f & 5) == 5) mark_tiles_near(seed.dirty, tm, p % m, p / m, m, n);
      } else {
        costs[p] = c;
      }
      if (conncomps) conncomps[p] = lab;
    }
  }
}

int ew_grid(int64_t N) {
  int64_t b = (N + 255) / 256;
  int64_t cap = (int64_t)sm_count() * 16;
  return (int)(b < cap ? (b > 0 ? b : 1) : cap);
}

}  // namespace

tt_cuda_status costs_dev(float *costs, ptrdiff_t *conncomps,
                         const int32_t *flats, const float *orig,
                         const float *filled, const GridDims &g,
                         cudaStream_t st, const GwdtSeed *seed) {
  const int64_t N = g.cells();
  Workspace &ws = workspace();
  const int T = g.tiles();
  const size_t nr = std::min((size_t)N, (size_t)T * kMaxRoots);
  if (!ws.reserve(align_up((size_t)N * 4) + align_up((size_t)N * 8) +
                  align_up(nr * sizeof(LocalRoot)) + align_up((size_t)T * 16) + 256))
    return TT_CUDA_ERR_ALLOC;
  int *nroots = (int *)ws.take(256);
  uint4 *edges = (uint4 *)ws.take((size_t)T * 16);
  LocalRoot *roots = (LocalRoot *)ws.take(nr * sizeof(LocalRoot));
  int *L = (int *)ws.take((size_t)N * 4);
  unsigned long long *best = (unsigned long long *)ws.take((size_t)N * 8);
  const int grid = ew_grid(N);
  TT_CHECK(cudaMemsetAsync(nroots, 0, sizeof(int), st));
  // one tile per block: the block scheduler evens out tiles whose labelling
  // takes longer (many runs, many unions)
  TT_LAUNCH(ccl_tile_kernel, T, kCclThreads, 0, st, L, best, roots, nroots, edges, flats, orig,
            filled, g.m, g.n, g.tm);
  const int per = std::max(1, std::min(kBorderTiles, T / (sm_count() * 48)));
  const int bwarps = (T + per - 1) / per;
  TT_LAUNCH_NEXT(ccl_border_kernel, (bwarps + kBorderWarps - 1) / kBorderWarps,
                 kBorderWarps * 32, 0, st, L, edges, g.m, g.tm, g.tn, per);
  TT_LAUNCH_NEXT(ccl_root_kernel, grid, 256, 0, st, L, roots, nroots, best);
  const int cgrid = (int)std::min<int64_t>((N + 1023) / 1024, (int64_t)sm_count() * 32);
  if (seed)
    TT_LAUNCH_NEXT(costs_kernel<true>, cgrid, 256, 0, st, costs, conncomps, L, best,
              flats, orig, filled, N, *seed, g.m, g.n, g.tm);
  else
    TT_LAUNCH_NEXT(costs_kernel<false>, cgrid, 256, 0, st, costs, conncomps, L, best,
              flats, orig, filled, N, GwdtSeed{nullptr, nullptr}, g.m, g.n, g.tm);
  TT_CHECK(cudaGetLastError());
  return TT_CUDA_SUCCESS;
}

}  // namespace tt
