// 3x3 stencil kernels: flat/sill/presill labelling, D8 carve directions,
// second-order gradients, hillshade and the hillshade adjoint.
//
// Each input byte is read from DRAM about once: labelling and directions walk
// along the columns with their window in registers, the gradients' kernels
// read tiles of 32 x 32 pixels and a halo.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "tt_internal.cuh"

namespace tt {
namespace {

constexpr int kBlockX = 32;  // along i
constexpr int kBlockY = 8;   // along j

// ------------------------------------------------------------------
// identifyflats (src/identifyflats.c:33-121)
//
// flat(p)    = interior pixel, not NaN, and no neighbour lower, a NaN
//              neighbour counting as -INF (src/identifyflats.c:64)
// sill(s)    = !flat(s) && exists flat neighbour f with z_f == z_s
// presill(f) =  flat(f) && exists non-flat neighbour s with z_s == z_f
// (the scatter at src/identifyflats.c:83-119 restated as a gather).
//
// Neither test needs the neighbours' equality one by one.  No neighbour of a
// flat pixel lies below it, so a pixel that is not flat has a flat neighbour
// at its own elevation exactly when the highest of its flat neighbours is at
// it, and a flat pixel has a neighbour of the other kind at its elevation
// exactly when the lowest of those is.  Both are separable three-input
// minima and maxima, NaN standing for "not of this kind".
//
// A warp walks along the columns of a strip of rows, four consecutive rows per
// lane (120 of its 128 rows are put out, the outer lanes are the halo), with
// the last three columns in registers: a column's vertical neighbours come
// from the lane's own rows and one shuffle each way, the flat bits of the rows
// beside them from two ballots.  Nothing is staged in shared memory, and a
// pixel costs some 20 operations instead of the 150 of a tile staged with its
// halo, which the ALU pipe bounded (85 % busy): 16384^2 1.51 ms with eight
// compares a pixel there, 1.30 with shared minima, 0.45 so (4.8 TB/s of 2.1
// GB); 4096^2 84 -> 37 us, 3001 x 5003 75 -> 42 us, 512^2 3.1 -> 3.6 us (both
// after the 1.30).
//
// WIDE: 16-byte loads and stores, where every column starts on a 16-byte
// boundary.  Elsewhere four strided ones, which L1 and L2 put together (one
// row a lane, 28 of 32 put out, reads whole lines but repeats the bits'
// arithmetic: 57 us for the 41).  A warp takes `cols` columns, and loads and
// labels four more as its own halo.
// ------------------------------------------------------------------
constexpr int kCountSlots = 64;
constexpr int kFlatBatch = 4;  // columns loaded ahead
constexpr int kFlatWarps = 4;  // warps per block

// Three-input minimum that is NaN when any operand is.
__device__ __forceinline__ float min3_nan(float a, float b, float c) {
  float d;
  asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Three-input minimum and maximum, ignoring NaN.
__device__ __forceinline__ float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Flat test of pixel z, `lowest` the min3_nan of its 3 x 3 neighbourhood, z
// included: not NaN and no neighbour lower, a NaN neighbour counting as -INF.
// For z = -INF every neighbour passes; otherwise the minimum is z exactly
// when no neighbour is lower or NaN.
__device__ __forceinline__ bool is_flat(float lowest, float z) {
  return (lowest == z) | (z == -INFINITY);
}

// A strip takes `lanes` lanes, the outer two its halo, and puts out
// (lanes - 2) * kFlatR rows: the 32 lanes of a warp along one, or NARROW along
// several strips of `seg` lanes each, in step (see strip_split).
constexpr int kFlatR = 4;  // rows per lane

template <bool WIDE>
__device__ __forceinline__ void flat_load(float (&v)[kFlatR], const float *dem,
                                          int64_t row, int64_t j, int64_t m, int64_t n,
                                          bool rows_ok) {
#pragma unroll
  for (int r = 0; r < kFlatR; r++) v[r] = NAN;
  if (rows_ok && j >= 0 && j < n) {
    const float *p = dem + j * m + row;
    if constexpr (WIDE) {
      const float4 w = *reinterpret_cast<const float4 *>(p);
      v[0] = w.x, v[1] = w.y, v[2] = w.z, v[3] = w.w;
    } else {
#pragma unroll
      for (int r = 0; r < kFlatR; r++)
        if (row + r < m) v[r] = p[r];
    }
  }
}

template <bool WIDE, bool NARROW>
__global__ void __launch_bounds__(kFlatWarps * 32)
identifyflats_kernel(int32_t *out, const float *dem, int64_t m,
                     int64_t n, int strips, int cols, int seg, unsigned long long *slots) {
  start_after_previous();
  constexpr int R = kFlatR;
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * kFlatWarps + (threadIdx.x >> 5);
  const int lanes = NARROW ? seg : 32, sl = NARROW ? lane & (seg - 1) : lane;
  const int64_t first = NARROW ? w * (32 / seg) : w;
  const int64_t walk = NARROW ? first + lane / seg : w;
  const int64_t jb = walk / strips * cols;  // first column put out
  if ((NARROW ? first / strips * cols : jb) >= n) return;
  const int64_t row = walk % strips * ((lanes - 2) * R) + (int64_t)(sl - 1) * R;
  const bool rows_ok = row >= 0 && row < m;  // WIDE: m is a multiple of 4, all rows or none
  const bool puts = rows_ok && sl >= 1 && sl < lanes - 1;  // sl: lane of the strip
  const int64_t je = min(n, jb + cols);
  const int64_t end = NARROW ? jb + cols : je;  // the strips of a warp walk in step
  bool inner_row[R];  // interior pixels may be flat
#pragma unroll
  for (int r = 0; r < R; r++) inner_row[r] = row + r >= 1 && row + r < m - 1;
  const uint32_t lane_up = sl ? 1u << (lane - 1) : 0u;
  const uint32_t lane_dn = sl < lanes - 1 ? 2u << lane : 0u;

  float next[kFlatBatch][R];
#pragma unroll
  for (int b = 0; b < kFlatBatch; b++)
    flat_load<WIDE>(next[b], dem, row, jb - 2 + b, m, n, rows_ok);

  // Columns j - 1 and j - 2 (z), row minima of j - 1 and j - 2, vertical
  // extremes over flats (g) and others (h) of j - 2 and j - 3, flat bits of
  // j - 2, rows above and below of j - 1.
  float z1[R] = {}, z2[R] = {}, m1[R] = {}, m2[R] = {};
  float g2[R] = {}, g3[R] = {}, h2[R] = {}, h3[R] = {};
  bool f2[R] = {};
  float up1 = 0.f, dn1 = 0.f;
  unsigned cnt = 0;
  for (int64_t j0 = jb - 2; j0 < end + 2; j0 += kFlatBatch) {
    float cur[kFlatBatch][R];
#pragma unroll
    for (int b = 0; b < kFlatBatch; b++)
#pragma unroll
      for (int r = 0; r < R; r++) cur[b][r] = next[b][r];
    if (j0 + kFlatBatch < end + 2)
#pragma unroll
      for (int b = 0; b < kFlatBatch; b++)
        flat_load<WIDE>(next[b], dem, row, j0 + kFlatBatch + b, m, n, rows_ok);
#pragma unroll
    for (int b = 0; b < kFlatBatch; b++) {
      const int64_t j = j0 + b;
      const float up0 = __shfl_up_sync(0xffffffffu, cur[b][R - 1], 1, lanes);
      const float dn0 = __shfl_down_sync(0xffffffffu, cur[b][0], 1, lanes);
      // flat test of column j - 1
      float m0[R], g1[R], h1[R], G[R + 2], H[R + 2];
      bool f1[R];
      const bool inner_col = j - 1 >= 1 && j - 1 < n - 1;
#pragma unroll
      for (int r = 0; r < R; r++)
        m0[r] = min3_nan(r ? cur[b][r - 1] : up0, cur[b][r], r < R - 1 ? cur[b][r + 1] : dn0);
#pragma unroll
      for (int r = 0; r < R; r++) {
        f1[r] = is_flat(min3_nan(m2[r], m1[r], m0[r]), z1[r]) & inner_row[r] & inner_col;
        G[r + 1] = f1[r] ? z1[r] : NAN;
        H[r + 1] = f1[r] ? NAN : z1[r];
      }
      const bool fu = __ballot_sync(0xffffffffu, f1[R - 1]) & lane_up;
      const bool fd = __ballot_sync(0xffffffffu, f1[0]) & lane_dn;
      G[0] = fu ? up1 : NAN, H[0] = fu ? NAN : up1;
      G[R + 1] = fd ? dn1 : NAN, H[R + 1] = fd ? NAN : dn1;
#pragma unroll
      for (int r = 0; r < R; r++) {
        g1[r] = max3(G[r], G[r + 1], G[r + 2]);
        h1[r] = min3(H[r], H[r + 1], H[r + 2]);
      }
      // sills and presills of column j - 2
      if (j - 2 >= jb && j - 2 < je) {
        int32_t o[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
          const int sill = max3(g3[r], g2[r], g1[r]) == z2[r] ? 2 : 0;
          const int presill = min3(h3[r], h2[r], h1[r]) == z2[r] ? 5 : 1;
          o[r] = f2[r] ? presill : sill;
          if (puts && (WIDE || row + r < m)) cnt += f2[r];
        }
        if (puts) {
          int32_t *p = out + (j - 2) * m + row;
          if constexpr (WIDE)
            *reinterpret_cast<int4 *>(p) = make_int4(o[0], o[1], o[2], o[3]);
          else
#pragma unroll
            for (int r = 0; r < R; r++)
              if (row + r < m) p[r] = o[r];
        }
      }
#pragma unroll
      for (int r = 0; r < R; r++) {
        z2[r] = z1[r], z1[r] = cur[b][r];
        m2[r] = m1[r], m1[r] = m0[r];
        g3[r] = g2[r], g2[r] = g1[r];
        h3[r] = h2[r], h2[r] = h1[r];
        f2[r] = f1[r];
      }
      up1 = up0, dn1 = dn0;
    }
  }
  if (!slots) return;  // the count was not asked for
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0 && cnt) atomicAdd(&slots[w % kCountSlots], (unsigned long long)cnt);
}

__global__ void sum_slots_kernel(const unsigned long long *__restrict__ slots,
                                 unsigned long long *__restrict__ count) {
  unsigned long long v = slots[threadIdx.x] + slots[threadIdx.x + 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (threadIdx.x == 0) *count = v;
}

// ------------------------------------------------------------------
// D8 carve directions (src/flow_routing.c:15-76)
//
// z = flat ? dist : dem; neighbours higher than the centre (in dem) are
// skipped; g = (z - z_n) / chamfer with chamfer = sqrtf(2) on odd bits; the
// first strictly largest positive g wins.  The subtraction and the IEEE
// division are written with explicit round-to-nearest intrinsics so that no
// contraction changes a bit.
// ------------------------------------------------------------------
//
// The first largest slope is found without a branch per neighbour.  The
// quotient fl(d / sqrt(2)) does not decrease with d, so the largest diagonal
// difference has the largest diagonal quotient: one quotient a pixel instead
// of one for each diagonal that beats the best so far.  Another diagonal has
// the same quotient only if its difference is equal or the float before (two
// floats further the exact quotients lie 1.4 units of the last place apart).
// The direction is the first neighbour in order that reaches the largest
// slope.  Quotients are a reciprocal product with an exact remainder; a warp
// that meets a drop below 2^-100, where that remainder would underflow, stops
// and takes its columns again with divisions (4096^2 of such drops 197 us, 232
// when it went on to its last column first).
//
// Warps walk along strips of rows as in identifyflats_kernel, dem and dist of
// three columns in registers and the next one loaded ahead (three ahead take
// registers that hold more warps: 1.04 ms for 0.93 at 16384^2); 13 bytes a
// pixel.  The selects of the drops and directions bound it (ALU pipe), so the
// drops are predicated subtractions (0.93 -> 0.86 ms).  Against a tile staged
// in shared memory with its halo and a branch per neighbour:
// 16384^2 1.76 -> 0.86 ms, 4096^2 111 -> 66 us, 3001 x 5003 104 -> 65 us,
// 512^2 4.3 -> 4.1 us.
constexpr float kSq2 = 1.41421353816986083984375f;      // sqrtf(2.0f) = 0x3FB504F3
constexpr float kInvSq2 = 0.707106769084930419921875f;  // the float next to 1 / kSq2

template <bool WIDE>
__device__ __forceinline__ void flag_load(int (&f)[kFlatR], const int32_t *flats,
                                          int64_t row, int64_t j, int64_t m, int64_t n,
                                          bool rows_ok) {
#pragma unroll
  for (int r = 0; r < kFlatR; r++) f[r] = 0;
  if (rows_ok && j >= 0 && j < n) {
    const int32_t *p = flats + j * m + row;
    if constexpr (WIDE) {
      const int4 w = *reinterpret_cast<const int4 *>(p);
      f[0] = w.x, f[1] = w.y, f[2] = w.z, f[3] = w.w;
    } else {
#pragma unroll
      for (int r = 0; r < kFlatR; r++)
        if (row + r < m) f[r] = p[r];
    }
  }
}

// fl(d / sqrt(2)): the quotient by the reciprocal and one exact remainder
// (Markstein 1990: with a correctly rounded reciprocal the corrected quotient
// is correctly rounded; checked for every float from 2^-100 up).  For finite d of 2^-100
// or more, where the remainder does not underflow.
__device__ __forceinline__ float quotient_sq2(float d) {
  const float q = __fmul_rn(d, kInvSq2);
  return __fmaf_rn(__fmaf_rn(-q, kSq2, d), kInvSq2, q);
}

// Drop from the centre to a neighbour: in dist for a flat centre, unless the
// neighbour is above it; in dem otherwise (negative in that case).  As a
// predicated subtraction: a select would go to the pipe that is the busiest.
__device__ __forceinline__ float drop_to(float zc, float zn, float dc, float dn, unsigned flat) {
  float e;
  asm("{.reg .pred f, p;\n"
      " setp.ne.u32 f, %5, 0;\n"
      " setp.leu.and.f32 p, %2, %1, f;\n"
      " sub.rn.f32 %0, %1, %2;\n"
      " @p sub.rn.f32 %0, %3, %4;}"
      : "=&f"(e)
      : "f"(zc), "f"(zn), "f"(dc), "f"(dn), "r"(flat));
  return e;
}

// Direction of the pixel at row r of the window's middle column (column c of
// the window is index (first + c) % 3), in byte r of the result.  FAST: the
// quotients by quotient_sq2, and `odd` set where they may not hold (drops
// below 2^-100); otherwise by divisions.
template <unsigned ORDER, bool FAST>
__device__ __forceinline__ uint32_t pixel_direction(const float (&z)[3][kFlatR + 2],
                                                    const float (&d)[3][kFlatR + 2], int first,
                                                    int r, unsigned fl, bool &odd) {
  constexpr unsigned A = ORDER ? kD8B : kD8A, B = ORDER ? kD8A : kD8B;
  const int mid = (first + 1) % 3;
  const float zc = z[mid][r + 1], dc = d[mid][r + 1];
  float e[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int di = (int)((A >> (2 * k)) & 3u) - 1, dj = (int)((B >> (2 * k)) & 3u) - 1;
    const float zn = z[(first + 1 + dj) % 3][r + 1 + di];
    const float dn = d[(first + 1 + dj) % 3][r + 1 + di];
    e[k] = drop_to(zc, zn, dc, dn, fl);
  }
  // NaN differences lose every maximum and every comparison below; the least
  // positive float as the floor is reached by none that is not positive
  const float least = __int_as_float(1);
  float best = max3(max3(e[0], e[2], least), e[4], e[6]);
  const float dmax = max3(max3(e[1], e[3], 0.0f), e[5], e[7]);
  const int bits = __float_as_int(dmax);
  const float before = __int_as_float(bits - 1);  // NaN for dmax = 0
  float q, qb;
  if (FAST) {
    odd |= (unsigned)(bits - 1) < 0x0d800000u;
    q = dmax == INFINITY ? dmax : quotient_sq2(dmax);
    qb = quotient_sq2(before);
  } else {
    q = __fdiv_rn(dmax, kSq2);
    qb = __fdiv_rn(before, kSq2);
  }
  // the least diagonal difference that reaches the largest slope (NaN: none)
  const float reach = q >= best ? (qb == q ? before : dmax) : NAN;
  best = fmaxf(best, q);
  uint32_t dv = 0;
#pragma unroll
  for (int k = 7; k >= 0; k--)
    if ((k & 1) ? e[k] >= reach : e[k] == best) dv = 1u << (k + 8 * r);
  return dv;
}

template <unsigned ORDER, bool FAST>
__device__ __forceinline__ uint32_t column_directions(const float (&z)[3][kFlatR + 2],
                                                      const float (&d)[3][kFlatR + 2],
                                                      int first, unsigned flat, bool &odd) {
  uint32_t o = 0;
#pragma unroll
  for (int r = 0; r < kFlatR; r++)
    o |= pixel_direction<ORDER, FAST>(z, d, first, r, flat & (1u << r), odd);
  return o;
}

// Directions of columns jb .. jb + cols - 1 of the strip whose rows start at `row` in
// this lane.  Returns whether a quotient may not hold (FAST: as soon as one of the
// warp's does not).
template <unsigned ORDER, bool WIDE, bool NARROW, bool FAST>
__device__ __forceinline__ bool walk_directions(uint8_t *dir, const float *dem,
                                                const float *dist, const int32_t *flats,
                                                int64_t m, int64_t n, int64_t row, int64_t jb,
                                                int cols, int lanes, int sl) {
  constexpr int R = kFlatR;
  const bool rows_ok = row >= 0 && row < m;  // WIDE: m is a multiple of 4, all rows or none
  const bool puts = rows_ok && sl >= 1 && sl < lanes - 1;
  const int64_t je = min(n, jb + cols);
  const int64_t end = NARROW ? jb + cols : je;  // the strips of a warp walk in step

  bool odd = false;
  float nz[R], nd[R];  // the next column
  int nf[R];
  flat_load<WIDE>(nz, dem, row, jb - 1, m, n, rows_ok);
  flat_load<WIDE>(nd, dist, row, jb - 1, m, n, rows_ok);
  flag_load<WIDE>(nf, flats, row, jb - 1, m, n, rows_ok);
  // Off-grid neighbours hold NaN: their slope is NaN and never selected,
  // exactly as the reference skips them, so no bounds checks are needed.
  float z[3][R + 2] = {}, d[3][R + 2] = {};
  unsigned f[3] = {};
  for (int64_t j0 = jb - 1; j0 < end + 1; j0 += 3) {
#pragma unroll
    for (int b = 0; b < 3; b++) {
      const int64_t j = j0 + b;  // this column enters the window at index b
#pragma unroll
      for (int r = 0; r < R; r++) z[b][r + 1] = nz[r], d[b][r + 1] = nd[r];
      f[b] = 0;
#pragma unroll
      for (int r = 0; r < R; r++) f[b] |= (unsigned)(nf[r] & 1) << r;
      if (j < end) {
        flat_load<WIDE>(nz, dem, row, j + 1, m, n, rows_ok);
        flat_load<WIDE>(nd, dist, row, j + 1, m, n, rows_ok);
        flag_load<WIDE>(nf, flats, row, j + 1, m, n, rows_ok);
      }
      z[b][0] = __shfl_up_sync(0xffffffffu, z[b][R], 1, lanes);
      d[b][0] = __shfl_up_sync(0xffffffffu, d[b][R], 1, lanes);
      z[b][R + 1] = __shfl_down_sync(0xffffffffu, z[b][1], 1, lanes);
      d[b][R + 1] = __shfl_down_sync(0xffffffffu, d[b][1], 1, lanes);
      if (j - 1 >= jb && j - 1 < je) {  // directions of column j - 1
        const unsigned fm = f[(b + 2) % 3];
        const uint32_t o = column_directions<ORDER, FAST>(z, d, (b + 1) % 3, fm, odd);
        if (puts) {
          uint8_t *p = dir + (j - 1) * m + row;
          if constexpr (WIDE) {
            *reinterpret_cast<uint32_t *>(p) = o;
          } else {
#pragma unroll
            for (int r = 0; r < R; r++)
              if (row + r < m) p[r] = (uint8_t)(o >> (8 * r));
          }
        }
      }
    }
    if (FAST && __any_sync(0xffffffffu, odd)) return true;  // walked again anyway
  }
  return odd;
}

template <unsigned ORDER, bool WIDE, bool NARROW>
__global__ void __launch_bounds__(kFlatWarps * 32)
directions_kernel(uint8_t *dir, const float *dem,
                  const float *dist, const int32_t *flats, int64_t m,
                  int64_t n, int strips, int cols, int seg) {
  start_after_previous();
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * kFlatWarps + (threadIdx.x >> 5);
  const int lanes = NARROW ? seg : 32, sl = NARROW ? lane & (seg - 1) : lane;
  const int64_t first = NARROW ? w * (32 / seg) : w;
  const int64_t walk = NARROW ? first + lane / seg : w;
  const int64_t jb = walk / strips * cols;  // first column put out
  if ((NARROW ? first / strips * cols : jb) >= n) return;
  const int64_t row = walk % strips * ((lanes - 2) * kFlatR) + (int64_t)(sl - 1) * kFlatR;
  const bool odd = walk_directions<ORDER, WIDE, NARROW, true>(dir, dem, dist, flats, m, n, row,
                                                              jb, cols, lanes, sl);
  if (__any_sync(0xffffffffu, odd))  // rare: the same walk with divisions
    walk_directions<ORDER, WIDE, NARROW, false>(dir, dem, dist, flats, m, n, row, jb, cols, lanes,
                                                sl);
}

// ------------------------------------------------------------------
// Second-order gradient and hillshade (src/hillshade.c:11-213)
// ------------------------------------------------------------------
struct Grad {
  float dx, dy;
};

// Gradient along one axis at position k of len, reading the stencil values
// a(-2..2) around the centre.  Mirrors src/hillshade.c:113-155.
__device__ __forceinline__ float axis_grad(float zm2, float zm1, float z0,
                                           float zp1, float zp2, int64_t k,
                                           int64_t len, float twoh) {
  if (k == 0) return (-zp2 + 4 * zp1 - 3 * z0) / twoh;
  if (k == len - 1) return (zm2 - 4 * zm1 + 3 * z0) / twoh;
  return isnan(z0) ? NAN : (zp1 - zm1) / twoh;
}

__device__ __forceinline__ float shade(float dx, float dy, float sx, float sy,
                                       float sz) {
  float inv = 1.0f / sqrtf(dx * dx + dy * dy + 1.0f);
  return (-dx * inv) * sx + (-dy * inv) * sy + inv * sz;
}

// ------------------------------------------------------------------
// Float-float (unevaluated sum hi + lo) arithmetic for the shading.  The
// cancellation in -dx*sx - dy*sy + sz would otherwise cost up to ~1e-5 of
// relative accuracy where the shade is near zero on steep terrain; carrying
// ~44 bits keeps the result within a few float32 ulps of the FP64 formula.
// Error-free transformations: TwoSum (Knuth) and TwoProduct via FMA.
// ------------------------------------------------------------------
struct F2 {
  float hi, lo;
};

__device__ __forceinline__ F2 two_sum(float a, float b) {
  float s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return {s, e};
}
__device__ __forceinline__ F2 two_prod(float a, float b) {
  float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ F2 f2_norm(float hi, float lo) {
  float s = __fadd_rn(hi, lo);
  return {s, __fsub_rn(lo, __fsub_rn(s, hi))};
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 s = two_sum(a.hi, b.hi);
  return f2_norm(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 p = two_prod(a.hi, b.hi);
  float t = __fmaf_rn(a.hi, b.lo, __fmul_rn(a.lo, b.hi));
  return f2_norm(p.hi, __fadd_rn(p.lo, t));
}

// Exact stencil sums: the one-sided [-3 4 -1] / [1 -4 3] and central
// [-1 0 1] combinations of float32 samples, as float-float.
__device__ __forceinline__ F2 axis_diff_f2(float zm2, float zm1, float z0,
                                           float zp1, float zp2, int64_t k,
                                           int64_t len) {
  if (k == 0) {
    F2 t = f2_add(two_prod(4.0f, zp1), two_prod(-3.0f, z0));
    return f2_add(t, F2{-zp2, 0.0f});
  }
  if (k == len - 1) {
    F2 t = f2_add(two_prod(-4.0f, zm1), two_prod(3.0f, z0));
    return f2_add(t, F2{zm2, 0.0f});
  }
  return two_sum(zp1, -zm1);
}

struct Sun2 {
  float sxh, sxl, syh, syl, szh, szl;
  float rh, rl;              // 1 / (2 * cellsize) as float-float
  float axh, axl, ayh, ayl;  // sx / (2 * cellsize), sy / (2 * cellsize)
};

// 1 / sqrt(q) within about half an ulp for q >= 1: the hardware's
// approximation and one Newton step (y += y * (1 - q y^2) / 2) with the
// residual in fused arithmetic.  Not finite where q is not.
__device__ __forceinline__ float rsqrt_newton(float q) {
  const float y = rsqrtf(q);
  return __fmaf_rn(__fmul_rn(0.5f, y), __fmaf_rn(-__fmul_rn(q, y), y, 1.0f), y);
}

// Hillshade of a pixel from its central differences.  Only the numerator
// sz - dzx ax - dzy ay cancels; its terms are taken without error (the
// differences and products as unevaluated sums) and their low parts added
// once.  Not finite where any input is not.
__device__ __forceinline__ float shade_central(float xp, float xm, float yp, float ym,
                                               const Sun2 &s) {
  const F2 dx = two_sum(xp, -xm), dy = two_sum(yp, -ym);
  const F2 px = two_prod(dx.hi, -s.axh), py = two_prod(dy.hi, -s.ayh);
  const float lx = __fmaf_rn(dx.hi, -s.axl, __fmaf_rn(dx.lo, -s.axh, px.lo));
  const float ly = __fmaf_rn(dy.hi, -s.ayl, __fmaf_rn(dy.lo, -s.ayh, py.lo));
  const F2 p = two_sum(px.hi, py.hi);
  const F2 t = two_sum(p.hi, s.szh);
  const float lo = __fadd_rn(__fadd_rn(lx, ly), __fadd_rn(__fadd_rn(p.lo, t.lo), s.szl));
  const float gx = __fmul_rn(dx.hi, s.rh), gy = __fmul_rn(dy.hi, s.rh);
  const float q = __fmaf_rn(gx, gx, __fmaf_rn(gy, gy, 1.0f));
  return __fmul_rn(__fadd_rn(t.hi, lo), rsqrt_newton(q));
}


constexpr int kHS = kTile + 4;  // 2-pixel halo for one-sided borders

// Block (x, y) computes tile (x, y + jt0): a launch may cover a band of tile
// columns, whose DEM columns (plus two on each side) must be in place.
template <int MODE>  // 0: hillshade, 1: gradients
__global__ void __launch_bounds__(kBlockX * kBlockY)
hillshade_kernel(float *__restrict__ out0, float *__restrict__ out1,
                 const float *__restrict__ dem, const float *__restrict__ gout,
                 int64_t m, int64_t n, float twoh, float sx, float sy, float sz,
                 Sun2 s2, int jt0) {
  __shared__ float z[kHS][kHS + 1];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int64_t i0 = (int64_t)blockIdx.x * kTile;
  const int64_t j0 = (int64_t)(blockIdx.y + jt0) * kTile;
  // Tiles away from every grid edge use central differences only.  A thread
  // takes four pixels of a row and reads their 14 neighbours straight from
  // global memory: a line serves the three rows that need it from L1, so
  // staging it in shared memory only added stores, loads and a barrier.  The
  // kernel is bound by its arithmetic (8192^2: 330 -> 169 us; the bytes take
  // 79 us).
  if (MODE == 0 && i0 >= 1 && i0 + kTile + 1 <= m && j0 >= 1 && j0 + kTile + 1 <= n) {
    const int64_t p0 = (j0 + 4 * ty) * m + i0 + tx;
    const float *const zp = dem + p0;
    float c[6], up[4], dn[4];
#pragma unroll
    for (int u = 0; u < 6; u++) c[u] = zp[(u - 1) * m];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      up[u] = zp[u * m - 1];
      dn[u] = zp[u * m + 1];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      float h = shade_central(dn[u], up[u], c[u + 2], c[u], s2);
      if (!isfinite(h) || c[u + 1] != c[u + 1]) {  // NaN / INF exactly as the reference
        const bool nan = c[u + 1] != c[u + 1];
        const float dx = nan ? NAN : __fdiv_rn(__fsub_rn(dn[u], up[u]), twoh);
        const float dy = nan ? NAN : __fdiv_rn(__fsub_rn(c[u + 2], c[u]), twoh);
        h = shade(dx, dy, sx, sy, sz);
      }
      out0[p0 + u * m] = h;
    }
    return;
  }
  {  // stage the DEM with every load in flight at once
    constexpr int kC = (kHS + kBlockY - 1) / kBlockY;
    float v[kC][2];
#pragma unroll
    for (int k = 0; k < kC; k++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = ty + k * kBlockY, r = tx + h * kBlockX;
        const int64_t i = i0 - 2 + r, j = j0 - 2 + c;
        v[k][h] = (c < kHS && r < kHS && i >= 0 && i < m && j >= 0 && j < n) ? dem[j * m + i] : 0.0f;
      }
#pragma unroll
    for (int k = 0; k < kC; k++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = ty + k * kBlockY, r = tx + h * kBlockX;
        if (c < kHS && r < kHS) z[c][r] = v[k][h];
      }
  }
  __syncthreads();
  for (int c = ty; c < kTile; c += kBlockY) {
    int64_t j = j0 + c;
    int64_t i = i0 + tx;
    if (j >= n || i >= m) continue;
    int r = tx + 2, cc = c + 2;
    int64_t p = j * m + i;
    {
      float dx = axis_grad(z[cc][r - 2], z[cc][r - 1], z[cc][r], z[cc][r + 1],
                           z[cc][r + 2], i, m, twoh);
      float dy = axis_grad(z[cc - 2][r], z[cc - 1][r], z[cc][r], z[cc + 1][r],
                           z[cc + 2][r], j, n, twoh);
      if (MODE == 0) {
        float h;
        if (isfinite(dx) && isfinite(dy)) {
          // Only the numerator -dx*sx - dy*sy + sz cancels; it is carried in
          // float-float from the exact stencil differences.  The rest is one
          // rounded square root and one division (a few ulps, no
          // cancellation).
          const F2 ex = f2_mul(axis_diff_f2(z[cc][r - 2], z[cc][r - 1], z[cc][r], z[cc][r + 1],
                                            z[cc][r + 2], i, m), F2{s2.rh, s2.rl});
          const F2 ey = f2_mul(axis_diff_f2(z[cc - 2][r], z[cc - 1][r], z[cc][r], z[cc + 1][r],
                                            z[cc + 2][r], j, n), F2{s2.rh, s2.rl});
          const F2 num = f2_add(f2_add(f2_mul(ex, F2{-s2.sxh, -s2.sxl}),
                                       f2_mul(ey, F2{-s2.syh, -s2.syl})),
                                F2{s2.szh, s2.szl});
          const float q = __fmaf_rn(ex.hi, ex.hi, __fmaf_rn(ey.hi, ey.hi, 1.0f));
          h = __fdiv_rn(__fadd_rn(num.hi, num.lo), __fsqrt_rn(q));
          if (!isfinite(h)) h = shade(dx, dy, sx, sy, sz);
        } else {
          h = shade(dx, dy, sx, sy, sz);  // NaN / INF exactly as the reference
        }
        out0[p] = h;
      } else {
        out0[p] = dx;
        out1[p] = dy;
      }
    }
  }
}

// Weight with which the stencil centred at k (axis length len) reads the
// sample at k + off (src/hillshade.c:23-76: central differences inside,
// second-order one-sided differences on the first and last sample).
__device__ __forceinline__ float stencil_weight(int64_t k, int64_t len, int off) {
  if (k == 0) return (off == 0) ? -3.f : (off == 1) ? 4.f : (off == 2) ? -1.f : 0.f;
  if (k == len - 1) return (off == 0) ? 3.f : (off == -1) ? -4.f : (off == -2) ? 1.f : 0.f;
  return (off == 1) ? 1.f : (off == -1) ? -1.f : 0.f;
}

// Adjoint of hillshade w.r.t. the DEM: grad_dem = S^T (dH/d(dx) * g, dH/d(dy)
// * g), S the gradient stencils.  A 32 x 32 output tile needs dH/d(dx),
// dH/d(dy) at centres up to two pixels away, whose stencils read the DEM up
// to four pixels away: the block stages the DEM with a 4-pixel halo and the
// upstream gradient with a 2-pixel halo, evaluates the 36 x 36 centres from
// shared memory, then applies the transposed stencils.
constexpr int kHB = kTile + 8;  // DEM tile with a 4-pixel halo
constexpr int kHG = kTile + 4;  // centres with a 2-pixel halo

__global__ void __launch_bounds__(kBlockX * kBlockY)
hillshade_bwd_kernel(float *__restrict__ gdem, const float *__restrict__ dem,
                     const float *__restrict__ gout, int64_t m, int64_t n,
                     float twoh, float sx, float sy, float sz) {
  __shared__ float z[kHB][kHB + 1];
  __shared__ float gx[kHG][kHG + 1];  // upstream gradient, then dL/d(dx)
  __shared__ float gy[kHG][kHG + 1];  // dL/d(dy)
  constexpr int kThreads = kBlockX * kBlockY;
  const int tid = threadIdx.y * kBlockX + threadIdx.x;
  const int64_t i0 = (int64_t)blockIdx.x * kTile;
  const int64_t j0 = (int64_t)blockIdx.y * kTile;
  // Tiles whose centres and samples lie inside the grid take a fast path:
  // central differences only, which need the centres of a one-pixel ring;
  // multiplication by 1 / (2h) and rsqrtf (each within an ulp or two of the
  // exact path, far inside the adjoint's 1e-5 tolerance), no per-pixel border
  // tests, and the samples read straight from global memory, where a line
  // serves its neighbours from L1 (8192^2: 445 -> 306 us; the bytes take 119).
  if (i0 >= 4 && i0 + kTile + 4 <= m && j0 >= 4 && j0 + kTile + 4 <= n) {
    const float r2h = 1.0f / twoh;
    const int64_t p0 = (j0 - 1) * m + i0 - 1;
    constexpr int kC = kTile + 2;
    constexpr int kE = (kC * kC + kThreads - 1) / kThreads;
#pragma unroll
    for (int u = 0; u < kE; u++) {
      const int e = tid + u * kThreads;
      if (e >= kC * kC) break;
      const int c = e / kC, r = e % kC;
      const float *const zp = dem + p0 + c * m + r;
      const float z0 = zp[0], g = gout[p0 + c * m + r];
      const float dx = (zp[1] - zp[-1]) * r2h;
      const float dy = (zp[m] - zp[-m]) * r2h;
      const float inv = rsqrtf(fmaf(dx, dx, fmaf(dy, dy, 1.0f)));
      const float num = fmaf(-dx, sx, fmaf(-dy, sy, sz));
      float ax = 0.f, ay = 0.f;
      if (z0 == z0 && !isnan(num * inv)) {
        const float tt = num * (inv * inv * inv);
        ax = g * (-sx * inv - dx * tt);
        ay = g * (-sy * inv - dy * tt);
      }
      gx[c][r] = ax;
      gy[c][r] = ay;
    }
    __syncthreads();
    for (int cy = threadIdx.y; cy < kTile; cy += kBlockY) {
      const int r = threadIdx.x + 1, cc = cy + 1;
      const float acc = ((gx[cc][r - 1] - gx[cc][r + 1]) + gy[cc - 1][r]) - gy[cc + 1][r];
      gdem[(j0 + cy) * m + i0 + threadIdx.x] = acc * r2h;
    }
    return;
  }
  {  // stage the DEM and the upstream gradient, every load in flight at once
    constexpr int kZ = (kHB * kHB + kThreads - 1) / kThreads;
    constexpr int kG = (kHG * kHG + kThreads - 1) / kThreads;
    float vz[kZ], vg[kG];
#pragma unroll
    for (int u = 0; u < kZ; u++) {
      const int e = tid + u * kThreads;
      const int c = e / kHB, r = e % kHB;
      const int64_t i = i0 - 4 + r, j = j0 - 4 + c;
      vz[u] = (e < kHB * kHB && i >= 0 && i < m && j >= 0 && j < n) ? dem[j * m + i] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kG; u++) {
      const int e = tid + u * kThreads;
      const int c = e / kHG, r = e % kHG;
      const int64_t i = i0 - 2 + r, j = j0 - 2 + c;
      vg[u] = (e < kHG * kHG && i >= 0 && i < m && j >= 0 && j < n) ? gout[j * m + i] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kZ; u++) {
      const int e = tid + u * kThreads;
      if (e < kHB * kHB) z[e / kHB][e % kHB] = vz[u];
    }
#pragma unroll
    for (int u = 0; u < kG; u++) {
      const int e = tid + u * kThreads;
      if (e < kHG * kHG) gx[e / kHG][e % kHG] = vg[u];
    }
  }
  __syncthreads();
  // dH/d(dx) * g and dH/d(dy) * g at the 36 x 36 centres.
  for (int e = tid; e < kHG * kHG; e += kThreads) {
    const int c = e / kHG, r = e % kHG;
    const int64_t i = i0 - 2 + r, j = j0 - 2 + c;
    float ax = 0.f, ay = 0.f;
    if (i >= 0 && i < m && j >= 0 && j < n) {
      const int zc = c + 2, zr = r + 2;
      const float dx = axis_grad(z[zc][zr - 2], z[zc][zr - 1], z[zc][zr], z[zc][zr + 1],
                                 z[zc][zr + 2], i, m, twoh);
      const float dy = axis_grad(z[zc - 2][zr], z[zc - 1][zr], z[zc][zr], z[zc + 1][zr],
                                 z[zc + 2][zr], j, n, twoh);
      const float q = dx * dx + dy * dy + 1.0f;
      const float inv = 1.0f / sqrtf(q);
      const float num = -dx * sx - dy * sy + sz;
      if (!isnan(num * inv)) {
        const float inv3 = inv * inv * inv;
        const float g = gx[c][r];
        ax = g * (-sx * inv - num * dx * inv3);
        ay = g * (-sy * inv - num * dy * inv3);
      }
    }
    gx[c][r] = ax;  // this thread alone read gx[c][r]
    gy[c][r] = ay;
  }
  __syncthreads();
  // Transposed stencils: sample (i, j) receives from the centres whose
  // stencil reads it.  Away from the borders only the two central neighbours
  // along each axis contribute.
  const int tx = threadIdx.x;
  const int64_t i = i0 + tx;
  for (int cy = threadIdx.y; cy < kTile; cy += kBlockY) {
    const int64_t j = j0 + cy;
    if (j >= n || i >= m) continue;
    const int r = tx + 2, cc = cy + 2;
    float acc;
    if (i >= 3 && i <= m - 4 && j >= 3 && j <= n - 4) {
      acc = gx[cc][r - 1] - gx[cc][r + 1];
      acc = acc + gy[cc - 1][r];
      acc = acc - gy[cc + 1][r];
    } else {
      acc = 0.0f;
#pragma unroll
      for (int d = -2; d <= 2; d++) {
        const int64_t k = i + d;  // centre position along i
        if (k < 0 || k >= m) continue;
        const float w = stencil_weight(k, m, (int)(i - k));
        if (w != 0.f) acc += w * gx[cc][r + d];
      }
#pragma unroll
      for (int d = -2; d <= 2; d++) {
        const int64_t k = j + d;
        if (k < 0 || k >= n) continue;
        const float w = stencil_weight(k, n, (int)(j - k));
        if (w != 0.f) acc += w * gy[cc + d][r];
      }
    }
    gdem[j * m + i] = acc / twoh;
  }
}

// Strips of rows, columns per warp and blocks of a strip walk.  64 columns a
// warp (a few more are loaded as halo), fewer until the chip has `warps_per_sm`
// warps per SM, not below `least`.  Flats: 24 warps per SM and 4 columns (12
// and 48 within 5 %; 8 columns at least cost 512^2 0.2 us, 2 cost 0.5).
// Directions, more work a column: 36 warps (4096^2 66 us, 70 with 24) and 2
// columns (512^2 4.1 us, 4.4 with 4 and 5.7 with 8).
//
// A strip takes all 32 lanes of a warp and 120 rows, unless strips of 16, 8 or 4
// lanes (56, 24 or 8 rows) leave at least a quarter fewer lanes without rows of
// their own, as on grids of few rows or of a few rows more than whole strips:
// 1 x 2^20 pixels flats 272 -> 41 us and directions 413 -> 61, 30 x 131072
// 41 -> 25 and 62 -> 39, 127 x 40000 30 -> 25 and 46 -> 39.
struct StripSplit {
  int strips, cols, lanes;
  unsigned blocks;
};
StripSplit strip_split(const GridDims &g, int warps_per_sm, int least) {
  auto strips_of = [&](int lanes) {
    const int rows = (lanes - 2) * kFlatR;
    return (int)((g.m + rows - 1) / rows);
  };
  int lanes = 32;
  for (int l = 16; l >= 4; l /= 2) {
    const int64_t now = (int64_t)strips_of(lanes) * lanes, then = (int64_t)strips_of(l) * l;
    if (4 * then <= 3 * now) lanes = l;
  }
  StripSplit s{strips_of(lanes), 64, lanes, 0};
  auto warps = [&] {
    return (s.strips * ((g.n + s.cols - 1) / s.cols) + 32 / lanes - 1) / (32 / lanes);
  };
  const int64_t want = (int64_t)sm_count() * warps_per_sm;
  while (s.cols > least && warps() < want) s.cols /= 2;
  s.blocks = (unsigned)((warps() + kFlatWarps - 1) / kFlatWarps);
  return s;
}

dim3 tile_grid(const GridDims &g) { return dim3(g.tm, g.tn); }

}  // namespace

tt_cuda_status identifyflats_dev(int32_t *flags, const float *dem,
                                 const GridDims &g,
                                 unsigned long long *count_dev,
                                 cudaStream_t st) {
  unsigned long long *slots = nullptr;
  if (count_dev) {
    Workspace &ws = workspace();
    if (!ws.reserve(1024)) return TT_CUDA_ERR_ALLOC;
    slots = (unsigned long long *)ws.take(kCountSlots * 8);
    TT_CHECK(cudaMemsetAsync(slots, 0, kCountSlots * 8, st));
  }
  // Wide accesses where every column of both arrays starts on a 16-byte boundary.
  const bool wide = g.m % 4 == 0 && (((uintptr_t)flags | (uintptr_t)dem) & 15) == 0;
  const StripSplit sp = strip_split(g, 24, 4);
  const auto kernel =
      sp.lanes < 32 ? (wide ? identifyflats_kernel<true, true> : identifyflats_kernel<false, true>)
                    : (wide ? identifyflats_kernel<true, false> : identifyflats_kernel<false, false>);
  TT_LAUNCH_NEXT(kernel, sp.blocks, kFlatWarps * 32, 0, st, flags, dem, g.m, g.n, sp.strips,
                 sp.cols, sp.lanes, slots);
  if (count_dev) TT_LAUNCH(sum_slots_kernel, 1, 32, 0, st, slots, count_dev);
  TT_CHECK(cudaGetLastError());
  return TT_CUDA_SUCCESS;
}

tt_cuda_status directions_dev(uint8_t *dir, const float *dem, const float *dist,
                              const int32_t *flats, const GridDims &g,
                              unsigned order, cudaStream_t st) {
  const bool wide =
      g.m % 4 == 0 && (((uintptr_t)dem | (uintptr_t)dist | (uintptr_t)flats) & 15) == 0 &&
      ((uintptr_t)dir & 3) == 0;
  const StripSplit sp = strip_split(g, 36, 2);
  auto pick = [&](auto ord) {
    constexpr unsigned O = decltype(ord)::value;
    return sp.lanes < 32
               ? (wide ? directions_kernel<O, true, true> : directions_kernel<O, false, true>)
               : (wide ? directions_kernel<O, true, false> : directions_kernel<O, false, false>);
  };
  const auto kernel = order & 1 ? pick(std::integral_constant<unsigned, 1>{})
                                : pick(std::integral_constant<unsigned, 0>{});
  TT_LAUNCH_NEXT(kernel, sp.blocks, kFlatWarps * 32, 0, st, dir, dem, dist, flats, g.m, g.n,
                 sp.strips, sp.cols, sp.lanes);
  TT_CHECK(cudaGetLastError());
  return TT_CUDA_SUCCESS;
}

tt_cuda_status gradient2_dev(float *p0, float *p1, const float *dem,
                             float cellsize, const GridDims &g,
                             cudaStream_t st) {
  TT_LAUNCH(hillshade_kernel<1>, tile_grid(g), dim3(kBlockX, kBlockY), 0, st,
            p0, p1, dem, nullptr, g.m, g.n, 2 * cellsize, 0.f, 0.f, 0.f, Sun2{}, 0);
  TT_CHECK(cudaGetLastError());
  return TT_CUDA_SUCCESS;
}

tt_cuda_status hillshade_cols_dev(float *out, const float *dem, float azimuth,
                                  float altitude, float cellsize, const GridDims &g,
                                  int jt0, int jt1, cudaStream_t st) {
  if (jt1 <= jt0) return TT_CUDA_SUCCESS;
  float sx, sy, sz;
  sun_vector(azimuth, altitude, &sx, &sy, &sz);
  double zen = 1.57079632679489661923132169163975 - (double)altitude;
  double dsx = std::sin(zen) * std::cos((double)azimuth);
  double dsy = std::sin(zen) * std::sin((double)azimuth);
  double dsz = std::cos(zen);
  const double rinv = 1.0 / (2.0 * (double)cellsize);
  const float rh = (float)rinv;
  const double ax = dsx * rinv, ay = dsy * rinv;
  const float axh = (float)ax, ayh = (float)ay;
  Sun2 s2{sx, (float)(dsx - (double)sx), sy, (float)(dsy - (double)sy),
          sz, (float)(dsz - (double)sz), rh, (float)(rinv - (double)rh),
          axh, (float)(ax - (double)axh), ayh, (float)(ay - (double)ayh)};
  TT_LAUNCH(hillshade_kernel<0>, dim3(g.tm, jt1 - jt0), dim3(kBlockX, kBlockY), 0, st,
            out, nullptr, dem, nullptr, g.m, g.n, 2 * cellsize, sx, sy, sz, s2, jt0);
  TT_CHECK(cudaGetLastError());
  return TT_CUDA_SUCCESS;
}

tt_cuda_status hillshade_dev(float *out, const float *dem, float azimuth,
                             float altitude, float cellsize, const GridDims &g,
                             cudaStream_t st) {
  return hillshade_cols_dev(out, dem, azimuth, altitude, cellsize, g, 0, g.tn, st);
}

tt_cuda_status hillshade_backward_dev(float *grad_dem, const float *dem,
                                      const float *grad_out, float azimuth,
                                      float altitude, float cellsize,
                                      const GridDims &g, cudaStream_t st) {
  float sx, sy, sz;
  sun_vector(azimuth, altitude, &sx, &sy, &sz);
  TT_LAUNCH(hillshade_bwd_kernel, tile_grid(g), dim3(kBlockX, kBlockY), 0, st,
            grad_dem, dem, grad_out, g.m, g.n, 2 * cellsize, sx, sy, sz);
  TT_CHECK(cudaGetLastError());
  return TT_CUDA_SUCCESS;
}

}  // namespace tt
