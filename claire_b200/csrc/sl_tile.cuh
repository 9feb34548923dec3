// Shared-memory tiled tricubic gathers.
//
// One CTA of 256 threads owns a tile of 8 (x1) x 8 (x2) x 16 (x3) output
// points.  A warp covers 2 x2 rows of 16 x3 points, and each thread holds the 4
// points of consecutive x1 planes in its row and column, as two pairs.
//
// The CTA takes the bounding box of every stencil tap over the tile (min / max of
// i + floor(d), widened by the stencil's -1 .. +2) and, when it fits, copies it
// into shared memory with 16-byte asynchronous copies (the periodic wrap is
// applied per row and per chunk).  The 64 taps per point are then served from
// shared memory; tiles whose box is too large (large, rough displacements)
// gather from global memory instead.
//
// What bounds a gather is the SM's data path and, close behind, instruction
// issue.  Counted per 32 points of one field at 128^3 (adjoint step, half the
// benchmark's velocity): 91 wavefronts, of which 50 taps and box copies, 22 bank
// conflicts where floors change inside a warp, 16 global loads and stores and 3
// spilled registers (64 a thread); three fields at one map 99 a field with 5 of
// spills, the three components of a characteristic 96 with 10.  The two points of a pair nearly always have the same
// floor(d) (all but 3-10% of them on the benchmark's velocities): their stencils
// then share 3 of 5 planes, and one pass over 5 planes of 16 words serves both
// (40 words a point).  A pair whose floors differ gathers its first point in
// that pass and lists the second; after a barrier the CTA gathers the listed
// points one per thread.
//
// Shared-memory layout of a box: x3 rows of pitch P = 48 floats (16 mod 32: the 2
// rows of a warp use opposite halves of the bank space; 32 where only that
// fits), x1 planes of stride Q = ext2 * P.  Every shared-memory index is inside the box by construction:
// each point's taps lie in [i + floor(d) - 1, i + floor(d) + 2] and the box spans
// the min / max of exactly those values over the tile's points; points outside
// the grid (partial tiles) repeat the last point inside and are never stored.
//
// The kernels are not persistent: several CTAs per SM (one tile each) overlap
// one another's copies with their gathers.
//
// Measured in situ, 8 problems of 128^3, all launches of a solve's first two
// Gauss-Newton iterations: adjoint steps 159 us (173 with a stencil per point,
// 64 words a point and a bulk copy per box row), incremental steps 156 (162), the
// 24 cached gradient fields 4.05 ms (4.61), characteristics 0.62 ms (0.72).
#pragma once

#include <climits>
#include <type_traits>

#include "sl.cuh"

namespace cb {

constexpr int kT1 = 8, kT2 = 8, kT3 = 16;
constexpr int kTileThreads = 256;
constexpr int kTilePts = 4;  // points per thread

// Shared memory of a CTA: one box and the list of single points (at most every
// second one).  4 CTAs of 256 threads per SM; the boxes stop here because what
// four CTAs leave of the 256 KB is the L1 cache of the displacement and operand
// loads (11648 floats and a 9 KB list: time steps 7% slower).
constexpr int kGatherBudget = 9856;  // floats
constexpr int kMaxListed = kTileThreads * kTilePts / 2;
constexpr int kGatherSmemBytes = kGatherBudget * 4 + kMaxListed * 2;
constexpr int kGatherMinBlocks = 4;

__host__ __device__ inline unsigned tile_count(const Dims& d) {
  return (unsigned)(((d.n1 + kT1 - 1) / kT1) * ((d.n2 + kT2 - 1) / kT2) * ((d.n3 + kT3 - 1) / kT3));
}

// q / m for 0 <= q < 2^22 and 1 <= m < 2^12 without an integer division:
// float estimate, then one correction each way.
CB_DEVICE int small_div(int q, int m) {
  int t = __float2int_rz((float)q * (1.f / (float)m));
  const int r = q - t * m;
  t += (r >= m) ? 1 : 0;
  t -= (r < 0) ? 1 : 0;
  return t;
}

// x mod n for x in [-n, 2n)
CB_DEVICE int wrap_near(int x, int n) {
  x += (x < 0) ? n : 0;
  x -= (x >= n) ? n : 0;
  return x;
}

// Tiles along x2 and x3 and the reciprocals that split a tile index without a
// division: umulhi(t, floor(2^32 / nb) + 1) exceeds t / nb by at most one.
struct TileGrid {
  unsigned nb2, nb3, m2, m3;
  __host__ __device__ explicit TileGrid(const Dims& d)
      : nb2((d.n2 + kT2 - 1) / kT2), nb3((d.n3 + kT3 - 1) / kT3),
        m2(nb2 == 1 ? 0u : (unsigned)((1ull << 32) / nb2) + 1u),
        m3(nb3 == 1 ? 0u : (unsigned)((1ull << 32) / nb3) + 1u) {}
};

CB_DEVICE unsigned tile_div(unsigned t, unsigned nb, unsigned m) {
  if (nb == 1) return t;
  const unsigned q = __umulhi(t, m);
  return q * nb > t ? q - 1 : q;
}

// This thread's points in the CTA's tile: 4 consecutive x1 planes of one row
// and column.  Coordinates are clamped to the grid: a point beyond it repeats
// the last one inside (same tile, so the same box), which makes every load and
// every stencil valid without a predicate; only its store is left out.  Point
// indices are 32-bit (grids up to 1024^3 points).
struct TileThread {
  int x1_, x2, x3;  // first plane, row, column (clamped)
  int amax;         // planes past the first that are inside the grid
  unsigned vmask;   // bit a: point a lies inside the grid
  unsigned idx0, plane;
  CB_DEVICE bool valid(int a) const { return (vmask >> a) & 1u; }
  CB_DEVICE int step(int a) const { return min(a, amax); }
  CB_DEVICE int x1(int a) const { return x1_ + step(a); }
  CB_DEVICE unsigned idx(int a) const { return idx0 + (unsigned)step(a) * plane; }
};

// Position of thread t's points in its tile (first x1 plane, x2 row, x3
// column): a warp covers 4 planes x 2 rows x 16 columns.
CB_DEVICE void tile_local(int t, int& l1, int& l2, int& l3) {
  l1 = 4 * (t >> 7);
  l2 = (t >> 4) & 7;
  l3 = t & 15;
}

// Origin of the CTA's tile.
CB_DEVICE void tile_origin(const TileGrid& tg, int& t1, int& t2, int& t3) {
  const unsigned t = blockIdx.x, r = tile_div(t, tg.nb3, tg.m3), c1 = tile_div(r, tg.nb2, tg.m2);
  t1 = (int)(c1 * kT1);
  t2 = (int)((r - c1 * tg.nb2) * kT2);
  t3 = (int)((t - r * tg.nb3) * kT3);
}

CB_DEVICE TileThread tile_thread(const Dims& d, const TileGrid& tg) {
  int t1, t2, t3, l1, l2, l3;
  tile_origin(tg, t1, t2, t3);
  tile_local(threadIdx.x, l1, l2, l3);
  const int p1 = t1 + l1, p2 = t2 + l2, p3 = t3 + l3;
  TileThread tt;
  const bool row_ok = (p2 < d.n2) && (p3 < d.n3);
  const int left = d.n1 - p1;  // planes inside the grid from p1 on
  tt.vmask = row_ok && left > 0 ? (left >= kTilePts ? 15u : (1u << left) - 1u) : 0u;
  tt.x1_ = min(p1, d.n1 - 1);
  tt.x2 = min(p2, d.n2 - 1);
  tt.x3 = min(p3, d.n3 - 1);
  tt.amax = max(left - 1, 0);
  tt.plane = (unsigned)d.n2 * (unsigned)d.n3;
  tt.idx0 = (unsigned)tt.x1_ * tt.plane + (unsigned)tt.x2 * (unsigned)d.n3 + (unsigned)tt.x3;
  return tt;
}

// x3 row pitches of a staged box: 48 floats (16 mod 32 banks), or 32 where only
// that fits (strong maps; the two rows of a warp then share their banks, which
// is far cheaper than gathering from global memory).  192 x 192 x 256, one field,
// every box of the map alike, against pitches 32 / 64 with a plane offset that
// keeps the two rows apart and 32 KB a box: 169 rows of 20 floats 125 us (140), 225
// rows (pitch 32) 174 (155), 256 and 289 rows 176 (261, global memory), 324 rows
// (global memory) 268 (262).  Rows of 49 to 64 floats go to global memory, 257-301
// us, which pitch 64 served in 178: such a map stretches x3 by 2.7 and more over a
// whole tile, and code for a third pitch cost every gather of three fields 1 to 3%.
constexpr int kPitch = 48, kPitchTight = 32;

struct TileBox {
  int lo[3];
  int e1, e2, e3;  // extents (e3 in whole 16-byte chunks)
  int P, Q;        // x3 row pitch, x1 plane stride (floats)
  bool fits;       // copyable (one wrap per axis, whole chunks) and within budget
};

// Box of the stencil bases b = i + floor(d) - 1 in [lo, hi] per axis (taps b .. b+3).
CB_DEVICE TileBox box_from_bounds(const int (&lo)[3], const int (&hi)[3], const Dims& d) {
  const int nk[3] = {d.n1, d.n2, d.n3};
  TileBox bx;
  int ext[3];
  bool fits = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const long long l = lo[k], e = (long long)hi[k] - l + 4;
    // one wrap per coordinate in the copy, origin within one period
    fits = fits && e > 0 && e <= nk[k] && l >= -nk[k] && l < nk[k];
    bx.lo[k] = fits ? (int)l : 0;
    ext[k] = fits ? (int)e : 4;
  }
  // x3: start on a multiple of 4 floats and cover whole 4-float chunks so the
  // box is copied in 16-byte pieces (N3 % 4 == 0: no chunk straddles the seam)
  const int lo3a = bx.lo[2] & ~3;
  bx.e3 = ((bx.lo[2] + ext[2] - lo3a) + 3) & ~3;
  bx.lo[2] = lo3a;
  bx.e1 = ext[0];
  bx.e2 = ext[1];
  const long long rows = (long long)bx.e1 * bx.e2;
  bx.P = bx.e3 <= kPitch && rows * kPitch <= kGatherBudget ? kPitch : kPitchTight;
  bx.Q = bx.e2 * bx.P;
  bx.fits = fits && bx.e3 <= d.n3 && bx.e3 <= bx.P && (d.n3 & 3) == 0 && rows * bx.P <= kGatherBudget;
  return bx;
}

// Block-wide min / max of the stencil bases of the tile's points.
// Contains __syncthreads: call once, from uniform control flow.
CB_DEVICE void tile_bounds(const float (&dd)[kTilePts][3], const TileThread& tt, int (&lo)[3], int (&hi)[3]) {
  __shared__ int red[6][kTileThreads / 32];
  int mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
#pragma unroll
  for (int a = 0; a < kTilePts; ++a) {
    const int b[3] = {tt.x1(a) + (int)floorf(dd[a][0]) - 1, tt.x2 + (int)floorf(dd[a][1]) - 1,
                      tt.x3 + (int)floorf(dd[a][2]) - 1};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      mn[k] = min(mn[k], b[k]);
      mx[k] = max(mx[k], b[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
    mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      red[k][warp] = mn[k];
      red[3 + k][warp] = mx[k];
    }
  }
  __syncthreads();
  // every warp reduces the 8 warp partials itself (lane l reads partial l % 8)
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = __reduce_min_sync(0xffffffffu, red[k][lane & 7]);
    hi[k] = __reduce_max_sync(0xffffffffu, red[3 + k][lane & 7]);
  }
}

// Per-tile box table of a displacement field: the tile's TileBox packed in two
// int4, {lo1, lo2, lo3, fits ? P : 0}, {e1, e2, e3, Q}.  It depends on the displacement
// only, so one table serves every gather at that characteristic (all time
// steps, all matvecs of a GN iterate).
CB_DEVICE void pack_box(const TileBox& bx, int4& a, int4& b) {
  a = make_int4(bx.lo[0], bx.lo[1], bx.lo[2], bx.fits ? bx.P : 0);
  b = make_int4(bx.e1, bx.e2, bx.e3, bx.Q);
}

CB_DEVICE TileBox box_from_table(const int4* __restrict__ tab) {
  const int4 a = __ldg(tab + 2 * blockIdx.x), b = __ldg(tab + 2 * blockIdx.x + 1);
  TileBox bx;
  bx.lo[0] = a.x;
  bx.lo[1] = a.y;
  bx.lo[2] = a.z;
  bx.fits = a.w != 0;
  bx.P = a.w;
  bx.e1 = b.x;
  bx.e2 = b.y;
  bx.e3 = b.z;
  bx.Q = b.w;
  return bx;
}

// ---- bounded wait (self-test of the device's failure counter) ---------------
// Count of bounded waits that ran out; read by stage_timeouts().
__device__ unsigned g_stage_timeouts = 0;

CB_DEVICE unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
CB_DEVICE void mbar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// the barrier's one arrival, announcing the bytes its copies will deliver
CB_DEVICE void mbar_arrive_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One try_wait on phase 0; a thread whose phase is not complete is suspended
// by the hardware for up to hint_ns (or until the phase completes).
CB_DEVICE bool mbar_test(unsigned bar, unsigned hint_ns) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0, %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// Wait for phase 0 of the barrier for at most limit_ns; a wait that runs out is
// counted and reported as false.
CB_DEVICE bool bounded_wait(unsigned bar, unsigned long long limit_ns) {
  if (mbar_test(bar, 1000u)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_test(bar, 1000u))
    if (global_ns() - t0 > limit_ns) {
      atomicAdd(&g_stage_timeouts, 1u);
      return false;
    }
  return true;
}

// ---- box copies ---------------------------------------------------------------
CB_DEVICE void copy16(unsigned dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Asynchronous copies of field f's box into the box at shared memory sb.  8
// threads copy a row (chunks of 16 bytes), the CTA 32 rows at a time; the next
// row of a thread is found without divisions.  Every chunk is 16-byte aligned
// (x3 starts on a multiple of 4 floats, N3 % 4 == 0, P and Q are multiples of 4,
// f is aligned) and none straddles the x3 seam.  (One bulk copy per row,
// completing on an mbarrier, took 58 instructions a point: it is issued one lane
// at a time, and the waiting warps spin.)
CB_DEVICE void issue_box(float* sb, const float* __restrict__ f, const TileBox& bx, const Dims& d) {
  constexpr int kRows = kTileThreads / 8;
  const int lc = threadIdx.x & 7, nck = bx.e3 >> 2;
  if (lc >= nck) return;
  const int w3 = wrap_near(bx.lo[2], d.n3);
  int g3 = w3 + 4 * lc, h3 = g3 + 32;  // rows of more than 32 floats: chunks 8 .. 11
  g3 -= g3 >= d.n3 ? d.n3 : 0;
  h3 -= h3 >= d.n3 ? d.n3 : 0;
  const bool hi = lc + 8 < nck;
  // row r = l1 e2 + l2; a step of kRows is s1 planes and s2 rows
  const int r0 = threadIdx.x >> 3;
  const int s1 = small_div(kRows, bx.e2), s2 = kRows - s1 * bx.e2;
  int l1 = small_div(r0, bx.e2), l2 = r0 - l1 * bx.e2;
  const int lo1 = wrap_near(bx.lo[0], d.n1), lo2 = wrap_near(bx.lo[1], d.n2);
  unsigned dst = (unsigned)__cvta_generic_to_shared(sb) + 4u * (unsigned)(r0 * bx.P + 4 * lc);  // Q = e2 P
  while (l1 < bx.e1) {
    int g1 = lo1 + l1, g2 = lo2 + l2;
    g1 -= g1 >= d.n1 ? d.n1 : 0;
    g2 -= g2 >= d.n2 ? d.n2 : 0;
    const float* src = f + (unsigned)(g1 * d.n2 + g2) * (unsigned)d.n3;
    copy16(dst, src + g3);
    if (hi) copy16(dst + 128u, src + h3);
    dst += 4u * kRows * (unsigned)bx.P;
    l1 += s1;
    l2 += s2;
    if (l2 >= bx.e2) {
      l2 -= bx.e2;
      ++l1;
    }
  }
}

// This thread's copies have landed; a barrier then publishes the box.
CB_DEVICE void copies_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// bf16 image field: the box is widened to FP32 while it is staged, with plain
// loads and stores.  Warp w copies x1 planes w, w + 8, ...; its lanes cover
// whole x3 rows of 4-element chunks, rows advancing without divisions (one
// conditional wrap per row along x2 and per plane along x1).  Each chunk is
// one 8-byte load (x3 offsets are multiples of 4 and N3 % 4 == 0, so every
// chunk is 8-byte aligned) and one 16-byte shared store; the shared-memory
// layout, and so the gather that reads it, is the FP32 one.
CB_DEVICE void issue_box(float* __restrict__ sb, const bf16* __restrict__ f, const TileBox& bx, const Dims& d) {
  const int nck = bx.e3 >> 2;
  const int rpi = small_div(32, nck);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lr = small_div(lane, nck), lc = lane - lr * nck;
  if (lr >= rpi || lr >= bx.e2) return;
  int g1 = wrap_near(bx.lo[0] + warp, d.n1);
  const int w2 = wrap_near(bx.lo[1] + lr, d.n2);
  int g3 = wrap_near(bx.lo[2], d.n3) + 4 * lc;
  g3 -= (g3 >= d.n3) ? d.n3 : 0;
  const bf16* fb = f + g3;
  const unsigned row = (unsigned)d.n3, plane = (unsigned)d.n2 * (unsigned)d.n3;
  constexpr int kWarps = kTileThreads / 32;
  for (int l1 = warp; l1 < bx.e1; l1 += kWarps) {
    const bf16* fp = fb + (unsigned)g1 * plane;
    float* sp = sb + l1 * bx.Q + lr * bx.P + 4 * lc;
    int g2 = w2;
    for (int l2 = lr; l2 < bx.e2; l2 += rpi) {
      const uint2 raw = __ldg(reinterpret_cast<const uint2*>(fp + (unsigned)g2 * row));
      const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
      const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
      *reinterpret_cast<float4*>(sp) = make_float4(lo.x, lo.y, hi.x, hi.y);
      sp += rpi * bx.P;
      g2 += rpi;
      while (g2 >= d.n2) g2 -= d.n2;
    }
    g1 += kWarps;
    g1 -= (g1 >= d.n1) ? d.n1 : 0;
  }
}

// Four consecutive floats at byte offset OFF from addr, weighted by w.
template <int OFF>
CB_DEVICE float row4(unsigned addr, const float (&w)[4]) {
  float x0, x1, x2, x3;
  asm volatile(
      "ld.shared.f32 %0, [%4+%5];\n\t"
      "ld.shared.f32 %1, [%4+%6];\n\t"
      "ld.shared.f32 %2, [%4+%7];\n\t"
      "ld.shared.f32 %3, [%4+%8];\n"
      : "=f"(x0), "=f"(x1), "=f"(x2), "=f"(x3)
      : "r"(addr), "n"(OFF), "n"(OFF + 4), "n"(OFF + 8), "n"(OFF + 12));
  return w[0] * x0 + w[1] * x1 + w[2] * x2 + w[3] * x3;
}

// 64-tap gather from a staged box with row pitch P (floats) and plane stride
// qb (bytes); base = shared address of the point's tap (0, 0, 0).
template <int P>
CB_DEVICE float gather_box(unsigned base, unsigned qb, const float (&w1)[4], const float (&w2)[4],
                           const float (&w3)[4]) {
  float acc = 0.f;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const unsigned pa = base + a * qb;
    const float t = w2[0] * row4<0>(pa, w3) + w2[1] * row4<P * 4>(pa, w3) + w2[2] * row4<P * 8>(pa, w3) +
                    w2[3] * row4<P * 12>(pa, w3);
    acc += w1[a] * t;
  }
  return acc;
}

// ---- packed FP32 pairs (fma.rn.f32x2) ------------------------------------------
// Two multiply-adds per instruction, each lane an ordinary round-to-nearest
// FP32 FMA.  The pairs are two x2 rows of a plane at one x3 column: their words
// arrive by separate 32-bit loads, so pairing them costs nothing.
typedef unsigned long long f32x2;

CB_DEVICE f32x2 pk2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
CB_DEVICE float2 upk2(f32x2 r) {
  float2 o;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
  return o;
}
CB_DEVICE f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
CB_DEVICE f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

CB_DEVICE f32x2 dup2(float c) { return pk2(c, c); }

// lagrange4 of two fractions at once (same Horner steps)
CB_DEVICE void lagrange4x2(f32x2 s, f32x2 (&w)[4]) {
  w[0] = mul2(s, fma2(s, fma2(s, dup2(-1.f / 6.f), dup2(0.5f)), dup2(-1.f / 3.f)));
  w[1] = fma2(s, fma2(s, fma2(s, dup2(0.5f), dup2(-1.f)), dup2(-0.5f)), dup2(1.f));
  w[2] = mul2(s, fma2(s, fma2(s, dup2(-0.5f), dup2(0.5f)), dup2(1.f)));
  w[3] = mul2(s, fma2(mul2(s, s), dup2(1.f / 6.f), dup2(-1.f / 6.f)));
}

template <int OFF>
CB_DEVICE float lds(unsigned addr) {
  float x;
  asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(x) : "r"(addr), "n"(OFF));
  return x;
}

// The first NC words of a row (byte offset OFF), and of the rows r and r + 2 as
// pairs.
template <int OFF, int NC>
CB_DEVICE void row1(unsigned addr, float (&x)[NC]) {
  x[0] = lds<OFF>(addr);
  x[1] = lds<OFF + 4>(addr);
  x[2] = lds<OFF + 8>(addr);
  x[3] = lds<OFF + 12>(addr);
  if constexpr (NC > 4) x[4] = lds<OFF + 16>(addr);
}
template <int OFF, int P, int NC>
CB_DEVICE void rows2(unsigned addr, f32x2 (&x)[NC]) {
  float a[NC], b[NC];
  row1<OFF>(addr, a);
  row1<OFF + 8 * P>(addr, b);
#pragma unroll
  for (int c = 0; c < NC; ++c) x[c] = pk2(a[c], b[c]);
}

template <int NC>
CB_DEVICE f32x2 row_sums(const f32x2 (&x)[NC], const f32x2 (&w3)[NC]) {
  f32x2 t = mul2(w3[0], x[0]);
#pragma unroll
  for (int c = 1; c < NC; ++c) t = fma2(w3[c], x[c], t);
  return t;
}

// Weights of points A and B (fractions s, t): along x1, along x2 as row pairs
// (r, r + 2), so that a sum runs over neighbouring rows before the two halves
// meet, along x3 duplicated.  The choice against pairs (r, r + 1) is one
// of roundoff: solves that sit on it (H3 with beta 1e-4 at 32^3) keep the oracle's
// Gauss-Newton counts with this order of sums and not with the other.
struct PairWeights {
  float w1[2][4];
  f32x2 w2[2][2], w3[2][4];
  CB_DEVICE PairWeights(const float (&s)[3], const float (&t)[3]) {
    f32x2 w[4];
    float2 u[4];
    lagrange4x2(pk2(s[0], t[0]), w);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      u[c] = upk2(w[c]);
      w1[0][c] = u[c].x;
      w1[1][c] = u[c].y;
    }
    lagrange4x2(pk2(s[1], t[1]), w);
#pragma unroll
    for (int c = 0; c < 4; ++c) u[c] = upk2(w[c]);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      w2[0][c] = pk2(u[c].x, u[c + 2].x);
      w2[1][c] = pk2(u[c].y, u[c + 2].y);
    }
    lagrange4x2(pk2(s[2], t[2]), w);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      u[c] = upk2(w[c]);
      w3[0][c] = dup2(u[c].x);
      w3[1][c] = dup2(u[c].y);
    }
  }
};

// Points A (planes 0..3 from base) and B (planes 1..4) in one pass over five
// planes qb bytes apart; `last` is the address of plane 4 (any box address where
// B is not wanted).  One row pair is live at a time.
template <int P>
CB_DEVICE float2 gather_pair(unsigned base, unsigned qb, unsigned last, const PairWeights& w) {
  float ra = 0.f, rb = 0.f;
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const unsigned pa = q < 4 ? base + q * qb : last;
    f32x2 ta = 0ull, tb = 0ull;
    {
      f32x2 x[4];
      rows2<0, P>(pa, x);
      if (q < 4) ta = mul2(w.w2[0][0], row_sums(x, w.w3[0]));
      if (q > 0) tb = mul2(w.w2[1][0], row_sums(x, w.w3[1]));
    }
    {
      f32x2 x[4];
      rows2<4 * P, P>(pa, x);
      if (q < 4) ta = fma2(w.w2[0][1], row_sums(x, w.w3[0]), ta);
      if (q > 0) tb = fma2(w.w2[1][1], row_sums(x, w.w3[1]), tb);
    }
    if (q < 4) {
      const float2 t = upk2(ta);
      ra = fmaf(w.w1[0][q], t.x + t.y, ra);
    }
    if (q > 0) {
      const float2 t = upk2(tb);
      rb = fmaf(w.w1[1][q - 1], t.x + t.y, rb);
    }
  }
  return make_float2(ra, rb);
}

// Fractions s of displacement dd and the shared address of the stencil's first
// tap, `origin` being the address of the tap at floor(d) = 0.  Addresses
// o1 Q + o2 P + o3 (o2 < ext2, o3 < P) are distinct for distinct taps.
template <int P>
CB_DEVICE unsigned point_stencil(const float (&dd)[3], unsigned origin, unsigned qb, float (&s)[3]) {
  const float f1 = floorf(dd[0]), f2 = floorf(dd[1]), f3 = floorf(dd[2]);
  s[0] = dd[0] - f1;
  s[1] = dd[1] - f2;
  s[2] = dd[2] - f3;
  return origin + (unsigned)(int)f1 * qb + (unsigned)(int)f2 * (4 * P) + 4u * (unsigned)(int)f3;
}

// Address of the first tap of point (x1, x2, x3) at floor(d) = 0 (taken modulo
// 2^32: it may lie outside the box).
CB_DEVICE unsigned tap_origin(unsigned sb, int x1, int x2, int x3, const TileBox& bx) {
  return sb + 4u * (unsigned)((x1 - 1 - bx.lo[0]) * bx.Q + (x2 - 1 - bx.lo[1]) * bx.P + (x3 - 1 - bx.lo[2]));
}

// Points of the tile that are gathered one by one.
struct PointList {
  unsigned short* id;  // 4 * thread + point
  int* count;
  CB_DEVICE void push(bool want, int point) const {
    const unsigned m = __ballot_sync(0xffffffffu, want);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    int at = 0;
    if (lane == 0) at = atomicAdd(count, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (want) id[at] = (unsigned short)(kTilePts * threadIdx.x + point);
  }
};

// Staged gather of the tile's points: epi(index, value, aux) for every point
// inside the grid.  Contains __syncthreads: call from uniform control flow.
template <int P, class Src, class Epi>
CB_DEVICE void gather_tile(unsigned sb, const PointList& list, const Src& src, const float (&dd)[kTilePts][3],
                           const float (&aux)[kTilePts], const TileThread& tt, const TileBox& bx, const Dims& d,
                           const TileGrid& tg, const Epi& epi) {
  const unsigned qb = (unsigned)bx.Q * 4u;
  const unsigned origin = tap_origin(sb, tt.x1_, tt.x2, tt.x3, bx);
#pragma unroll
  for (int a = 0; a < kTilePts; a += 2) {
    float s[3], t[3];
    const unsigned base = point_stencil<P>(dd[a], origin + (unsigned)tt.step(a) * qb, qb, s);
    const unsigned baseb = point_stencil<P>(dd[a + 1], origin + (unsigned)tt.step(a + 1) * qb, qb, t);
    const bool shared = baseb == base + qb;
    list.push(tt.valid(a + 1) && !shared, a + 1);
    const float2 r = gather_pair<P>(base, qb, shared ? base + 4 * qb : base, PairWeights(s, t));
    if (tt.valid(a)) epi(tt.idx(a), r.x, aux[a]);
    if (shared && tt.valid(a + 1)) epi(tt.idx(a + 1), r.y, aux[a + 1]);
  }
  __syncthreads();
  const int n = *list.count;
  if (threadIdx.x >= n) return;
  int t1, t2, t3;
  tile_origin(tg, t1, t2, t3);
  for (int i = threadIdx.x; i < n; i += kTileThreads) {
    const int id = list.id[i];
    int l1, l2, l3;
    tile_local(id / kTilePts, l1, l2, l3);
    const int x1 = t1 + l1 + id % kTilePts, x2 = t2 + l2, x3 = t3 + l3;
    const unsigned at = (unsigned)x1 * tt.plane + (unsigned)x2 * (unsigned)d.n3 + (unsigned)x3;
    float de[3], s[3], w1[4], w2[4], w3[4];
    src.at(de, at, d);
    const float ae = epi.aux ? __ldg(epi.aux + at) : 0.f;
    const unsigned base = point_stencil<P>(de, tap_origin(sb, x1, x2, x3, bx), qb, s);
    lagrange4(s[0], w1);
    lagrange4(s[1], w2);
    lagrange4(s[2], w3);
    epi(at, gather_box<P>(base, qb, w1, w2, w3), ae);
  }
}

// The same for the few tiles whose box is only staged at the tight pitch: point
// by point, plane by plane, in few registers (a second copy of the pair pass
// makes the common one spill).
template <class Epi>
CB_DEVICE void gather_tight(unsigned sb, const float (&dd)[kTilePts][3], const float (&aux)[kTilePts],
                            const TileThread& tt, const TileBox& bx, const Epi& epi) {
  const unsigned qb = (unsigned)bx.Q * 4u;
  const unsigned origin = tap_origin(sb, tt.x1_, tt.x2, tt.x3, bx);
#pragma unroll
  for (int a = 0; a < kTilePts; ++a) {
    float s[3], w1[4], w2[4], w3[4];
    unsigned at = point_stencil<kPitchTight>(dd[a], origin + (unsigned)tt.step(a) * qb, qb, s);
    lagrange4(s[0], w1);
    lagrange4(s[1], w2);
    lagrange4(s[2], w3);
    float r = 0.f;
#pragma unroll 1
    for (int q = 0; q < 4; ++q, at += qb) {
      const float w = q < 2 ? (q ? w1[1] : w1[0]) : (q == 2 ? w1[2] : w1[3]);
      r += w * (w2[0] * row4<0>(at, w3) + w2[1] * row4<4 * kPitchTight>(at, w3) +
                w2[2] * row4<8 * kPitchTight>(at, w3) + w2[3] * row4<12 * kPitchTight>(at, w3));
    }
    if (tt.valid(a)) epi(tt.idx(a), r, aux[a]);
  }
}

// Global-memory gather of the thread's points (tiles whose box does not fit).
template <class T, class Epi>
CB_DEVICE void gather_unstaged(const T* __restrict__ f, const float (&dd)[kTilePts][3], const float (&aux)[kTilePts],
                               const TileThread& tt, const Dims& d, const Epi& epi) {
#pragma unroll
  for (int a = 0; a < kTilePts; ++a) {
    if (!tt.valid(a)) continue;
    Stencil st;
    make_stencil(tt.x1(a), tt.x2, tt.x3, dd[a][0], dd[a][1], dd[a][2], d, st);
    epi(tt.idx(a), gather(f, st), aux[a]);
  }
}

// Fields whose rows cannot be copied in 16-byte chunks (8 for bf16) gather from
// global memory.
template <class T>
CB_DEVICE bool aligned_field(const T* f) {
  return (reinterpret_cast<uintptr_t>(f) & (4 * sizeof(T) - 1)) == 0;
}

CB_DEVICE PointList point_list(float* sb, int* count) {
  return PointList{reinterpret_cast<unsigned short*>(sb + kGatherBudget), count};
}

// Displacements of the tile's points from a displacement field (3 arrays n apart).
struct DispSource {
  const float* ds;
  CB_DEVICE void at(float (&dd)[3], unsigned i, const Dims& d) const {
    const float* d2 = ds + d.n();
    dd[0] = __ldg(ds + i);
    dd[1] = __ldg(d2 + i);
    dd[2] = __ldg(d2 + d.n() + i);
  }
};

template <class Src>
CB_DEVICE void load_points(const Src& src, float (&dd)[kTilePts][3], const TileThread& tt, const Dims& d) {
#pragma unroll
  for (int a = 0; a < kTilePts; ++a) src.at(dd[a], tt.idx(a), d);
}

// Tile gather of the fields f + k ff, k < nf, at the displacements of Src, one
// after another: the displacements, their box and the tile set-up are shared.
// tab (may be null) is the displacement's box table: with it the first copy is
// issued before the displacements load; without it the CTA reduces its box
// itself.  epi(k) is field k's epilogue, called as (index, value, aux) with
// aux = epi(k).aux[index] (0 where it has none).  sb holds kGatherSmemBytes
// (16-byte aligned).  A bf16 field is widened to FP32 while it is staged.
template <class T, class Src, class MakeEpi>
CB_DEVICE void tile_gather(float* sb, const Src& src, const int4* __restrict__ tab, const T* __restrict__ f,
                           long long ff, int nf, const Dims& d, const TileGrid& tg, const MakeEpi& epi) {
  __shared__ int listed[2];
  const TileThread tt = tile_thread(d, tg);
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(sb);
  float dd[kTilePts][3];
  TileBox bx;
  if (threadIdx.x == 0) listed[0] = 0;
  if (tab) {
    bx = box_from_table(tab);
    if (bx.fits && aligned_field(f)) issue_box(sb, f, bx, d);
    load_points(src, dd, tt, d);
  } else {
    load_points(src, dd, tt, d);
    int lo[3], hi[3];
    tile_bounds(dd, tt, lo, hi);
    bx = box_from_bounds(lo, hi, d);
    if (bx.fits && aligned_field(f)) issue_box(sb, f, bx, d);
  }
#pragma unroll 1
  for (int k = 0; k < nf; ++k, f += ff) {
    const auto e = epi(k);
    const bool staged = bx.fits && aligned_field(f);
    if (k) {
      __syncthreads();  // field k - 1 is done with the box and its list
      if (staged) issue_box(sb, f, bx, d);
    }
    float aux[kTilePts];
#pragma unroll
    for (int a = 0; a < kTilePts; ++a) aux[a] = e.aux ? __ldg(e.aux + tt.idx(a)) : 0.f;
    if (threadIdx.x == 0) listed[(k + 1) & 1] = 0;  // the next field's
    if (!staged) {
      gather_unstaged(f, dd, aux, tt, d, e);
      continue;
    }
    copies_landed();
    __syncthreads();
    // opaque per field: weights hoisted out of this loop would not fit in
    // registers (here, after every load is issued: the statement waits for dd)
#pragma unroll
    for (int a = 0; a < kTilePts; ++a) asm volatile("" : "+f"(dd[a][0]), "+f"(dd[a][1]), "+f"(dd[a][2]));
    const PointList list = point_list(sb, &listed[k & 1]);
    if (bx.P == kPitch) gather_tile<kPitch>(sbase, list, src, dd, aux, tt, bx, d, tg, e);
    else gather_tight(sbase, dd, aux, tt, bx, e);
  }
}

// The same for one field with a table (the time steps), without the loop's
// state: 5% faster than tile_gather with nf = 1.
template <class T, class Src, class Epi>
CB_DEVICE void tile_step(float* sb, const Src& src, const int4* __restrict__ tab, const T* __restrict__ f,
                         const Dims& d, const TileGrid& tg, const Epi& e) {
  __shared__ int listed;
  const TileBox bx = box_from_table(tab);
  const bool staged = bx.fits && aligned_field(f);
  if (staged) issue_box(sb, f, bx, d);
  const TileThread tt = tile_thread(d, tg);
  if (threadIdx.x == 0) listed = 0;
  float dd[kTilePts][3], aux[kTilePts];
  load_points(src, dd, tt, d);
#pragma unroll
  for (int a = 0; a < kTilePts; ++a) aux[a] = e.aux ? __ldg(e.aux + tt.idx(a)) : 0.f;
  if (!staged) return gather_unstaged(f, dd, aux, tt, d, e);
  copies_landed();
  __syncthreads();
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(sb);
  const PointList list = point_list(sb, &listed);
  if (bx.P == kPitch) gather_tile<kPitch>(sbase, list, src, dd, aux, tt, bx, d, tg, e);
  else gather_tight(sbase, dd, aux, tt, bx, e);
}

}  // namespace cb
