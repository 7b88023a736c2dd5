// Level 0's smoothing passes of the plane-stress FP32 V-cycle, two grid columns a lane.
#pragma once

#include "mg.cuh"

namespace stt {

// The chained passes (l0_presmooth_kernel, l0_postsmooth_kernel) are bound by instruction
// issue.  Here a lane owns the columns 2 j and 2 j + 1 of one displacement component in a
// float2, so that an operation of the modal stage is one paired instruction for two columns
// with nothing to move between the halves, the neighbour column is in the same lane every
// other time (half the shuffles), and a strip's halo is a smaller part of it: 250 instructions
// a row of 58 columns against 159 a row of 27.  And since the lane's even column is a coarse
// column of a 2 x 2 coarsening, the transfers join: the pre-smoothing pass restricts the
// residual as it appears (it is never written), the post-smoothing pass adds the prolonged
// correction to the iterate as it loads it.
//
// The state of two columns takes 142-152 registers, so 12 warps an SM, too few to wait out a
// memory latency at each row: a row's data comes by asynchronous copies into a ring of four to
// seven rows ahead in shared memory.  All of it does, flags and coarse values too: plain
// loads two rows ahead of their use, queued behind the copies in the L1, cost half the time.
//
// Rows and columns outside the grid load the nearest node inside and are masked (w and the
// density zero), so no load is tested.  On B200 at 2048x1024 x 16 rows: pre-smoothing and
// restriction 263 + 60 -> 245 us, prolongation and post-smoothing 105 + 296 -> 244 us, the
// V-cycle 1718 -> 1434 us; without the ring 343 and 445; at 128 registers and 16 warps an SM,
// spilled, 468 and 634.  They are as good on small grids (540x270 x 4 rows: a V-cycle of 110 us
// with the old passes, 105 with these; 256x128 x 8: 92 and 91), so they run wherever they apply.
struct PairQ {
  float2 m00, m01, m11, m22, m44, m55;  // MQ's coefficients, twice each
  float2 neg, half;                     // -1 and 1/2: the paired instructions have no negation
  float kd, kr;                         // kd0 and kd1 / kd0
};
inline PairQ pair_q(const MQ<float>& q) {
  auto two = [](float v) { return float2{v, v}; };
  return PairQ{two(q.m00), two(q.m01), two(q.m11), two(q.m22),  two(q.m44),
               two(q.m55), two(-1.f),  two(0.5f),  q.kd0,       q.kd1 / q.kd0};
}

// ModalStage<2, float> for a pair of columns (index: component); the operations round alike.
struct PairStage {
  float2 sT[2], dT[2], co[2], cr[2], ut[2];

  STT_DEV void reset() {
#pragma unroll
    for (int d = 0; d < 2; ++d) sT[d] = dT[d] = co[d] = cr[d] = ut[d] = make_float2(0.f, 0.f);
  }
  STT_DEV static float2 sub(const PairQ& q, float2 a, float2 b) { return __ffma2_rn(b, q.neg, a); }
  STT_DEV void step(const PairQ& q, const float2 (&u)[2], float2 rho, float2 (&Ku)[2]) {
    float2 Gx[2], Gy[2], H[2], own[2], send[2];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const float vr = __shfl_down_sync(0xffffffffu, u[d].x, 1);
      const float2 sB = make_float2(u[d].x + u[d].y, u[d].y + vr), dB = make_float2(u[d].y - u[d].x, vr - u[d].y);
      Gx[d] = __fadd2_rn(dB, dT[d]);
      Gy[d] = sub(q, sT[d], sB);
      H[d] = sub(q, dT[d], dB);
      sT[d] = sB;
      dT[d] = dB;
      ut[d] = u[d];
    }
    const float2 p = __fmul2_rn(rho, Gx[0]), pq = __fmul2_rn(rho, Gy[1]);
    const float2 a = __ffma2_rn(q.m01, pq, __fmul2_rn(q.m00, p));
    const float2 cc = __ffma2_rn(q.m01, p, __fmul2_rn(q.m11, pq));
    const float2 b = __fmul2_rn(__fmul2_rn(rho, q.m22), __fadd2_rn(Gy[0], Gx[1]));
    corners(q, a, b, __fmul2_rn(__fmul2_rn(rho, q.m44), H[0]), co[0], cr[0], own[0], send[0]);
    corners(q, b, cc, __fmul2_rn(__fmul2_rn(rho, q.m55), H[1]), co[1], cr[1], own[1], send[1]);
#pragma unroll
    for (int d = 0; d < 2; ++d)
      Ku[d] = make_float2(own[d].x + __shfl_up_sync(0xffffffffu, send[d].y, 1), own[d].y + send[d].x);
  }
  STT_DEV static void corners(const PairQ& q, float2 al, float2 be, float2 ga, float2& co, float2& cr, float2& own,
                              float2& send) {
    const float2 s = __fadd2_rn(al, be), t = sub(q, al, be);
    own = sub(q, co, __fadd2_rn(t, ga));
    send = __fadd2_rn(cr, __fadd2_rn(s, ga));
    co = sub(q, ga, s);
    cr = sub(q, t, ga);
  }
};

// A front row's data, by column: right-hand side, iterate (post only), density, flags.
struct PairFront {
  float4 b, x;
  float2 rho;
  uint2 fl;  // the words that hold the two nodes' flags
};
// What the stages need of a row one and two rows later, by component: w = omega / diag, zero
// on fixed dofs and off the grid; `fl` its fixed dofs (bits 0, 1: the even column's, 2, 3: the
// odd one's), `any` whether any lane has one.
struct PairRow {
  float2 b[2], w[2], rho;
  unsigned fl;
  bool any;
};
STT_DEV void pair_mask(float2 (&v)[2], unsigned fl) {
  if (fl & 1) v[0].x = 0.f;
  if (fl & 2) v[1].x = 0.f;
  if (fl & 4) v[0].y = 0.f;
  if (fl & 8) v[1].y = 0.f;
}

// A warp's strip: where its lanes load.  Everything that belongs to a row (f, and the address of
// its first node) is uniform over the warp, so a lane's part of an address is a constant offset.
struct PairStrip {
  int c0, nnx, nny;
  unsigned a0, a1;          // the lane's two nodes in a row, the nearest ones in the grid
  unsigned e0, e1;          // byte offsets of the two elements
  unsigned off;             // fl of the columns off the grid
  bool el0, el1, cols;      // the column is an element's; every lane's columns are

  STT_DEV PairStrip(int c, int nelx, int nely) : c0(c), nnx(nelx + 1), nny(nely + 1) {
    a0 = min(max(c, 0), nelx);
    a1 = min(max(c + 1, 0), nelx);
    e0 = min(a0, (unsigned)(nelx - 1)) * 4u;
    e1 = min(a1, (unsigned)(nelx - 1)) * 4u;
    off = (c >= 0 && c <= nelx ? 0u : 3u) | (c + 1 >= 0 && c + 1 <= nelx ? 0u : 12u);
    el0 = c >= 0 && c < nelx;
    el1 = c + 1 >= 0 && c + 1 < nelx;
    cols = __all_sync(0xffffffffu, el0 && el1);
  }
  STT_DEV long long node_row(int f) const { return (long long)min(max(f, 0), nny - 1) * nnx; }
  STT_DEV const float* elem_row(const float* rh, int f) const {
    return rh + (long long)min(max(f, 0), nny - 2) * (nnx - 1);
  }
  // element row f's densities (the strip stands on it), zero off the grid
  STT_DEV float2 rho_ok(float2 v, int f) const {
    if (!cols || (unsigned)f >= (unsigned)(nny - 1)) {
      const bool ok = (unsigned)f < (unsigned)(nny - 1);
      v.x = ok && el0 ? v.x : 0.f;
      v.y = ok && el1 ? v.y : 0.f;
    }
    return v;
  }
  STT_DEV static void copy8(unsigned to, const void* p, unsigned o) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(static_cast<const char*>(p) + o) : "memory");
  }
  STT_DEV static void copy4(unsigned to, const void* p, unsigned o) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(static_cast<const char*>(p) + o) : "memory");
  }
  // Copies row f into a slot of the warp's ring.  Each lane
  // copies its own columns (so it waits for its own copies only): per lane b (16 bytes), x (16,
  // post only), rho (8), the words around the flags (8), and what the caller adds in `more`.
  // Everything a row needs goes this way: a plain load's data would queue behind the copies.
  template <bool X, typename More>
  STT_DEV void fetch(int f, unsigned slot, const float2* bs, const float2* xs, const float* rh, const uint8_t* fixed,
                     More more) {
    const unsigned lane = threadIdx.x & 31, t16 = slot + lane * 16, t8 = slot + (X ? 1024 : 512) + lane * 8;
    const long long row = node_row(f);
    copy8(t16, bs + row, a0 * 8);
    copy8(t16 + 8, bs + row, a1 * 8);
    if constexpr (X) {
      copy8(t16 + 512, xs + row, a0 * 8);
      copy8(t16 + 520, xs + row, a1 * 8);
    }
    const float* er = elem_row(rh, f);
    copy4(t8, er, e0);
    copy4(t8 + 4, er, e1);
    const unsigned sh = (unsigned)row & 3;
    copy4(t8 + 256, fixed + (row - sh), (sh + a0) & ~3u);
    copy4(t8 + 260, fixed + (row - sh), (sh + a1) & ~3u);
    more(slot + (X ? 1536 : 1024));
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  STT_DEV float2 rho_at(const float* rh, int f) const {
    const char* p = reinterpret_cast<const char*>(elem_row(rh, f));
    return make_float2(__ldg(reinterpret_cast<const float*>(p + e0)), __ldg(reinterpret_cast<const float*>(p + e1)));
  }
  template <bool X>
  STT_DEV static void read(const char* slot, PairFront& F) {
    const unsigned lane = threadIdx.x & 31;
    F.b = reinterpret_cast<const float4*>(slot)[lane];
    if constexpr (X) F.x = reinterpret_cast<const float4*>(slot + 512)[lane];
    F.rho = reinterpret_cast<const float2*>(slot + (X ? 1024 : 512))[lane];
    F.fl = reinterpret_cast<const uint2*>(slot + (X ? 1280 : 768))[lane];
  }
  // the row's PairRow; rho_prev: the element row above (masked), replaced by this one
  STT_DEV void row(const PairFront& F, int f, const PairQ& q, float omega, float2& rho_prev, PairRow& R) const {
    R.rho = rho_ok(F.rho, f);
    const float2 rs = __fadd2_rn(R.rho, rho_prev);
    rho_prev = R.rho;
    const float d0 = rs.x + __shfl_up_sync(0xffffffffu, rs.y, 1), d1 = rs.y + rs.x;
    R.w[0] = make_float2(sweep_div(omega, q.kd * d0), sweep_div(omega, q.kd * d1));
    R.w[1] = make_float2(R.w[0].x * q.kr, R.w[0].y * q.kr);
    // (neighbours in the same words may set `any`: then only the mask is formed for nothing)
    R.any = __any_sync(0xffffffffu, F.fl.x | F.fl.y | off) || (unsigned)f >= (unsigned)nny;
    R.fl = 0;
    if (R.any) {
      const unsigned sh = (unsigned)node_row(f) & 3;
      R.fl = (F.fl.x >> ((sh + a0) & 3) * 8 & 3) | (F.fl.y >> ((sh + a1) & 3) * 8 & 3) << 2 | off |
             ((unsigned)f < (unsigned)nny ? 0u : 15u);
      pair_mask(R.w, R.fl);
    }
    R.b[0] = make_float2(F.b.x, F.b.z);
    R.b[1] = make_float2(F.b.y, F.b.w);
  }
  STT_DEV void store(float2* __restrict__ o, int r, const float2 (&v)[2]) const {
    float2* p = o + (long long)r * nnx;
    if (c0 < nnx) p[(unsigned)c0] = make_float2(v[0].x, v[1].x);
    if (c0 + 1 < nnx) p[(unsigned)(c0 + 1)] = make_float2(v[0].y, v[1].y);
  }
};

constexpr int kPairPreCols = 58, kPairPostCols = 60;

// Rows a warp marches: even, so that a band starts on a coarse row; the longest that gives each
// SM its 12 warps, but 4 rows (with 6 of halo) only where 8 would leave it fewer than 8 warps.
// A V-cycle of 540x270 x 4 rows: 110 us with 4-row bands, 105 with 8; 256x128 x 8: 92 with 4, 97
// with 8; 512x256 x 33: 362 with 32, 372 with 64.
inline int pair_band(int strips, int nny, int rows) {
  int band = 64;
  while (band > 4 && (long long)strips * ((nny + band - 1) / band) * rows < 148LL * (band > 8 ? 12 : 8)) band /= 2;
  return band;
}
// A launch: warps numbered (band, strip), kQWarps a block.
struct PairGrid {
  int strips, band, bands;
  dim3 g;
};
inline PairGrid pair_grid(int cols, int nelx, int nely, int rows) {
  PairGrid p;
  p.strips = (nelx + 1 + cols - 1) / cols;
  p.band = pair_band(p.strips, nely + 1, rows);
  p.bands = (nely + 1 + p.band - 1) / p.band;
  p.g = dim3((p.strips * p.bands + kQWarps - 1) / kQWarps, 1, rows);
  return p;
}

// Two pre-smoothing sweeps from zero and the residual of row f - 2 behind the front row f
// (l0_presmooth_kernel).  DOWN: the residual goes restricted to the 2 x 2 coarser level's
// right-hand side `out_r` (restrict_t_kernel's sums), else as it is.
// Lanes 2 .. 30 are output; DOWN also needs the residual one row above the band.
template <bool DOWN>
__global__ void __launch_bounds__(kQThreads, 3) l0_pre_pair_kernel(
    const float* __restrict__ b, long long b_rs, float* __restrict__ out_x, long long ox_rs, float* __restrict__ out_r,
    long long or_rs, const float* __restrict__ rho, long long rho_rs, const uint8_t* __restrict__ fixed,
    const uint8_t* __restrict__ cfixed, const int* __restrict__ row_map, int hrows, const RowState* __restrict__ rst,
    int nelx, int nely, int strips, int band, float omega, PairQ q) {
  grid_wait();
  const int s = blockIdx.z;
  if (rst && !rst[s].active) return;
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // (known to be uniform)
  const int wid = blockIdx.x * kQWarps + warp;
  const int r0 = wid / strips * band;
  if (r0 > nely) return;
  const int r1 = min(r0 + band, nely + 1);
  const int f0 = DOWN ? r0 - 4 : r0 - 2, f1 = DOWN ? ((r1 - 1) | 1) + 2 : r1 + 1;  // front rows, inclusive
  PairStrip ps(wid % strips * kPairPreCols - 4 + 2 * lane, nelx, nely);
  const bool out_lane = lane >= 2 && lane <= 30;
  const float* rh = rho + (size_t)hier_row(row_map, hrows, s) * rho_rs;
  const float2* bs = reinterpret_cast<const float2*>(b + (size_t)s * b_rs);
  float2* ox = reinterpret_cast<float2*>(out_x + (size_t)s * ox_rs);
  float2* orr = reinterpret_cast<float2*>(out_r + (size_t)s * or_rs);
  const int cnnx = nelx / 2 + 1, cnny = nely / 2 + 1, C = ps.c0 >> 1;
  const bool c_lane = out_lane && C < cnnx;
  PairStage A, B;
  A.reset();
  B.reset();
  PairRow d1{}, d2{};
  d1.fl = d2.fl = 15u;
  d1.any = d2.any = true;
  float2 gE = make_float2(0.f, 0.f), gP = gE;  // DOWN: x-restricted residual of the even row, of the odd row above
  constexpr int SB = 1024 + (DOWN ? 128 : 0), NR = 8;  // a ring slot's bytes, the ring's rows
  __shared__ __align__(16) char ring[kQWarps * NR * SB];
  char* const rw = ring + warp * NR * SB;
  const unsigned ra = (unsigned)__cvta_generic_to_shared(rw);
  float2 rho_prev = ps.rho_ok(ps.rho_at(rh, f0 - 1), f0 - 1);
  // DOWN: at even rows f also the flags of the coarse row that row f - 1 completes
  auto cnode = [&](int f) { return (unsigned)min(max((f - 2) >> 1, 0), cnny - 1) * cnnx + min(max(C, 0), cnnx - 1); };
  auto fetch = [&](int f, int slot, bool even) {
    ps.fetch<false>(f, ra + slot, bs, nullptr, rh, fixed, [&](unsigned to) {
      if (DOWN && even) PairStrip::copy4(to + lane * 4, cfixed, cnode(f) & ~3u);
    });
  };
  for (int k = 0; k < NR - 1; ++k) fetch(f0 + k, k * SB, !(k & 1));
  int at = 0;
  for (int fb = f0; fb <= f1; fb += 2) {
    unsigned cfl = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int f = fb + k;
      PairFront F;
      asm volatile("cp.async.wait_group %0;" ::"n"(NR - 2) : "memory");
      ps.read<false>(rw + at, F);
      if (DOWN && k == 0) cfl = reinterpret_cast<const unsigned*>(rw + at + 1024)[lane] >> (cnode(f) & 3) * 8;
      at = at + SB == NR * SB ? 0 : at + SB;
      fetch(f + NR - 1, at >= 2 * SB ? at - 2 * SB : at + (NR - 2) * SB, k == 1);  // into the slot read a row ago
      PairRow cur;
      ps.row(F, f, q, omega, rho_prev, cur);
      float2 x1[2], K[2], xo[2], xa[2], rb[2];
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        x1[d] = __fmul2_rn(cur.w[d], cur.b[d]);
        xo[d] = A.ut[d];
      }
      A.step(q, x1, d1.rho, K);
#pragma unroll
      for (int d = 0; d < 2; ++d) xa[d] = __ffma2_rn(d1.w[d], PairStage::sub(q, d1.b[d], K[d]), xo[d]);
      B.step(q, xa, d2.rho, K);
#pragma unroll
      for (int d = 0; d < 2; ++d) rb[d] = PairStage::sub(q, d2.b[d], K[d]);
      if (d2.any) pair_mask(rb, d2.fl);
      if (out_lane && f - 1 >= r0 && f - 1 < r1) ps.store(ox, f - 1, xa);
      if constexpr (DOWN) {
        float2 g;
        g.x = fmaf(0.5f, __shfl_up_sync(0xffffffffu, rb[0].y, 1), fmaf(0.5f, rb[0].y, rb[0].x));
        g.y = fmaf(0.5f, __shfl_up_sync(0xffffffffu, rb[1].y, 1), fmaf(0.5f, rb[1].y, rb[1].x));
        if (k == 0) {
          gE = g;
        } else {  // row f - 2 = 2 R + 1 completes coarse row R
          if (c_lane && f - 3 >= r0 && f - 3 < r1) {
            const float vx = fmaf(0.5f, gP.x, fmaf(0.5f, g.x, gE.x)), vy = fmaf(0.5f, gP.y, fmaf(0.5f, g.y, gE.y));
            orr[(long long)((f - 3) >> 1) * cnnx + C] = make_float2(cfl & 1 ? 0.f : vx, cfl & 2 ? 0.f : vy);
          }
          gP = g;
        }
      } else {
        if (out_lane && f - 2 >= r0 && f - 2 < r1) ps.store(orr, f - 2, rb);
      }
      d2 = d1;
      d1 = cur;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// The two post-smoothing sweeps (l0_postsmooth_kernel).  UP: from x0 + P e with e the 2 x 2
// coarser level's correction (prolong_t_kernel's sums), else from x0 (prolonged already).
// RZ: also the PCG's r.z, as l0_postsmooth_kernel.  Lanes 1 .. 30 are output.
template <bool UP, bool RZ>
__global__ void __launch_bounds__(kQThreads, 3) l0_post_pair_kernel(
    const float* __restrict__ x0, long long x_rs, const float* __restrict__ ec, long long e_rs,
    const float* __restrict__ b, long long b_rs, float* __restrict__ out, long long o_rs,
    const float* __restrict__ rho, long long rho_rs, const uint8_t* __restrict__ fixed,
    const int* __restrict__ row_map, int hrows, const RowState* __restrict__ rst, int nelx, int nely, int strips,
    int band, float omega, PairQ q, RzFuse<float> rz) {
  grid_wait();
  const int s = blockIdx.z;
  if (rst && !rst[s].active) return;
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // (known to be uniform)
  const int wid = blockIdx.x * kQWarps + warp;
  const int r0 = wid / strips * band;
  const int r1 = min(r0 + band, nely + 1);  // <= r0 for the last block's warps past the last band
  const int f0 = r0 - 2, f1 = r1 + 1;  // front rows, inclusive
  PairStrip ps(wid % strips * kPairPostCols - 2 + 2 * lane, nelx, nely);
  const bool out_lane = lane >= 1 && lane <= 30;
  const float* rh = rho + (size_t)hier_row(row_map, hrows, s) * rho_rs;
  const float2* xs = reinterpret_cast<const float2*>(x0 + (size_t)s * x_rs);
  const float2* bs = reinterpret_cast<const float2*>(b + (size_t)s * b_rs);
  const float2* es = UP ? reinterpret_cast<const float2*>(ec + (size_t)s * e_rs) : nullptr;
  float2* os = reinterpret_cast<float2*>(out + (size_t)s * o_rs);
  const int cnnx = nelx / 2 + 1, cnny = nely / 2 + 1;
  const int C0 = min(max(ps.c0 >> 1, 0), cnnx - 1), C1 = min(max((ps.c0 >> 1) + 1, 0), cnnx - 1);
  double dots[1] = {0.0};
  if (r0 < r1) {
    // a coarse row's values at columns C0 and C1 on the lane's fine columns, by component
    auto xpro = [](const float4& e, float2(&t)[2]) {
      t[0] = make_float2(e.x, fmaf(0.5f, e.z, 0.5f * e.x));
      t[1] = make_float2(e.y, fmaf(0.5f, e.w, 0.5f * e.y));
    };
    PairStage A, B;
    A.reset();
    B.reset();
    PairRow d1{}, d2{};
    constexpr int SB = 1536 + (UP ? 512 : 0), NR = UP ? 5 : 6;  // a ring slot's bytes, the ring's rows
    __shared__ __align__(16) char ring[kQWarps * NR * SB];
    char* const rw = ring + warp * NR * SB;
    const unsigned ra = (unsigned)__cvta_generic_to_shared(rw);
    float2 rho_prev = ps.rho_ok(ps.rho_at(rh, f0 - 1), f0 - 1);
      // UP: at even rows f also the coarse row below the one that f stands on
    auto fetch = [&](int f, int slot, bool even) {
      ps.fetch<true>(f, ra + slot, bs, xs, rh, fixed, [&](unsigned to) {
        if (UP && even) {
          const float2* p = es + (long long)min(max((f >> 1) + 1, 0), cnny - 1) * cnnx;
          PairStrip::copy8(to + lane * 16, p, C0 * 8u);
          PairStrip::copy8(to + lane * 16 + 8, p, C1 * 8u);
        }
      });
    };
    for (int k = 0; k < NR - 1; ++k) fetch(f0 + k, k * SB, !(k & 1));
    int at = 0;
    float2 tE[2], tN[2];  // UP: coarse rows R and R + 1 on the fine columns
    if constexpr (UP) {
      const float2* p = es + (long long)max(f0 >> 1, 0) * cnnx;
      const float2 l = __ldg(p + C0), r = __ldg(p + C1);
      xpro(make_float4(l.x, l.y, r.x, r.y), tE);
    }
    for (int fb = f0; fb <= f1; fb += 2) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int f = fb + k;
        PairFront F;
        asm volatile("cp.async.wait_group %0;" ::"n"(NR - 2) : "memory");
        ps.read<true>(rw + at, F);
        if (UP && k == 0) xpro(reinterpret_cast<const float4*>(rw + at + 1536)[lane], tN);
        at = at + SB == NR * SB ? 0 : at + SB;
        // into the slot read a row ago; NR - 1 rows on, with that row's parity
        fetch(f + NR - 1, at >= 2 * SB ? at - 2 * SB : at + (NR - 2) * SB, ((k + NR - 1) & 1) == 0);
        PairRow cur;
        ps.row(F, f, q, omega, rho_prev, cur);
        float2 xi[2], K[2], xo[2], xa[2], xb[2];
        xi[0] = make_float2(F.x.x, F.x.z);
        xi[1] = make_float2(F.x.y, F.x.w);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          if constexpr (UP)
            xi[d] = __fadd2_rn(xi[d], k == 0 ? tE[d] : __ffma2_rn(q.half, tN[d], __fmul2_rn(q.half, tE[d])));
          xo[d] = A.ut[d];
        }
        if (cur.any) pair_mask(xi, cur.fl);
        A.step(q, xi, d1.rho, K);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          xa[d] = __ffma2_rn(d1.w[d], PairStage::sub(q, d1.b[d], K[d]), xo[d]);
          xo[d] = B.ut[d];
        }
        B.step(q, xa, d2.rho, K);
#pragma unroll
        for (int d = 0; d < 2; ++d) xb[d] = __ffma2_rn(d2.w[d], PairStage::sub(q, d2.b[d], K[d]), xo[d]);
        if (out_lane && f - 2 >= r0 && f - 2 < r1) {
          ps.store(os, f - 2, xb);
          if constexpr (RZ) {  // off the grid xb is zero
            const float2 t = __ffma2_rn(d2.b[1], xb[1], __fmul2_rn(d2.b[0], xb[0]));
            dots[0] += (double)t.x;
            dots[0] += (double)t.y;
          }
        }
        d2 = d1;
        d1 = cur;
      }
      if constexpr (UP) {
#pragma unroll
        for (int d = 0; d < 2; ++d) tE[d] = tN[d];
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  if constexpr (RZ)
    grid_reduce<1, kQThreads>(rz.red, s, blockIdx.x, dots, [&](const double* t) {
      RowState& S = rz.rst[s];
      const double t2[2] = {t[0], S.rz_mix};
      pcg_rz_finish(S, t2, rz.first, rz.flexible);
    });
}

}  // namespace stt
