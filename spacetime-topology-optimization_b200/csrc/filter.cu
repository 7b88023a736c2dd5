// Cone density filter and Heaviside projection (the density field's upstream step).
//
// Reference: filters.density_filter / apply_density_filter (sttopt/filters.py:38-85):
// H[e1, e2] = max(0, rmin - dist(e1, e2)) over the square of offsets |d| <= ceil(rmin) - 1,
// xTilde = H x / Hs with Hs the row sums, and heaviside_projection /
// heaviside_projection_derivative (:109-133).  H is a stencil with zero padding outside
// the grid, so it is applied as one here: a block stages its output tile plus the stencil's
// halo in shared memory (coalesced rows), and a thread slides down its column, holding the
// sums of one or two rows, so that an input value is read once for the rows it enters.
// Hs is the sum of the in-grid weights: a constant away from the border (summed on the
// host), formed from the element's position near it (no matrix, no row-sum array).  H is
// symmetric, so the adjoint, H (g * P'(xTilde) / Hs), is the same stencil applied to the
// scaled field.  FP64 throughout; rows of the batch with their own strides.
#include <cmath>
#include <vector>

#include "common.cuh"
#include "errors.h"

namespace stt {

constexpr int kFiltMaxR = 7;  // ceil(rmin) - 1 <= 7 (rmin <= 8)
constexpr int kFiltTX = 32;  // threads along x: a tile's width

struct FiltW {
  double w[(2 * kFiltMaxR + 1) * (2 * kFiltMaxR + 1)];  // w[(dj + R) * (2R + 1) + (di + R)]
  double hs;  // their sum: Hs of an element at least R from every edge
};

// The projection's constants (beta > 0; beta = inf is the step with 1/2 at the threshold).
struct FiltP {
  double beta, eta;
  double t0, den;  // tanh(beta eta), tanh(beta eta) + tanh(beta (1 - eta))
};

// Hs of element (i, j): the sum of the weights whose offset stays in the grid.
template <int R>
STT_DEV double filt_hs(const FiltW& W, int i, int j, int nelx, int nely) {
  if (i >= R && i < nelx - R && j >= R && j < nely - R) return W.hs;
  constexpr int n = 2 * R + 1;
  double s = 0.0;
#pragma unroll 1
  for (int dj = -R; dj <= R; ++dj) {
    if (j + dj < 0 || j + dj >= nely) continue;
#pragma unroll
    for (int di = -R; di <= R; ++di)
      if (i + di >= 0 && i + di < nelx) s += W.w[(dj + R) * n + (di + R)];
  }
  return s;
}

STT_DEV double heaviside(double x, const FiltP& P) {
  if (isinf(P.beta)) return x > P.eta ? 1.0 : (x < P.eta ? 0.0 : 0.5);
  return (P.t0 + tanh(P.beta * (x - P.eta))) / P.den;
}
STT_DEV double heaviside_d(double x, const FiltP& P) {
  if (isinf(P.beta)) return 0.0;
  const double t = tanh(P.beta * (x - P.eta));
  return P.beta * (1.0 - t * t) / P.den;
}

// ADJ = 0: xt = H x / Hs (and xp = P(xt) when beta > 0);
// ADJ = 1: out = H (g * s / Hs), s = P'(xt) when beta > 0 (xt given), else 1.
// Bound by instruction issue ((2R + 1)^2 FP64 multiply-adds, a tanh and two divisions an element)
// and by the latency of the staging loads and of Hs near the border, a chain of up to (2R + 1)^2
// sums, with a row of it unrolled.  A thread takes two rows of a 32 x 32 tile: more rows mean
// fewer shared-memory loads but fewer warps (at rmin 4 and 2048 x 1024, before the unrolling: 8 rows a
// thread 45 us forward with the projection and 55 the adjoint, 4 rows 36 and 45, 2 rows 32 and 40, 1
// row 40 and 51; now 29 and 36).  Launches of fewer such tiles than SMs take 32 x 8 tiles and one row:
// 180 x 60 at rmin 4 3.8 and 5.9 us, 5.8 and 6.9 with the other, at rmin 8 8 and 16 against 14 and 20;
// at 540 x 270 (153 tiles) 5.4 and 7.8 against 6.4 and 7.4.
template <int ADJ, int R, int VY, int TY>
__global__ void __launch_bounds__(kFiltTX * TY) cone_filter_kernel(
    const double* __restrict__ in, long long in_rs, const double* __restrict__ xt_in, long long xt_rs,
    double* __restrict__ out, double* __restrict__ xp, long long o_rs, int nelx, int nely, FiltW W, FiltP P) {
  constexpr int n = 2 * R + 1, tw = kFiltTX + 2 * R, th = TY * VY + 2 * R;
  __shared__ double tile[th * tw];
  const int s = blockIdx.z;
  const int i0 = blockIdx.x * kFiltTX, j0 = blockIdx.y * (TY * VY);
  const double* xs = in + (size_t)s * in_rs;
  const double* ts = ADJ ? xt_in + (size_t)s * xt_rs : nullptr;
  const bool proj = P.beta > 0.0;
  for (int t = threadIdx.y * kFiltTX + threadIdx.x; t < tw * th; t += kFiltTX * TY) {
    const int tj = t / tw, ti = t - tj * tw;
    const int i = i0 - R + ti, j = j0 - R + tj;
    double v = 0.0;
    if (i >= 0 && i < nelx && j >= 0 && j < nely) {
      const long long e = (long long)j * nelx + i;
      v = __ldg(xs + e);
      if (ADJ) {
        if (proj && ts) v *= heaviside_d(__ldg(ts + e), P);
        v /= filt_hs<R>(W, i, j, nelx, nely);
      }
    }
    tile[t] = v;
  }
  __syncthreads();
  const int i = i0 + threadIdx.x, jl = threadIdx.y * VY;  // this thread's column and first row in the tile
  if (i >= nelx || j0 + jl >= nely) return;
  // input row r of the column's window adds its taps to the output rows r - 2R .. r; each
  // output takes its taps in row-major order
  double acc[VY];
#pragma unroll
  for (int y = 0; y < VY; ++y) acc[y] = 0.0;
  // (a weight depends on |di| and |dj|, in either order: (R + 1)(R + 2) / 2 distinct ones)
  auto weight = [&](int dj, int di) {
    const int a = dj < 0 ? -dj : dj, b = di < 0 ? -di : di;
    return W.w[((a >= b ? a : b) + R) * n + (a >= b ? b : a) + R];
  };
#pragma unroll
  for (int r = 0; r < VY + 2 * R; ++r) {
    double v[n];
#pragma unroll
    for (int c = 0; c < n; ++c) v[c] = tile[(jl + r) * tw + threadIdx.x + c];
#pragma unroll
    for (int y = 0; y < VY; ++y)
      if (r - y >= 0 && r - y <= 2 * R)
#pragma unroll
        for (int c = 0; c < n; ++c) acc[y] = fma(weight(r - y - R, c - R), v[c], acc[y]);
  }
  double* os = out + (size_t)s * o_rs;
#pragma unroll
  for (int y = 0; y < VY; ++y) {
    const int j = j0 + jl + y;
    if (j >= nely) break;
    const long long e = (long long)j * nelx + i;
    if (ADJ) {
      os[e] = acc[y];
    } else {
      const double x = acc[y] / filt_hs<R>(W, i, j, nelx, nely);
      os[e] = x;
      if (proj && xp) xp[(size_t)s * o_rs + e] = heaviside(x, P);
    }
  }
}

// The weights max(0, rmin - hypot(di, dj)) of the reference (filters.py:52-55).
static bool filt_weights(double rmin, int& R, FiltW& W) {
  if (!(rmin > 0.0) || !std::isfinite(rmin)) return false;
  R = (int)std::ceil(rmin) - 1;
  if (R < 0 || R > kFiltMaxR) return false;
  const int n = 2 * R + 1;
  for (int dj = -R; dj <= R; ++dj)
    for (int di = -R; di <= R; ++di) W.w[(dj + R) * n + (di + R)] = std::fmax(0.0, rmin - std::hypot((double)di, (double)dj));
  W.hs = 0.0;
  for (int t = 0; t < n * n; ++t) W.hs += W.w[t];
  return true;
}

template <int ADJ>
static int launch_filter(int nelx, int nely, int nrows, double rmin, const double* in, long long in_rs,
                         const double* xt, long long xt_rs, double* out, double* xp, long long o_rs, double beta,
                         double eta, cudaStream_t st) {
  int R;
  FiltW W;
  if (!filt_weights(rmin, R, W))
    return set_error(STT_ERR_INVALID, "cone filter: rmin must be in (0, 8]");
  FiltP P{beta, eta, 0.0, 1.0};
  if (beta > 0.0 && !std::isinf(beta)) {
    P.t0 = std::tanh(beta * eta);
    P.den = P.t0 + std::tanh(beta * (1.0 - eta));
  }
  const int gx = (nelx + kFiltTX - 1) / kFiltTX;
  // 32 x 32 tiles, two rows a thread; 32 x 8 and one row where there are fewer of those than SMs
  const bool small = (long long)gx * ((nely + 31) / 32) * nrows < 148;
#define STT_FILT_TILE(RR, VY, TY)                                                                       \
  cone_filter_kernel<ADJ, RR, VY, TY><<<dim3(gx, (nely + VY * TY - 1) / (VY * TY), nrows), dim3(kFiltTX, TY), 0, st>>>( \
      in, in_rs, xt, xt_rs, out, xp, o_rs, nelx, nely, W, P)
#define STT_FILT(RR)                  \
  if (small) STT_FILT_TILE(RR, 1, 8); \
  else STT_FILT_TILE(RR, 2, 16)
  switch (R) {
    case 0:
      STT_FILT(0);
      break;
    case 1:
      STT_FILT(1);
      break;
    case 2:
      STT_FILT(2);
      break;
    case 3:
      STT_FILT(3);
      break;
    case 4:
      STT_FILT(4);
      break;
    case 5:
      STT_FILT(5);
      break;
    case 6:
      STT_FILT(6);
      break;
    default: STT_FILT(7);
  }
#undef STT_FILT
#undef STT_FILT_TILE
  return check_launch("cone filter");
}

}  // namespace stt

using namespace stt;

extern "C" int stt_cone_filter(int nelx, int nely, int nrows, double rmin, const double* x, long long x_rs,
                               double* xt, double* xp, long long o_rs, double beta, double eta,
                               stt_stream_t stream) {
  if (nelx <= 0 || nely <= 0 || nrows <= 0 || nrows > 65535 || !x || !xt || (beta > 0.0 && !xp))
    return set_error(STT_ERR_INVALID, "stt_cone_filter: bad sizes or null pointer");
  return launch_filter<0>(nelx, nely, nrows, rmin, x, x_rs, nullptr, 0, xt, xp, o_rs, beta, eta,
                          (cudaStream_t)stream);
}

extern "C" int stt_cone_filter_adjoint(int nelx, int nely, int nrows, double rmin, const double* g,
                                       long long g_rs, const double* xt, long long xt_rs, double beta,
                                       double eta, double* out, long long o_rs, stt_stream_t stream) {
  if (nelx <= 0 || nely <= 0 || nrows <= 0 || nrows > 65535 || !g || !out || (beta > 0.0 && !xt))
    return set_error(STT_ERR_INVALID, "stt_cone_filter_adjoint: bad sizes or null pointer");
  return launch_filter<1>(nelx, nely, nrows, rmin, g, g_rs, xt, xt_rs, out, nullptr, o_rs, beta, eta,
                          (cudaStream_t)stream);
}
