// Cone density filter and Heaviside projection (the density field's upstream step).
//
// Reference: filters.density_filter / apply_density_filter (sttopt/filters.py:38-85):
// H[e1, e2] = max(0, rmin - dist(e1, e2)) over the square of offsets |d| <= ceil(rmin) - 1,
// xTilde = H x / Hs with Hs the row sums, and heaviside_projection /
// heaviside_projection_derivative (:109-133).  H is a stencil with zero padding outside
// the grid, so it is applied as one here: a block stages its output tile plus the stencil's
// halo in shared memory (coalesced rows), and a thread slides down its column, holding the
// sums of VY rows, so that an input value is read once for the up to VY rows it enters.
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
constexpr int kFiltTX = 32, kFiltTY = 16;  // threads a block
constexpr int kFiltVY = 2;                 // rows a thread: a tile is 32 x 32 elements

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
#pragma unroll 1
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
// Bound by instruction issue (0.55-0.6 of the cycles: (2R + 1)^2 FP64 multiply-adds, a tanh
// and two divisions an element) and by the staging loads' latency, so a thread takes only
// two rows: more rows mean fewer shared-memory loads but fewer warps (8 rows a thread, 5
// blocks of 256 an SM: 45 and 55 us; 4 rows 36 and 45; 1 row 40 and 51).  With the weights
// read from the constant bank, Hs summed for every element and three tanh each (in the
// adjoint for every staged element, twice over with an 8-row tile's halo), 2048 x 1024 at
// rmin 4 took 95 us forward with the projection and 171 us the adjoint; now 34 and 41.
template <int ADJ, int R>
__global__ void __launch_bounds__(kFiltTX * kFiltTY) cone_filter_kernel(
    const double* __restrict__ in, long long in_rs, const double* __restrict__ xt_in, long long xt_rs,
    double* __restrict__ out, double* __restrict__ xp, long long o_rs, int nelx, int nely, FiltW W, FiltP P) {
  constexpr int VY = kFiltVY, n = 2 * R + 1, tw = kFiltTX + 2 * R, th = kFiltTY * VY + 2 * R;
  __shared__ double tile[th * tw];
  const int s = blockIdx.z;
  const int i0 = blockIdx.x * kFiltTX, j0 = blockIdx.y * (kFiltTY * VY);
  const double* xs = in + (size_t)s * in_rs;
  const double* ts = ADJ ? xt_in + (size_t)s * xt_rs : nullptr;
  const bool proj = P.beta > 0.0;
  for (int t = threadIdx.y * kFiltTX + threadIdx.x; t < tw * th; t += kFiltTX * kFiltTY) {
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
  // the distinct weights (they depend on |di|, |dj|, in either order) held in registers: a
  // multiply-add takes no constant-bank operand in FP64, so each would reload its weight
  double w[R + 1][R + 1];
#pragma unroll
  for (int a = 0; a <= R; ++a)
#pragma unroll
    for (int b = 0; b <= a; ++b) {
      w[a][b] = W.w[(a + R) * n + (b + R)];
      asm volatile("" : "+d"(w[a][b]));
    }
  auto weight = [&](int dj, int di) {
    const int a = dj < 0 ? -dj : dj, b = di < 0 ? -di : di;
    return a >= b ? w[a][b] : w[b][a];
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
  const unsigned th = kFiltTY * kFiltVY;
  const dim3 grid((nelx + kFiltTX - 1) / kFiltTX, (nely + th - 1) / th, nrows), block(kFiltTX, kFiltTY);
#define STT_FILT(RR)                                                                                        \
  cone_filter_kernel<ADJ, RR><<<grid, block, 0, st>>>(in, in_rs, xt, xt_rs, out, xp, o_rs, nelx, nely, W, P)
  switch (R) {
    case 0: STT_FILT(0); break;
    case 1: STT_FILT(1); break;
    case 2: STT_FILT(2); break;
    case 3: STT_FILT(3); break;
    case 4: STT_FILT(4); break;
    case 5: STT_FILT(5); break;
    case 6: STT_FILT(6); break;
    default: STT_FILT(7);
  }
#undef STT_FILT
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
