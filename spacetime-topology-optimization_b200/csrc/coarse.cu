// The coarsest level's direct solve (sttopt/torch_mg.py:269-290, the dense Cholesky of the
// reference), in FP64 for both cycle precisions.
//
// The unknowns are grouped by grid line (a node row or column, along the shorter side), so
// the matrix is block tridiagonal with blocks of B = d * (nodes a line), padded to a
// multiple of 8.  The blocks are eliminated in odd-even order: at stride s = 1, 2, 4, ...
// every block i = s (2k + 1) still present is eliminated at once, which couples its
// neighbours i - s and i + s; block 0 is left last.  It is a Cholesky factorisation under
// a permutation, X_i = L_i^{-1}, F_l = X_i A_{i,i-s}, F_r = X_i A_{i,i+s}, so
//     forward   y_i = X_i b_i,  b_{i-s} -= F_l^T y_i,  b_{i+s} -= F_r^T y_i
//     backward  x_i = X_i^T (y_i - F_l x_{i-s} - F_r x_{i+s}).
// A chain over the lines (block k needs block k - 1) has nb dependent steps each way; this
// order has log2(nb), and the steps of one stride run side by side on a cluster of up to eight
// CTAs a row (fewer where there are many rows), which exchange through distributed shared memory.
//
// The order of the sums below was chosen among equally accurate ones: the parity tests of the
// product element form hold FP64 results to 1e-9 of dc and 5e-8 of the floating stage's c, which is
// what a change of omega by 1e-13 moves them by, so a change of rounding here can trip them.
#include "coarse.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "errors.h"
#include "smem.h"

namespace stt {

namespace cg = cooperative_groups;

constexpr int kTreeCluster = 8;  // CTAs a row, at most
constexpr int kTreeGroups = 2;   // thread groups of 4 B threads a CTA
constexpr size_t kTreeSmem = 225 << 10;  // dynamic shared memory a CTA of the solve may take

// One 8 x 8 tile product on the FP64 tensor cores (tcgen05 has no FP64 kind): lane
// (g, t) = (lane / 4, lane % 4) gives A[g][t] and B[t][g] and holds D[g][2t], D[g][2t + 1].
STT_DEV void dmma884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// ---- assembly ------------------------------------------------------------------------

// Entry between dof i of node a and dof j of node b from the half stencil (0 when the nodes
// are not neighbours); fixed dofs get a unit diagonal (their stencil rows are zero).
template <int D>
STT_DEV double line_entry(const double* __restrict__ sn, const uint8_t* __restrict__ fixed, long long nnode, int nnx,
                          int ra, int ca, int i, int rb, int cb, int j) {
  int dr = rb - ra, dc = cb - ca;
  if (dr < 0 || (dr == 0 && dc < 0)) {  // the half stencil is stored at the earlier node
    int t = ra; ra = rb; rb = t;
    t = ca; ca = cb; cb = t;
    t = i; i = j; j = t;
    dr = -dr;
    dc = -dc;
  }
  if (dr > 1 || dc > 1 || dc < -1) return 0.0;
  const long long n = (long long)ra * nnx + ca;
  int blk;
  if (dr == 0) {
    blk = dc;  // centre, E
    if (dc == 0) {
      if (i == j && ((fixed[n] >> i) & 1)) return 1.0;
      if (i < j) {
        const int t = i;
        i = j;
        j = t;
      }
    }
  } else {
    blk = dc == 0 ? 2 : (dc == 1 ? 3 : 4);  // S, SE, SW
  }
  return sn[(size_t)(blk * D * D + i * D + j) * nnode + n];
}

// A block's unknowns: `per` grid lines of `line` dofs each, one after the other (the last block may
// have fewer lines).
struct TreeBlock {
  int per, line, lines;
  // unknown i of block k as grid line and dof on it; false past the last
  STT_DEV bool at(int k, int i, int& row, int& dof) const {
    const int q = i / line, r = k * per + q;
    dof = i - q * line;
    row = r;
    return q < per && r < lines;
  }
};

// Diagonal blocks (slot 0) and the couplings to the previous block (slot 2), one CTA a block.
template <int D, bool SHARED>
__global__ void __launch_bounds__(256) tree_assemble_kernel(const double* __restrict__ st,
                                                            const uint8_t* __restrict__ fixed, int nnx, int nny,
                                                            int by_col, int B, double* __restrict__ blocks,
                                                            TreeBlock of) {
  const int k = blockIdx.x, h = blockIdx.y, nb = gridDim.x;
  const long long nnode = (long long)nnx * nny;
  const double* sn = st + (size_t)h * 5 * D * D * nnode;
  double* blk = blocks + ((size_t)h * nb + k) * 4 * B * B;
  // between dofs p and q of lines l and m
  auto entry = [&](int l, int p, int m, int q) {
    const int pa = p / D, i = p - pa * D, pb = q / D, j = q - pb * D;
    const int ra = by_col ? pa : l, ca = by_col ? l : pa;
    return line_entry<D>(sn, fixed, nnode, nnx, ra, ca, i, by_col ? pb : m, by_col ? m : pb, j);
  };
  for (int t = threadIdx.x; t < B * B; t += 256) {
    const int ii = t / B, jj = t - ii * B;
    double v = ii == jj ? 1.0 : 0.0, w = 0.0;  // the padding is an identity
    if constexpr (SHARED) {
      int l, m, p, q;
      if (of.at(k, ii, l, p)) {
        if (of.at(k, jj, m, q)) v = entry(l, p, m, q);
        if (k > 0 && of.at(k - 1, jj, m, q)) w = entry(l, p, m, q);
      }
    } else if (ii < of.line && jj < of.line) {
      v = entry(k, ii, k, jj);
      if (k > 0) w = entry(k, ii, k - 1, jj);
    }
    blk[t] = v;
    blk[(size_t)2 * B * B + t] = w;
  }
}

// ---- factorisation -------------------------------------------------------------------

// Tiles are 8 x 8; warp w of the CTA's 8 takes tiles w, w + 8, ... .  Shared rows are
// padded to B + 4 doubles, so the fragment loads of a half-warp hit distinct banks.
template <int NB>
struct TreeShared {
  static constexpr int B = 8 * NB, LD = B + 4;
  double A[B * LD];   // the block, then its factor L below the diagonal tiles
  double X[B * LD];   // L^{-1}
  double Cl[B * LD];  // A_{i,l}, then F_l
  double Cr[B * LD];  // A_{r,i}, then F_r
};

// Cholesky of the 8 x 8 diagonal tile p and its inverse by one warp: every lane factors the
// tile in registers (no shuffles on the pivots' chain), lane c < 8 forms column c of the
// inverse.
template <int NB>
STT_DEV bool tile_inverse(TreeShared<NB>& S, int p, int lane) {
  constexpr int LD = TreeShared<NB>::LD;
  double a[8][8], r[8];
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j) a[i][j] = S.A[(8 * p + i) * LD + 8 * p + j];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const double t = a[j][j];
    ok = ok && t > 0.0;
    r[j] = rsqrt(t > 0.0 ? t : 1.0);
#pragma unroll
    for (int i = j + 1; i < 8; ++i) a[i][j] *= r[j];
#pragma unroll
    for (int i = j + 1; i < 8; ++i)
#pragma unroll
      for (int k = j + 1; k <= i; ++k) a[i][k] = fma(-a[i][j], a[k][j], a[i][k]);
  }
  // column c of the inverse; the columns of lanes >= 8 repeat those of lane % 8
  const int c = lane & 7;
  double x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    double s = i == c ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < i; ++k) s = fma(-a[i][k], x[k], s);
    x[i] = s * r[i];
  }
  if (lane < 8)
#pragma unroll
    for (int i = 0; i < 8; ++i) S.X[(8 * p + i) * LD + 8 * p + c] = x[i];
  return ok;
}

// S.X = L^{-1} of S.A (lower tiles).  Right-looking over the diagonal tiles, the identity's
// columns carried along; three barriers a tile.
template <int NB>
STT_DEV void tree_cholesky_inverse(TreeShared<NB>& S, int* bad) {
  constexpr int LD = TreeShared<NB>::LD;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int p = 0; p < NB; ++p) {
    if (warp == 0 && !tile_inverse<NB>(S, p, lane) && lane == 0) *bad = 1;
    __syncthreads();
    // the panel: L_ip = A_ip X_pp^T below, X_pj = X_pp W_pj to the left
    if (warp < NB - 1) {
      const int i = warp < p ? warp : warp + 1;
      double d[2] = {0.0, 0.0};
      double* T = i < p ? &S.X[(8 * p) * LD + 8 * i] : &S.A[(8 * i) * LD + 8 * p];
      const double* Xp = &S.X[(8 * p) * LD + 8 * p];
#pragma unroll
      for (int k = 0; k < 8; k += 4) {
        if (i < p) dmma884(d, Xp[g * LD + k + t], T[(k + t) * LD + g]);
        else dmma884(d, T[g * LD + k + t], Xp[g * LD + k + t]);
      }
      __syncwarp();
      T[g * LD + 2 * t] = d[0];
      T[g * LD + 2 * t + 1] = d[1];
    }
    __syncthreads();
    // row tiles i > p: W_ij -= L_ip X_pj (j <= p), A_ij -= L_ip L_jp^T (p < j <= i)
    int idx = warp;
#pragma unroll 1
    for (int i = p + 1; i < NB; ++i) {
      const double* Li = &S.A[(8 * i) * LD + 8 * p];
#pragma unroll 1
      for (; idx <= i; idx += 8) {
        const int j = idx;
        double d[2] = {0.0, 0.0};
        double* T;
        if (j <= p) {
          T = &S.X[(8 * i) * LD + 8 * j];
          const double* Y = &S.X[(8 * p) * LD + 8 * j];
#pragma unroll
          for (int k = 0; k < 8; k += 4) dmma884(d, Li[g * LD + k + t], Y[(k + t) * LD + g]);
        } else {
          T = &S.A[(8 * i) * LD + 8 * j];
          const double* Lj = &S.A[(8 * j) * LD + 8 * p];
#pragma unroll
          for (int k = 0; k < 8; k += 4) dmma884(d, Li[g * LD + k + t], Lj[g * LD + k + t]);
        }
        double* o = T + g * LD + 2 * t;
        const bool fresh = j == p;  // W_ip starts at zero
        o[0] = (fresh ? 0.0 : o[0]) - d[0];
        o[1] = (fresh ? 0.0 : o[1]) - d[1];
      }
      idx -= i + 1;
    }
    __syncthreads();
  }
}

template <int NB>
STT_DEV void tree_load(double* s, const double* gsrc) {
  constexpr int B = 8 * NB, LD = B + 4;
  for (int t = threadIdx.x; t < B * B / 2; t += 256) {
    const int i = t / (B / 2), j = t - i * (B / 2);
    *reinterpret_cast<double2*>(s + i * LD + 2 * j) = __ldcg(reinterpret_cast<const double2*>(gsrc) + t);
  }
}

// The warp's tiles of op(P) Q over the whole depth: TP: P is used transposed, TQ: Q is.
// LOW: P is lower triangular (tiles above the diagonal are not read).
template <int NB, bool TP, bool TQ, bool LOW>
STT_DEV void tree_product(const double* P, const double* Q, double (&acc)[NB][2]) {
  constexpr int LD = 8 * NB + 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int q = 0; q < NB; ++q) acc[q][0] = acc[q][1] = 0.0;
#pragma unroll 1
  for (int k = 0; k < 8 * NB; k += 4) {
#pragma unroll
    for (int q = 0; q < (NB * NB + 7) / 8; ++q) {
      const int id = warp + 8 * q, i = id / NB, j = id - i * NB;
      if (id < NB * NB && !(LOW && k >= 8 * (i + 1))) {
        const double a = TP ? P[(k + t) * LD + 8 * i + g] : P[(8 * i + g) * LD + k + t];
        const double b = TQ ? Q[(8 * j + g) * LD + k + t] : Q[(k + t) * LD + 8 * j + g];
        dmma884(acc[q], a, b);
      }
    }
  }
}

// Calls put(row, column, pair) for each of the warp's accumulator pairs.
template <int NB, typename Put>
STT_DEV void tree_tiles(const double (&acc)[NB][2], Put put) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int q = 0; q < (NB * NB + 7) / 8; ++q) {
    const int id = warp + 8 * q, i = id / NB, j = id - i * NB;
    if (id < NB * NB) put(8 * i + g, 8 * j + 2 * t, make_double2(acc[q][0], acc[q][1]));
  }
}

// One row's factorisation on a cluster.  Latency-bound: a block's elimination is a chain of
// B pivots (about B/8 tile steps of one warp) and three B^3 products on the FP64 tensor
// cores; a stride's blocks are spread over the row's CTAs.  132 us for 33 lines of 40
// unknowns at 1 to 15 rows, 190 at 16 to 33, 706 at 128, 95 us for 46 lines of 32, where the banded factorisation (a chain
// over all unknowns on one CTA a row) took 871 and 1118 us.  Slots of block i: 0 the matrix
// block, then X_i; 1 F_l; 2 the coupling to the left neighbour still present; 3 F_r.
template <int NB>
__global__ void __launch_bounds__(256) tree_factor_kernel(double* blocks, int nb, int* status) {
  constexpr int B = 8 * NB, BB = B * B;
  extern __shared__ __align__(16) unsigned char tree_raw[];
  TreeShared<NB>& S = *reinterpret_cast<TreeShared<NB>*>(tree_raw);
  constexpr int LD = TreeShared<NB>::LD;
  __shared__ int bad;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x;
  double* bh = blocks + (size_t)blockIdx.y * nb * 4 * BB;
  if (tid == 0) bad = 0;
  __syncthreads();
  auto slot = [&](int i, int q) { return bh + ((size_t)i * 4 + q) * BB; };
  double acc[NB][2], acc2[NB][2];

  // factors block i with its neighbours l and r (-1: none); leaves F_l in S.Cl, F_r in S.Cr
  auto eliminate = [&](int i, int l, int r) {
    tree_load<NB>(S.A, slot(i, 0));
    if (l >= 0) tree_load<NB>(S.Cl, slot(i, 2));
    if (r >= 0) tree_load<NB>(S.Cr, slot(r, 2));
    __syncthreads();
    tree_cholesky_inverse<NB>(S, &bad);
    if (l >= 0) tree_product<NB, false, false, true>(S.X, S.Cl, acc);
    if (r >= 0) tree_product<NB, false, true, true>(S.X, S.Cr, acc2);
    __syncthreads();
    double* X = slot(i, 0);
    for (int t = tid; t < BB; t += 256) {
      const int a = t / B, c = t - a * B;
      X[t] = c <= a ? S.X[a * LD + c] : 0.0;
    }
    if (l >= 0) {
      double* F = slot(i, 1);
      tree_tiles<NB>(acc, [&](int a, int c, double2 v) {
        *reinterpret_cast<double2*>(S.Cl + a * LD + c) = v;
        *reinterpret_cast<double2*>(F + a * B + c) = v;
      });
    }
    if (r >= 0) {
      double* F = slot(i, 3);
      tree_tiles<NB>(acc2, [&](int a, int c, double2 v) {
        *reinterpret_cast<double2*>(S.Cr + a * LD + c) = v;
        *reinterpret_cast<double2*>(F + a * B + c) = v;
      });
    }
    __syncthreads();
  };
  auto subtract = [&](double* A) {
    tree_tiles<NB>(acc, [&](int a, int c, double2 v) {
      double2* o = reinterpret_cast<double2*>(A + a * B + c);
      const double2 u = __ldcg(o);
      *o = make_double2(u.x - v.x, u.y - v.y);
    });
  };

  for (int s = 1; s < nb; s *= 2) {
    const int step = 2 * s * (int)gridDim.x;
    int last = -1;
    for (int i = s * (2 * rank + 1); i < nb; i += step) {
      const int r = i + s < nb ? i + s : -1;
      eliminate(i, i - s, r);
      last = i;
      if (r >= 0) {  // the right neighbour's block and its new coupling
        tree_product<NB, true, false, false>(S.Cr, S.Cr, acc);
        tree_product<NB, true, false, false>(S.Cr, S.Cl, acc2);
        subtract(slot(r, 0));
        double* C = slot(r, 2);
        tree_tiles<NB>(acc2, [&](int a, int c, double2 v) {
          *reinterpret_cast<double2*>(C + a * B + c) = make_double2(-v.x, -v.y);
        });
        __syncthreads();
      }
    }
    cluster.sync();  // a block gets its two updates one after the other
    const int first = s * (2 * rank + 1);
    for (int i = first; i < nb; i += step) {
      if (first != last) {  // several blocks: S.Cl holds the last one's F_l
        __syncthreads();
        tree_load<NB>(S.Cl, slot(i, 1));
        __syncthreads();
      }
      tree_product<NB, true, false, false>(S.Cl, S.Cl, acc);
      subtract(slot(i - s, 0));
    }
    cluster.sync();
  }
  if (rank == 0) eliminate(0, -1, -1);
  if (tid == 0 && bad) atomicOr(status, 1);
}

// ---- solve ---------------------------------------------------------------------------

template <int NB>
STT_DEV void group_sync(int grp) {
  asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(32 * NB) : "memory");
}
STT_DEV void tree_cp16(void* smem, const void* gmem) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(gmem));
}

// Shared memory of a CTA (doubles): the solution in block order, then for each group its
// blocks' right-hand sides, the updates that arrive for them and scratch, then the staged
// matrices.
// (all: the row's thread groups)
__host__ __device__ inline int tree_own(int nb, int all) { return (nb + all - 1) / all; }  // blocks a group
__host__ __device__ inline size_t tree_vectors(int nb, int B, int all) {
  return (size_t)nb * B + kTreeGroups * (5 * (size_t)tree_own(nb, all) * B + 10 * B);
}
__host__ __device__ inline size_t tree_task(int B) { return 3 * (size_t)B * B; }  // X, F_l, F_r of one block

// One row's solve on a cluster: 2 log2(nb) steps, each a group of 4 B threads' two dependent
// block products.  Bound by the steps' latency, so the blocks (constant over the solve) are
// fetched once, at the start, into the shared memory of the CTA that will use them (the
// first `staged` blocks of a group; later ones are read from L2 when their turn comes):
// loads issued before a cluster barrier are waited for by it, and cost a memory latency a
// step.  33 lines of 40 unknowns, from L2 and from memory: 24 and 24 to 27 us at 1 to 15 rows (30
// unstaged), 34 and 46 to 48 at 16 to 33, 42 and 63 at 64, 75 and 92 at 128; the chain of banded
// block solves this replaces took 125 us.  (One product with an explicit inverse took less for few
// rows of wide lines: a V-cycle over 27 lines of 54 at one row in FP32 29 us, 37 with this, after
// 1.7 ms of forming the hierarchy where 0.33 are enough.)  The blocks are
// dealt out to the groups in the order of their elimination, so every group has nearly the
// same number.  A block's right-hand side lives in the CTA whose group owns it; its two
// neighbours' updates arrive there by remote stores into a buffer a side (two sets, used by
// alternate strides, so that a set is read before it is written again) and are added by the
// owner in a fixed order; a solution block is written to all of the row's CTAs.
template <int NB, int CL>
struct TreeRow {
  static constexpr int B = 8 * NB, NC = 2 * NB, BB = B * B, kGroup = 4 * B;
  static constexpr int kThreads = kTreeGroups * kGroup;

  const double* bh;  // the row's factor [nb][4][B][B]
  int nb, staged, own, levels, rank, grp, t, gi;
  int lg, all;  // the row's thread groups, 2^lg
  double *vx, *vb, *in, *tv, *part, *stage;

  STT_DEV void init(double* sm, const double* factor, int nblocks, int nstaged) {
    cg::cluster_group cluster = cg::this_cluster();
    bh = factor;
    nb = nblocks;
    staged = nstaged;
    all = (CL ? CL : (int)gridDim.x) * kTreeGroups;
    lg = 31 - __clz(all);
    own = tree_own(nb, all);
    levels = 0;
    while ((1 << levels) < nb) ++levels;
    rank = (int)cluster.block_rank();
    grp = (int)threadIdx.x / kGroup;
    t = (int)threadIdx.x - grp * kGroup;
    gi = rank * kTreeGroups + grp;
    vx = sm;
    vb = vx + (size_t)nb * B;                       // [grp][own][B]: right-hand sides, then y
    in = vb + (size_t)kTreeGroups * own * B;        // [set][side][grp][own][B]
    tv = in + (size_t)4 * kTreeGroups * own * B + grp * 10 * B;
    part = tv + 2 * B;
    stage = vx + tree_vectors(nb, B, all) + (size_t)grp * staged * 3 * BB;
  }

  // blocks in the order of elimination: those of stride 2^l are numbers base(l) .. base(l + 1),
  // the root (block 0) is the last; number o is the o / all-th block of group o % all
  STT_DEV int base(int l) const { return nb - ((nb + (1 << l) - 1) >> l); }
  STT_DEV int number(int e) const {
    if (e == 0) return nb - 1;
    const int l = __ffs(e) - 1;
    return base(l) + (e >> (l + 1));
  }
  STT_DEV int block_of(int o, int l) const { return (1 << l) * (2 * (o - base(l)) + 1); }
  // where block e's vectors live: the CTA, and the offset in an array [grp][own][B]
  STT_DEV int owner(int e) const { return (number(e) & (all - 1)) / kTreeGroups; }
  STT_DEV int place(int e) const {
    const int o = number(e);
    return ((o % kTreeGroups) * own + (o >> lg)) * B;
  }
  STT_DEV double* updates(int set, int side) const { return in + (size_t)((2 * set + side) * kTreeGroups) * own * B; }
  // calls f(block, j) for the group's blocks in their order, j = 0, 1, ...
  template <typename F>
  STT_DEV void each_block(F f) const {
    int l = 0, j = 0;
    for (int o = gi; o < nb; o += all, ++j) {
      while (l < levels && o >= base(l + 1)) ++l;
      f(o == nb - 1 ? 0 : block_of(o, l), j, l);
    }
  }

  // starts fetching the blocks (the first in a copy group of its own)
  STT_DEV void prefetch() {
    each_block([&](int i, int j, int l) {
      if (j < staged) {
        double* dst = stage + (size_t)j * 3 * BB;
        const double* src = bh + (size_t)i * 4 * BB;
        const int n01 = i == 0 ? BB : 2 * BB;  // X and F_l lie side by side
        for (int c = 2 * t; c < n01; c += 2 * kGroup) tree_cp16(dst + c, src + c);
        if (i != 0 && i + (1 << l) < nb)
          for (int c = 2 * t; c < BB; c += 2 * kGroup) tree_cp16(dst + 2 * BB + c, src + 3 * BB + c);
      }
      if (j == 0) asm volatile("cp.async.commit_group;\n" ::);
    });
    asm volatile("cp.async.commit_group;\n" ::);
  }

  // the matrices (k = 0: X, 1: F_l, 2: F_r) of the group's j-th block, i
  STT_DEV const double* matrix(int j, int i, int k) const {
    return j < staged ? stage + ((size_t)j * 3 + k) * BB : bh + ((size_t)i * 4 + (k == 2 ? 3 : k)) * BB;
  }
  // row-wise product: row t / 4, column pairs t % 4, t % 4 + 4, ...; summed over the quad
  STT_DEV double row_dot(const double* M, const double* v) const {
    const int q = t & 3;
    const double2* m = reinterpret_cast<const double2*>(M + (size_t)(t >> 2) * B) + q;
    const double2* w = reinterpret_cast<const double2*>(v) + q;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int c = 0; c < NC / 2; ++c) {
      const double2 mm = m[4 * c], ww = w[4 * c];
      s0 = fma(mm.x, ww.x, s0);
      s1 = fma(mm.y, ww.y, s1);
    }
    return s0 + s1;
  }
  STT_DEV static double quad(double s) {
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s;
  }
  // column-wise partial product: column t % B, quarter t / B of the rows
  STT_DEV double col_dot(const double* M, const double* v) const {
    const int p4 = t / B, j4 = t - p4 * B;
    const double* m = M + (size_t)(p4 * NC) * B + j4;
    const double2* w = reinterpret_cast<const double2*>(v + p4 * NC);
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int c = 0; c < NC / 2; ++c) {
      const double2 ww = w[c];
      s0 = fma(m[(2 * c) * B], ww.x, s0);
      s1 = fma(m[(2 * c + 1) * B], ww.y, s1);
    }
    return s0 + s1;
  }
  STT_DEV static double parts(const double* pp, int j) { return (pp[j] + pp[B + j]) + (pp[2 * B + j] + pp[3 * B + j]); }

  // Solves for the right-hand sides in vb (complete and visible: the caller synchronises the
  // cluster first); publish(i, t, v) is called by the owner for each unknown t of block i.
  template <typename Publish>
  STT_DEV void solve(Publish publish) {
    cg::cluster_group cluster = cg::this_cluster();
    int o = gi, j = 0;  // the group's next block
    bool landed = false;
    auto wait_stage = [&](bool first) {
      if (landed) return;
      if (first) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
      else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      landed = !first;
    };
    const int q = t & 3, i4 = t >> 2;
    const size_t go = (size_t)grp * own * B;
    double* vg = vb + go;
    for (int l = 0; l < levels; ++l) {
      const int s = 1 << l, end = base(l + 1);
      double* inL = updates(l & 1, 0);
      double* inR = updates(l & 1, 1);
      for (; o < end; o += all, ++j) {
        const int i = block_of(o, l);
        const bool right = i + s < nb;
        wait_stage(j == 0);
        if (t < B) tv[t] = vg[j * B + t];
        group_sync<NB>(grp);
        const double y = quad(row_dot(matrix(j, i, 0), tv));
        if (q == 0) {
          tv[B + i4] = y;
          vg[j * B + i4] = y;
        }
        group_sync<NB>(grp);
        part[t] = col_dot(matrix(j, i, 1), tv + B);
        if (right) part[4 * B + t] = col_dot(matrix(j, i, 2), tv + B);
        group_sync<NB>(grp);
        if (t < B)
          cluster.map_shared_rank(inR, owner(i - s))[place(i - s) + t] = parts(part, t);
        else if (t < 2 * B && right)
          cluster.map_shared_rank(inL, owner(i + s))[place(i + s) + (t - B)] = parts(part + 4 * B, t - B);
        group_sync<NB>(grp);
      }
      cluster.sync();
      // the updates of the own blocks that are left
      if (t < B) {
        int l2 = l + 1, j2 = j;
        for (int o2 = o; o2 < nb; o2 += all, ++j2) {
          while (l2 < levels && o2 >= base(l2 + 1)) ++l2;
          const int a = j2 * B + t;
          if (o2 == nb - 1)
            vg[a] -= inR[go + a];
          else
            vg[a] = (vg[a] - inL[go + a]) - (block_of(o2, l2) + s < nb ? inR[go + a] : 0.0);
        }
      }
    }
    auto finish = [&](int i, bool share) {  // x_i = X_i^T z from the group's partial sums
      if (t < B) {
        const double v = parts(part, t);
        if (share)
#pragma unroll
          for (int rk = 0; rk < kTreeCluster; ++rk)
            if (rk < (CL ? CL : (int)gridDim.x)) cluster.map_shared_rank(vx, rk)[i * B + t] = v;
        publish(i, t, v);
      }
    };
    if (o == nb - 1) {  // the root's group
      wait_stage(j == 0);
      if (t < B) tv[t] = vg[j * B + t];
      group_sync<NB>(grp);
      const double y = quad(row_dot(matrix(j, 0, 0), tv));
      if (q == 0) tv[B + i4] = y;
      group_sync<NB>(grp);
      part[t] = col_dot(matrix(j, 0, 0), tv + B);
      group_sync<NB>(grp);
      finish(0, nb > 1);
    }
    o -= all;
    --j;
    for (int l = levels - 1; l >= 0; --l) {
      const int s = 1 << l, begin = base(l);
      cluster.sync();
      for (; o >= begin; o -= all, --j) {
        const int i = block_of(o, l);
        group_sync<NB>(grp);
        double z = row_dot(matrix(j, i, 1), vx + (i - s) * B);
        if (i + s < nb) z += row_dot(matrix(j, i, 2), vx + (i + s) * B);
        z = quad(z);
        if (q == 0) tv[i4] = vg[j * B + i4] - z;
        group_sync<NB>(grp);
        part[t] = col_dot(matrix(j, i, 0), tv);
        group_sync<NB>(grp);
        finish(i, l > 0);
      }
    }
  }
};

// One row's coarse solve on a cluster (TreeRow), between global vectors.  SHARED: a block may hold
// several grid lines (24 or 32 unknowns; without it the index arithmetic of one line a block is
// simpler, and the kernel 0.7 us shorter).  CL: the CTAs a row, or 0
// for any (tree_eight).
template <int NB, int D, typename T, bool SHARED, int CL>
__global__ void __launch_bounds__(TreeRow<NB, CL>::kThreads)
    tree_solve_kernel(const T* __restrict__ b, T* __restrict__ x, long long rs, const double* __restrict__ blocks,
                      int nb, int staged, int by_col, int nnx, int nny, const uint8_t* __restrict__ fixed,
                      const int* __restrict__ row_map, int hrows, const RowState* __restrict__ rst, TreeBlock of) {
  constexpr int B = 8 * NB;
  extern __shared__ __align__(16) double sm[];
  const int srow = blockIdx.y;
  TreeRow<NB, CL> tree;
  // The factor is fetched beside the kernel before: it is complete when its solves are launched
  // (the stream has waited for its event).  A row map is the caller's, and on a hierarchy of one
  // level the kernel before may be the one that writes it.
  if (row_map) grid_wait();
  tree.init(sm, blocks + (size_t)hier_row(row_map, hrows, srow) * nb * 4 * B * B, nb, staged);
  tree.prefetch();
  if (!row_map) grid_wait();
  if (rst && !rst[srow].active) {  // the whole cluster
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    return;
  }
  const T* bs = b + (size_t)srow * rs;
  T* xs = x + (size_t)srow * rs;
  const int used = D * (by_col ? nny : nnx);
  auto has = [&](int k, int ii) {
    if constexpr (!SHARED) return ii < used;
    int row, dof;
    return of.at(k, ii, row, dof);
  };
  auto dof_of = [&](int k, int ii, long long& node, int& d) {
    if constexpr (SHARED) of.at(k, ii, k, ii);
    const int pos = ii / D;
    d = ii - pos * D;
    node = by_col ? (long long)pos * nnx + k : (long long)k * nnx + pos;
  };
  tree.each_block([&](int i, int j, int) {
    if (tree.t >= B) return;
    double v = 0.0;
    if (has(i, tree.t)) {
      long long node;
      int d;
      dof_of(i, tree.t, node, d);
      v = (double)bs[node * D + d];
    }
    tree.vb[(tree.grp * tree.own + j) * B + tree.t] = v;
  });
  cg::this_cluster().sync();
  tree.solve([&](int i, int ii, double v) {
    if (!has(i, ii)) return;
    long long node;
    int d;
    dof_of(i, ii, node, d);
    xs[node * D + d] = ((fixed[node] >> d) & 1) ? T(0) : T(v);
  });
}

// ---- host ----------------------------------------------------------------------------

#define STT_TREE_DISPATCH(B, M) \
  switch ((B) / 8) {            \
    case 1: M(1); break;        \
    case 2: M(2); break;        \
    case 3: M(3); break;        \
    case 4: M(4); break;        \
    case 5: M(5); break;        \
    case 6: M(6); break;        \
    case 7: M(7); break;        \
    default: M(8); break;       \
  }

// Lines of up to 64 unknowns go by odd-even elimination; wider ones (a coarsest grid of more
// than ~700 elements) by the banded factorisation, whose blocks are a multiple of 32 no
// smaller than the half bandwidth.  Many short lines go several to a block of up to 32 unknowns (a
// step costs hardly more than with 8, and there are fewer): 601 lines of 2 unknowns one by one took 91 us
// a V-cycle at 1 row and 500 at 128, the banded chain 82 and 116, in blocks of 16 lines 28 and 96.
// A long grid's vectors fill a CTA's shared memory, so a row takes all eight CTAs and 15 rows run at
// once: 501 lines of 28 unknowns 129 us at 1 row, 614 at 33, 1970 at 128, where the chain takes 771,
// 1110 and 1160.  Past kLongUnknowns (the rule of tree_launch needs that much room) more than
// kLongRows rows take the chain, and all where the vectors do not fit.
constexpr int kLongUnknowns = 5376, kLongRows = 64;
void coarse_plan(const LevelDesc& c, int d, int hrows, CoarseDesc& co) {
  co.n = (int)c.ndof;
  co.by_col = c.nny < c.nnx ? 1 : 0;
  const int nmin = co.by_col ? c.nny : c.nnx, lines = co.by_col ? c.nnx : c.nny;
  co.per = lines > 64 ? std::max(1, 32 / (d * nmin)) : 1;  // (more than one: 22 to 32 unknowns)
  co.B = (co.per * d * nmin + 7) / 8 * 8;
  co.nb = (lines + co.per - 1) / co.per;
  co.tree = co.B <= 64 && 8 * tree_vectors(co.nb, co.B, kTreeCluster * kTreeGroups) <= kTreeSmem &&
                    (hrows <= kLongRows || (long long)co.B * co.nb <= kLongUnknowns)
                ? 1
                : 0;
  if (co.tree) return;
  const int bw = d * (nmin + 2) - 1;  // max |P - Q| of a nonzero
  co.B = (bw + 31) / 32 * 32;
  co.nb = (co.n + co.B - 1) / co.B;
}

// How many clusters of `cluster` CTAs the device holds at once, 0 if none (several kinds of launch a
// kernel: the answers are kept, at most kMax of them).
template <auto Kernel>
static int resident_clusters(int cluster, int threads, size_t smem, int* n) {
  struct Known {
    int dev, cluster, n;
    size_t smem;
  };
  constexpr int kMax = 64;
  static std::mutex mu;
  static Known known[kMax];
  static int count = 0;
  int dev = 0;
  STT_TRY(check_cuda(cudaGetDevice(&dev), "cudaGetDevice"));
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < count; ++i)
    if (known[i].dev == dev && known[i].cluster == cluster && known[i].smem == smem) {
      *n = known[i].n;
      return STT_OK;
    }
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(n, Kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    *n = 0;  // the device takes none of this size
  }
  // clusters of eight with more than one CTA an SM leave gaps: of 33 and of 48, 28 and 40 ran at once
  if (cluster == kTreeCluster && *n * cluster > 148) *n -= *n / 8;
  if (count == kMax) count = 0;
  known[count++] = Known{dev, cluster, *n, smem};
  return STT_OK;
}

// Dependent block eliminations of one sweep over the strides with `units` blocks side by side.
static int tree_steps(int nb, int units) {
  int steps = 1;  // the root
  for (int n = nb; n > 1; n = (n + 1) / 2) steps += (n / 2 + units - 1) / units;
  return steps;
}

// The launch that is expected to end first: its waves of resident clusters times a row's steps,
// times what a step costs there.  Fewer CTAs a row take more steps but let more rows run at once
// (15 clusters of eight, 33 of four, 74 of two on B200's 148 SMs at one CTA each).  A V-cycle of a
// one-level hierarchy, 33 lines of 40 unknowns, always eight CTAs -> this rule: 16 rows 51 -> 39 us,
// 33 rows 74 -> 40, 64 rows 122 -> 55, 128 rows 223 -> 86 (the chain over the lines: 147 to 162); 27
// lines of 54 at 128 rows 404 -> 179 (204), their factorisation 2.2 -> 1.35 ms (1.33).  The
// rows' results do not depend on it.
struct TreeLaunch {
  int cluster = 0, staged = 0;
  size_t smem = 0;
  long long cost = 0;
  void consider(int rows, int resident, int cl, int st, size_t bytes, int row_cost) {
    if (resident < 1) return;
    const long long c = (long long)((rows + resident - 1) / resident) * row_cost;
    if (cluster == 0 || c < cost) *this = TreeLaunch{cl, st, bytes, c};
  }
};

static TreeBlock tree_block(const stt_hier* h) {
  const LevelDesc& lv = h->lv[h->nlevels - 1];
  const bool col = h->co.by_col;
  return TreeBlock{h->co.per, h->d * (col ? lv.nny : lv.nnx), col ? lv.nnx : lv.nny};
}

template <int NB>
static int tree_factor(const CoarseDesc& co, int hrows, int* status, cudaStream_t st) {
  constexpr int kThreads = 256;
  STT_TRY(allow_smem<tree_factor_kernel<NB>>());
  TreeLaunch best;
  for (int cl = kTreeCluster; cl >= 1; cl /= 2) {
    int n = 0;
    STT_TRY(resident_clusters<tree_factor_kernel<NB>>(cl, kThreads, sizeof(TreeShared<NB>), &n));
    best.consider(hrows, n, cl, 0, sizeof(TreeShared<NB>), tree_steps(co.nb, cl));
  }
  if (best.cluster == 0) return set_error(STT_ERR_CUDA, "coarse factor: no cluster fits the device");
  launch_clusters(tree_factor_kernel<NB>, best.cluster, dim3(best.cluster, hrows), kThreads, best.smem, st, false,
                  co.blocks, co.nb, status);
  return check_launch("coarse factor");
}

// The form of the kernel for eight CTAs a row: with their number fixed it is 0.5 us shorter up to 32
// unknowns a block (17.0 us for 25 lines of 26), and longer from 40 on (24.1 and 23.7 us for 33
// lines of 34, 39.8 and 33.6 for 27 of 54).
template <int NB>
constexpr int tree_eight() {
  return NB <= 4 ? kTreeCluster : 0;
}

// A solve's launch: each cluster size with as many blocks staged as fit its CTAs, and with none
// (more CTAs an SM).  A step without its block staged takes about 1.4 times as long.
template <int NB, int D, typename T, bool SHARED>
static int tree_launch(const CoarseDesc& co, int nrows, TreeLaunch& best) {
  constexpr auto eight = tree_solve_kernel<NB, D, T, SHARED, tree_eight<NB>()>;
  constexpr auto any = tree_solve_kernel<NB, D, T, SHARED, 0>;
  constexpr int kThreads = TreeRow<NB, 0>::kThreads;
  STT_TRY(allow_smem<eight>());
  STT_TRY(allow_smem<any>());
  const size_t task = 8 * kTreeGroups * tree_task(co.B);
  for (int cl = kTreeCluster; cl >= 1; cl /= 2) {
    const int all = cl * kTreeGroups, own = tree_own(co.nb, all), steps = tree_steps(co.nb, all);
    const size_t vec = 8 * tree_vectors(co.nb, co.B, all);
    if (vec > kTreeSmem) break;
    const int most = (int)std::min<size_t>(own, (kTreeSmem - vec) / task);
    for (int st : {most, 0}) {
      const size_t bytes = vec + st * task;
      int n = 0;
      STT_TRY(cl == kTreeCluster ? resident_clusters<eight>(cl, kThreads, bytes, &n)
                                 : resident_clusters<any>(cl, kThreads, bytes, &n));
      best.consider(nrows, n, cl, st, bytes, steps * (st == own ? 5 : 7));
    }
    if (cl == kTreeCluster && most == own && best.cost == 5 * steps) break;  // one wave: nothing is faster
  }
  return best.cluster ? STT_OK : set_error(STT_ERR_CUDA, "coarse solve: no cluster fits the device");
}

template <int NB, int D, typename T, bool SHARED>
static int tree_run(const stt_hier* h, int nrows, const T* b, T* x, long long rs, const RowState* rst,
                    cudaStream_t st) {
  const LevelDesc& lv = h->lv[h->nlevels - 1];
  const CoarseDesc& co = h->co;
  TreeLaunch l;
  STT_TRY((tree_launch<NB, D, T, SHARED>(co, nrows, l)));
  auto* const kernel = l.cluster == kTreeCluster ? tree_solve_kernel<NB, D, T, SHARED, tree_eight<NB>()>
                                                 : tree_solve_kernel<NB, D, T, SHARED, 0>;
  launch_clusters(kernel, l.cluster, dim3(l.cluster, nrows), TreeRow<NB, 0>::kThreads, l.smem, st, true, b, x, rs,
                  co.blocks, co.nb, l.staged, co.by_col, lv.nnx, lv.nny, lv.fixed, h->row_map, h->hrows, rst,
                  tree_block(h));
  return check_launch("coarse solve");
}

template <int NB, int D, typename T>
static int tree_solve(const stt_hier* h, int nrows, const T* b, T* x, long long rs, const RowState* rst,
                      cudaStream_t st) {
  if constexpr (NB == 3 || NB == 4)
    if (h->co.per > 1) return tree_run<NB, D, T, true>(h, nrows, b, x, rs, rst, st);
  return tree_run<NB, D, T, false>(h, nrows, b, x, rs, rst, st);
}

int coarse_factor(const stt_hier* h, cudaStream_t st) {
  const LevelDesc& lv = h->lv[h->nlevels - 1];
  const CoarseDesc& co = h->co;
  const dim3 g(co.nb, h->hrows);
#define STT_ASSEMBLE(D, SHARED)                                                                                     \
  tree_assemble_kernel<D, SHARED><<<g, 256, 0, st>>>(lv.st64, lv.fixed, lv.nnx, lv.nny, co.by_col, co.B, co.blocks, \
                                                     tree_block(h))
  if (h->d == 2) {
    if (co.per > 1) STT_ASSEMBLE(2, true);
    else STT_ASSEMBLE(2, false);
  } else {
    if (co.per > 1) STT_ASSEMBLE(1, true);
    else STT_ASSEMBLE(1, false);
  }
#undef STT_ASSEMBLE
  STT_TRY(check_launch("coarse assemble"));
#define STT_FACTOR(NB) return tree_factor<NB>(co, h->hrows, h->status, st)
  STT_TREE_DISPATCH(co.B, STT_FACTOR)
#undef STT_FACTOR
}

template <typename T>
int coarse_tree_solve(const stt_hier* h, int nrows, const T* b, T* x, long long rs, const RowState* rst,
                      cudaStream_t st) {
#define STT_SOLVE(NB)                                                       \
  return h->d == 2 ? tree_solve<NB, 2, T>(h, nrows, b, x, rs, rst, st)      \
                   : tree_solve<NB, 1, T>(h, nrows, b, x, rs, rst, st)
  STT_TREE_DISPATCH(h->co.B, STT_SOLVE)
#undef STT_SOLVE
}

template int coarse_tree_solve<float>(const stt_hier*, int, const float*, float*, long long, const RowState*,
                                      cudaStream_t);
template int coarse_tree_solve<double>(const stt_hier*, int, const double*, double*, long long, const RowState*,
                                       cudaStream_t);

}  // namespace stt
