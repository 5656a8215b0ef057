// jg_linelet.cu -- the line-implicit preconditioner of BCGSTAB_LINELET.
//
// initializeLinelet (src/joe/JoeWithModels.cpp:7471-7559) grows, from each
// cell on a WALL face, a line of cells in the direction of strong coupling;
// solveCvVectorR5BcgstabLine (src/common/UgpWithCv.cpp:3627-3992) is
// BiCGSTAB whose preconditioner solves the block-tridiagonal system of each
// line exactly (block Thomas elimination) and the block diagonal elsewhere.
//
// Here the lines are built once per handle on the host.  The LINE relaxation
// (below) uses the same rule with one relaxation: where several neighbours
// pass, the line goes on to the strongest if it is 1.1 times the next one,
// so that a line crosses from the last prism row into the hexahedron above
// (whose other lower neighbour is the quad's second prism).  On the device the
// elimination is split in two: k_line_factor runs once per linear solve (the
// matrix does not change inside BiCGSTAB) and keeps, per line cell, the
// inverse of the eliminated diagonal block, the multiplier
// A(c_i, c_{i-1}) inv_{i-1} and the upper block A(c_{i-1}, c_i); k_line_apply
// then does the forward and backward substitutions for one right-hand side
// (twice per BiCGSTAB iteration).  The reference recomputes the elimination
// inside every application; the factors are the same numbers.  One warp per
// line: the lines are independent, and inside a line the work is a chain of
// 5x5 block operations, so the warp's lanes hold the 25 entries (factor) or
// the 5 rows (substitutions) of one block step.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "jg_internal.h"
#include "jg_sweep.cuh"

namespace jg {

namespace {

// findFace (JoeWithModels.cpp:7572-7587): the first face of a's list that b also has
int find_face(const jg_mesh& m, int a, int b) {
  if (a == b) return -1;
  for (int i = m.faocv_i[a]; i < m.faocv_i[a + 1]; i++)
    for (int j = m.faocv_i[b]; j < m.faocv_i[b + 1]; j++)
      if (m.faocv_v[i] == m.faocv_v[j]) return m.faocv_v[i];
  return -1;
}

double coupling(const jg_mesh& m, int a, int b) {
  int f = find_face(m, a, b);
  const double* n = &m.fa_normal[3 * f];
  double area = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
  return 0.5 * area * ((1.0 / m.cv_volume[a]) + (1.0 / m.cv_volume[b]));
}

}  // namespace

int build_lines(const jg_mesh& m, const std::vector<std::vector<int>>& wall_zones, std::vector<int>& off,
                std::vector<int>& cv, bool relaxed) {
  const int N = m.ncv;
  std::vector<char> free_cv(N, 1);
  // each WALL zone replaces the sources of the one before it (relaxed: every WALL zone's cells are
  // sources, so that each case of a batch grows its own lines); all of their cells leave the pool
  std::vector<int> src;
  for (const auto& z : wall_zones) {
    if (!relaxed) src.clear();
    for (int f : z) {
      src.push_back(m.cvofa[2 * f]);
      free_cv[m.cvofa[2 * f]] = 0;
    }
  }
  off.assign(1, 0);
  cv.clear();
  // a cell with several WALL faces is a source for each of them.  The reference grows a line from each;
  // relaxed: one line only, since the LINE relaxation solves a cell's system once (the cell's couplings
  // to two lines would be counted in both, and both would write its unknowns)
  std::vector<char> headed(relaxed ? N : 0, 0);
  for (int s : src) {
    if (relaxed) {
      if (headed[s]) continue;
      headed[s] = 1;
    }
    const size_t first = cv.size();
    cv.push_back(s);
    for (;;) {
      const int icv = cv.back();
      double wmax = 0.0;
      for (int k = m.nbocv_i[icv] + 1; k < m.nbocv_i[icv + 1]; k++)
        wmax = std::max(wmax, coupling(m, icv, m.nbocv_v[k]));
      // the one free neighbour (not the cell the line came from) with more than half the largest
      // coupling; relaxed: or, among several, the strongest when it is 1.1 times the next one
      int next = -1, count = 0;
      double best_w = 0.0, second_w = 0.0;
      const int prev = cv.size() - first >= 2 ? cv[cv.size() - 2] : -1;
      for (int k = m.nbocv_i[icv] + 1; k < m.nbocv_i[icv + 1]; k++) {
        const int nb = m.nbocv_v[k];
        const double w = coupling(m, icv, nb);
        if (free_cv[nb] && w / wmax > 0.5 && nb != prev) {
          count++;
          if (w > best_w) {
            second_w = best_w;
            best_w = w;
            next = nb;
          } else if (w > second_w) {
            second_w = w;
          }
        }
      }
      if (count == 0 || (count > 1 && !(relaxed && best_w > 1.1 * second_w))) break;
      cv.push_back(next);
      free_cv[next] = 0;
    }
    off.push_back((int)cv.size());
  }
  return JG_OK;
}

namespace {

constexpr int LW = 4;  // warps (lines) per block

// ludeco (UgpWithCv.cpp:2489-2516) on a row-major 5x5 block
__device__ void ludeco5(double* A) {
#pragma unroll
  for (int jc = 1; jc < 5; jc++) A[jc] /= A[0];
#pragma unroll
  for (int jrjc = 1; jrjc < 5; jrjc++) {
#pragma unroll
    for (int jr = jrjc; jr < 5; jr++) {
      double sum = A[5 * jr + jrjc];
#pragma unroll
      for (int jm = 0; jm < jrjc; jm++) sum -= A[5 * jr + jm] * A[5 * jm + jrjc];
      A[5 * jr + jrjc] = sum;
    }
    if (jrjc == 4) break;
#pragma unroll
    for (int jc = jrjc + 1; jc < 5; jc++) {
      double sum = A[5 * jrjc + jc];
#pragma unroll
      for (int jm = 0; jm < jrjc; jm++) sum -= A[5 * jrjc + jm] * A[5 * jm + jc];
      A[5 * jrjc + jc] = sum / A[5 * jrjc + jrjc];
    }
  }
}

// column `col` of the inverse from the ludeco factors, as luinv (UgpWithCv.cpp:2542-2577)
__device__ void luinv_col(const double* A, int col, double* c) {
#pragma unroll
  for (int i = 0; i < 5; i++) c[i] = (i == col) ? 1.0 : 0.0;
  c[0] = c[0] / A[0];
#pragma unroll
  for (int jr = 1; jr < 5; jr++) {
    double sum = c[jr];
#pragma unroll
    for (int jm = 0; jm < jr; jm++) sum -= A[5 * jr + jm] * c[jm];
    c[jr] = sum / A[5 * jr + jr];
  }
#pragma unroll
  for (int jr = 3; jr >= 0; jr--) {
    double sum = c[jr];
#pragma unroll
    for (int jm = 4; jm > jr; jm--) sum -= A[5 * jr + jm] * c[jm];
    c[jr] = sum;
  }
}

// entry e of the matrix block A(row, col): the ELL columns of `row` whose neighbour is `col`
__device__ double ell_block(const Mesh& m, const double* O, int row, int col, int e) {
  const int s = row / SLICE, lane = row % SLICE;
  double v = 0.0;
  for (int j = m.ell_off[s]; j < m.ell_off[s + 1]; j++)
    if (m.ell_nb[(size_t)j * SLICE + lane] == col) v += O[((size_t)j * 25 + e) * SLICE + lane];
  return v;
}
// the block at ELL row j (Lines::jlo / jup), or the search where the two cells share several faces
__device__ __forceinline__ double ell_block_j(const Mesh& m, const double* O, int row, int col, int j, int e) {
  if (j >= 0) return O[((size_t)j * 25 + e) * SLICE + row % SLICE];
  return j == -1 ? 0.0 : ell_block(m, O, row, col, e);
}

__global__ void __launch_bounds__(32 * LW) k_line_factor(Mesh m, State st, Lines L) {
  __shared__ double sh[LW][5][25];
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int line = blockIdx.x * LW + w;
  if (line >= L.nlines) return;
  double *b = sh[w][0], *inv = sh[w][1], *lo = sh[w][2], *up = sh[w][3], *mh = sh[w][4];
  const int p0 = L.off[line], n = L.off[line + 1] - p0;
  const int N = m.ncv;
  const double* D = (const double*)st.D;
  const double* O = (const double*)st.O;
  const int e = lane < 25 ? lane : 24, r = e / 5, k = e % 5;
  if (lane < 25) b[e] = D[(size_t)e * N + L.cv[p0]];
  __syncwarp();
  for (int i = 1;; i++) {
    // inverse of the eliminated diagonal block of position i-1
    if (lane < 5) {
      double A[25], c[5];
#pragma unroll
      for (int q = 0; q < 25; q++) A[q] = b[q];
      ludeco5(A);
      luinv_col(A, lane, c);
#pragma unroll
      for (int q = 0; q < 5; q++) inv[5 * q + lane] = c[q];
    }
    __syncwarp();
    if (lane < 25) L.inv[(size_t)(p0 + i - 1) * 25 + e] = inv[e];
    if (i == n) break;
    const int cp = L.cv[p0 + i - 1], c = L.cv[p0 + i];
    if (lane < 25) {
      lo[e] = ell_block_j(m, O, c, cp, L.jlo[p0 + i], e);
      up[e] = ell_block_j(m, O, cp, c, L.jup[p0 + i], e);
      L.up[(size_t)(p0 + i) * 25 + e] = up[e];
    }
    __syncwarp();
    // mhat = A(c, cp) inv (getMultMatrix order: sums from 0.0 over q)
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 5; q++) s += lo[5 * r + q] * inv[5 * q + k];
    if (lane < 25) {
      mh[e] = s;
      L.low[(size_t)(p0 + i) * 25 + e] = s;
    }
    __syncwarp();
    // next diagonal: A(c, c) - mhat A(cp, c)
    double a0 = 0.0;
#pragma unroll
    for (int q = 0; q < 5; q++) a0 += mh[5 * r + q] * up[5 * q + k];
    const double bn = D[(size_t)e * N + c] - a0;
    __syncwarp();
    if (lane < 25) b[e] = bn;
    __syncwarp();
  }
}

// y (cells of the lines) = the block-tridiagonal solve of x along each line; x, y are [5][N]
__global__ void __launch_bounds__(32 * LW) k_line_apply(Mesh m, Lines L, const double* x, double* y) {
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int line = blockIdx.x * LW + w;
  if (line >= L.nlines) return;
  const int p0 = L.off[line], n = L.off[line + 1] - p0;
  const size_t N = m.ncv;
  const int r = lane % 5;
  const bool row = lane < 5;
  // forward: v_0 = x_0, v_i = x_i - mhat_i v_{i-1}
  double v = x[r * N + L.cv[p0]];
  if (row) L.v[(size_t)p0 * 5 + r] = v;
  for (int i = 1; i < n; i++) {
    const double* Mi = &L.low[(size_t)(p0 + i) * 25 + 5 * r];
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 5; q++) s += Mi[q] * __shfl_sync(0xffffffffu, v, q);
    v = x[r * N + L.cv[p0 + i]] - s;
    if (row) L.v[(size_t)(p0 + i) * 5 + r] = v;
  }
  // backward: y_{n-1} = inv_{n-1} v_{n-1}, y_i = inv_i (v_i - A(c_i, c_{i+1}) y_{i+1})
  const double* I = &L.inv[(size_t)(p0 + n - 1) * 25 + 5 * r];
  double yv = 0.0;
#pragma unroll
  for (int q = 0; q < 5; q++) yv += I[q] * __shfl_sync(0xffffffffu, v, q);
  if (row) y[r * N + L.cv[p0 + n - 1]] = yv;
  for (int i = n - 2; i >= 0; i--) {
    const double* U = &L.up[(size_t)(p0 + i + 1) * 25 + 5 * r];
    double s2 = 0.0;
#pragma unroll
    for (int q = 0; q < 5; q++) s2 += U[q] * __shfl_sync(0xffffffffu, yv, q);
    const double a1 = L.v[(size_t)(p0 + i) * 5 + r] - s2;
    const double* Ii = &L.inv[(size_t)(p0 + i) * 25 + 5 * r];
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 5; q++) s += Ii[q] * __shfl_sync(0xffffffffu, a1, q);
    yv = s;
    if (row) y[r * N + L.cv[p0 + i]] = yv;
  }
}

}  // namespace

void launch_line_factor(const Mesh& m, const State& st, const Lines& L, cudaStream_t s) {
  if (L.nlines) k_line_factor<<<(L.nlines + LW - 1) / LW, 32 * LW, 0, s>>>(m, st, L);
}

void launch_line_precond(const Mesh& m, const State& st, const Lines& L, const double* x, double* y,
                         cudaStream_t s) {
  launch_precond(m, st, x, y, s);  // the block diagonal everywhere, then the lines overwrite their cells
  if (L.nlines) k_line_apply<<<(L.nlines + LW - 1) / LW, 32 * LW, 0, s>>>(m, L, x, y);
}

}  // namespace jg

// ---------------------------------------------------------------------------
// LINE relaxation: block line-Jacobi sweeps for B x B blocks (B = 5, 6, 7) in
// the matrix precision BT.  A sweep is x' = T^-1 (b - (A - T) x), T the
// block-tridiagonal part of A along the lines (the block diagonal elsewhere):
//   k_sweep (LINE): per cell r = b - sum of the off-diagonal blocks that are not
//                 a line coupling times x; off the lines x' = Dinv r, on the
//                 lines r is left in line order for
//   k_lsolve:     the block Thomas substitutions of each line, into x'.
// k_lfactor computes the line factors once per step from D and the ELL
// blocks, in FP64 arithmetic, and stores them in BT.  (The LINE relaxation has
// no reference counterpart; the reference's own line solver, BCGSTAB_LINELET,
// keeps the reference's ludeco/luinv arithmetic in k_line_factor above.)
// ---------------------------------------------------------------------------
namespace jg {
namespace {

template <typename BT, int B>
__device__ double ell_block_b(const Mesh& m, const BT* O, int row, int col, int e) {
  const int s = row / SLICE, lane = row % SLICE;
  double v = 0.0;
  for (int j = m.ell_off[s]; j < m.ell_off[s + 1]; j++)
    if (m.ell_nb[(size_t)j * SLICE + lane] == col) v += (double)O[((size_t)j * B * B + e) * SLICE + lane];
  return v;
}
template <typename BT, int B>
__device__ __forceinline__ double ell_block_bj(const Mesh& m, const BT* O, int row, int col, int j, int e) {
  if (j >= 0) return (double)O[((size_t)j * B * B + e) * SLICE + row % SLICE];
  return j == -1 ? 0.0 : ell_block_b<BT, B>(m, O, row, col, e);
}

// The block Thomas factors along one line per warp: inv_i = (the eliminated diagonal block)^-1,
// low_i = A(c_i, c_i-1) inv_i-1, up_i = A(c_i-1, c_i).  The elimination is serial along the line,
// so each step is kept short: the eliminated block is inverted in place by all lanes together
// (Gauss-Jordan without pivoting, the reference's ludeco/luinv having none either: B pivot
// steps, each one shared-memory read per entry), and the next step's blocks (its coupling
// blocks and diagonal block) are loaded while the current step computes.
template <typename BT, int B>
__global__ void __launch_bounds__(32 * LW) k_lfactor(Mesh m, State st, Lines L) {
  constexpr int BB = B * B, EP = (BB + 31) / 32;  // entries per lane
  __shared__ double sh[LW][4][BB];
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int line = blockIdx.x * LW + w;
  if (line >= L.nlines) return;
  double *b = sh[w][0], *lo = sh[w][1], *up = sh[w][2], *mh = sh[w][3];
  const int p0 = L.off[line], n = L.off[line + 1] - p0;
  const int N = m.ncv;
  const BT* D = (const BT*)st.D;
  const BT* O = (const BT*)st.O;
  BT* Linv = (BT*)L.binv;
  BT* Llow = (BT*)L.blow;
  BT* Lup = (BT*)L.bup;
  for (int e = lane; e < BB; e += 32) b[e] = (double)D[(size_t)e * N + L.cv[p0]];
  // the next step's operands, a step ahead: coupling blocks and diagonal block of position 1
  double nlo[EP], nup[EP], nd[EP];
  auto load_step = [&](int i) {
    const int cp = L.cv[p0 + i - 1], c = L.cv[p0 + i];
    const int jl = L.jlo[p0 + i], ju = L.jup[p0 + i];
#pragma unroll
    for (int t = 0; t < EP; t++) {
      const int e = lane + 32 * t;
      if (e < BB) {
        nlo[t] = ell_block_bj<BT, B>(m, O, c, cp, jl, e);
        nup[t] = ell_block_bj<BT, B>(m, O, cp, c, ju, e);
        nd[t] = (double)D[(size_t)e * N + c];
      }
    }
  };
  if (n > 1) load_step(1);
  __syncwarp();
  for (int i = 1;; i++) {
    // b <- b^-1 in place
#pragma unroll
    for (int k = 0; k < B; k++) {
      const double rp = 1.0 / b[B * k + k];
      double nv[EP];
#pragma unroll
      for (int t = 0; t < EP; t++) {
        const int e = lane + 32 * t, ri = e / B, cj = e % B;
        if (e < BB) {
          if (ri == k) nv[t] = (cj == k) ? rp : b[e] * rp;
          else nv[t] = (cj == k) ? -b[B * ri + k] * rp : b[e] - b[B * ri + k] * (b[B * k + cj] * rp);
        }
      }
      __syncwarp();
#pragma unroll
      for (int t = 0; t < EP; t++)
        if (lane + 32 * t < BB) b[lane + 32 * t] = nv[t];
      __syncwarp();
    }
    for (int e = lane; e < BB; e += 32) Linv[(size_t)(p0 + i - 1) * BB + e] = (BT)b[e];
    if (i == n) break;
    // this step's coupling blocks (loaded a step ahead), the next step's requested now
#pragma unroll
    for (int t = 0; t < EP; t++) {
      const int e = lane + 32 * t;
      if (e < BB) {
        lo[e] = nlo[t];
        up[e] = nup[t];
        Lup[(size_t)(p0 + i) * BB + e] = (BT)nup[t];
      }
    }
    double dc[EP];
#pragma unroll
    for (int t = 0; t < EP; t++) dc[t] = nd[t];
    if (i + 1 < n) load_step(i + 1);
    __syncwarp();
    for (int e = lane; e < BB; e += 32) {
      const int r = e / B, k = e % B;
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < B; q++) s += lo[B * r + q] * b[B * q + k];
      mh[e] = s;
      Llow[(size_t)(p0 + i) * BB + e] = (BT)s;
    }
    __syncwarp();
    double bn[EP];
#pragma unroll
    for (int t = 0; t < EP; t++) {
      const int e = lane + 32 * t;
      bn[t] = 0.0;
      if (e < BB) {
        const int r = e / B, k = e % B;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < B; q++) s += mh[B * r + q] * up[B * q + k];
        bn[t] = dc[t] - s;
      }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < EP; t++)
      if (lane + 32 * t < BB) b[lane + 32 * t] = bn[t];
    __syncwarp();
  }
}

// Bulk copies from global to shared memory (the copy engine, one instruction a run of positions) and
// the barrier a stage of them completes on.  A copy starts and ends on 16-byte boundaries, so one of
// `len` bytes at p takes the aligned bytes around it; shift16(p) is where p then lies.
__device__ __forceinline__ unsigned sh_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned shift16(const void* p) { return (unsigned)((uintptr_t)p & 15); }
__device__ __forceinline__ unsigned bulk_bytes(const void* p, unsigned len) { return (shift16(p) + len + 15) & ~15u; }
__device__ __forceinline__ void bulk_copy(void* dst, const void* p, unsigned len, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   sh_addr(dst)),
               "l"((const char*)p - shift16(p)), "r"(bulk_bytes(p, len)), "r"(sh_addr(bar))
               : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sh_addr(bar)), "r"(bytes) : "memory");
}
// false if the barrier's phase has not completed after `tries` tries
__device__ __forceinline__ bool bar_wait(uint64_t* bar, unsigned parity, int tries) {
  for (int i = 0; i < tries; i++) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(sh_addr(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

constexpr int LG = 8;         // lanes per line
constexpr int LPW = 32 / LG;  // lines per warp

// a stage holds LK positions of each of a warp's lines: two blocks and a vector a position, and room
// for the bytes an unaligned start or end adds
template <typename BT, int B>
struct LineRing {
  static constexpr int LK = 32 / sizeof(BT), LS = 3;
  static constexpr int BLK = LK * B * B * sizeof(BT) + 16, VEC = LK * B * sizeof(BT) + 16;
  static constexpr int LINE = 2 * BLK + VEC;
};

// a row of a block (B elements), in 16- or 8-byte loads where rows are so aligned
template <typename BT, int B>
__device__ __forceinline__ void load_row(BT o[B], const BT* p) {
  if constexpr (B == 6) {
    using V = typename std::conditional<sizeof(BT) == 8, double2, float2>::type;
#pragma unroll
    for (int q = 0; q < B; q += 2) {
      const V v = *reinterpret_cast<const V*>(p + q);
      o[q] = v.x;
      o[q + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < B; q++) o[q] = p[q];
  }
}

// x (cells of a line) = T_line^-1 r, r in line order in L.bv (the pass before left it there).  Four
// lines per warp, eight lanes per line (lanes < B of a group hold the rows of its blocks): the chain
// along a line is serial, so a warp's lines advance together.  The operands of the steps do not
// depend on the chain and lie in line order, so the copy engine brings them LS - 1 stages ahead
// into shared memory and a step's instructions are its row loads, shuffles and multiply-adds: with
// about one warp per scheduler it is the instructions of a step that cost.  2,048 lines of 20 to 80
// cells, register double-buffering before -> now: 6x6 FP64 44 -> 39 us, FP32 36 -> 25; 7x7 FP32 32 -> 21.
// The shuffles run on every lane; a group past the end of its line only skips the update.  A wait
// that runs out (tries) ends the warp's work with the steps of its stage, whose values are then
// undefined: no further copies or steps; the warp waits for the copies it has in flight, within a
// limit, sets flag 8 in err and returns.  (The vote on it stands after a stage's steps: between the
// wait and the steps it costs 2-4% of the kernel.)
template <typename BT, int B>
__global__ void __launch_bounds__(32) k_lsolve(Mesh m, Lines L, BT* __restrict__ x, int* err, int tries) {
  static_assert(B <= LG, "a line's rows fit its lane group");
  using R = LineRing<BT, B>;
  constexpr int BB = B * B, K = R::LK, S = R::LS;
  __shared__ __align__(16) unsigned char ring[S][LPW][R::LINE];
  __shared__ uint64_t bars[S];
  const int lane = threadIdx.x, r = lane % LG, g = lane / LG;
  const int line = blockIdx.x * LPW + g;
  const bool has = line < L.nlines;
  const int p0 = has ? L.off[line] : 0, n = has ? L.off[line + 1] - p0 : 0;
  const bool row = has && r < B;
  const int rr = r < B ? r : 0;  // lanes past the rows mirror row 0 and never store
  if (lane == 0) {
    for (int s = 0; s < S; s++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sh_addr(&bars[s])), "r"(LPW) : "memory");
    asm volatile("fence.proxy.async;" ::: "memory");
  }
  __syncwarp();
  int nmax = n;
  for (int o = LG; o < 32; o *= 2) nmax = max(nmax, __shfl_xor_sync(0xffffffffu, nmax, o));
  const size_t N = m.ncv;
  const BT* Linv = (const BT*)L.binv;
  const BT* Llow = (const BT*)L.blow;
  const BT* Lup = (const BT*)L.bup;
  BT* Lv = (BT*)L.bv;
  const int chunks = (nmax - 1 + K - 1) / K;  // steps 0 .. nmax - 2 of each pass
  // the stages q .. asked - 1 are still in flight: wait for them, report, and the caller returns
  auto give_up = [&](int q, int asked) {
    for (; q < asked; q++) bar_wait(&bars[q % S], (q / S) & 1, WAIT_TRIES);
    if (lane == 0) atomicOr(err, 8);
  };
  // forward: v_0 = r_0, v_i = r_i - low_i v_{i-1}; step j is position j + 1.  Stage q % S holds the
  // q-th chunk asked for, forward chunks first
  auto ask_fwd = [&](int c) {
    if (r != 0 || c >= chunks) return;
    const int i = c * K + 1, cnt = min(K, n - i);
    uint64_t* bar = &bars[c % S];
    if (cnt <= 0) {
      bar_expect(bar, 0);
      return;
    }
    unsigned char* d = ring[c % S][g];
    const BT *lo = Llow + (size_t)(p0 + i) * BB, *rv = Lv + (size_t)(p0 + i) * B;
    const unsigned lb = cnt * BB * sizeof(BT), vb = cnt * B * sizeof(BT);
    bar_expect(bar, bulk_bytes(lo, lb) + bulk_bytes(rv, vb));
    bulk_copy(d, lo, lb, bar);
    bulk_copy(d + 2 * R::BLK, rv, vb, bar);
  };
  for (int c = 0; c < S - 1; c++) ask_fwd(c);
  BT v = has ? Lv[(size_t)p0 * B + rr] : BT(0);
  for (int c = 0; c < chunks; c++) {
    const bool ok = bar_wait(&bars[c % S], (c / S) & 1, tries);
    const int i0 = c * K + 1;
    const unsigned char* d = ring[c % S][g];
    const BT* lo = reinterpret_cast<const BT*>(d + shift16(Llow + (size_t)(p0 + i0) * BB)) + B * rr;
    const BT* rv = reinterpret_cast<const BT*>(d + 2 * R::BLK + shift16(Lv + (size_t)(p0 + i0) * B)) + rr;
    BT* out = Lv + (size_t)(p0 + i0) * B + r;
#pragma unroll
    for (int t = 0; t < K; t++) {
      BT a[B];
      load_row<BT, B>(a, lo + t * BB);
      const BT ri = rv[t * B];
      BT s = 0;
#pragma unroll
      for (int q = 0; q < B; q++) s += a[q] * __shfl_sync(0xffffffffu, v, q, LG);
      if (i0 + t < n) {
        v = ri - s;
        if (row) out[t * B] = v;
      }
    }
    __syncwarp();
    if (!__all_sync(0xffffffffu, ok)) return give_up(c, min(c + S - 1, chunks));
    ask_fwd(c + S - 1);
  }
  // the copy engine reads v back: the stores above first
  asm volatile("fence.proxy.async;" ::: "memory");
  __syncwarp();
  // backward: y_{n-1} = inv_{n-1} v_{n-1}, y_i = inv_i (v_i - up_{i+1} y_{i+1}); step j is position
  // n - 2 - j of each line
  auto ask_bwd = [&](int c) {
    if (r != 0 || c >= chunks) return;
    const int q = chunks + c, hi = n - 2 - c * K, lo = max(0, hi - K + 1), cnt = hi - lo + 1;
    uint64_t* bar = &bars[q % S];
    if (cnt <= 0) {
      bar_expect(bar, 0);
      return;
    }
    unsigned char* d = ring[q % S][g];
    const BT *up = Lup + (size_t)(p0 + lo + 1) * BB, *iv = Linv + (size_t)(p0 + lo) * BB;
    const BT* vv = Lv + (size_t)(p0 + lo) * B;
    const unsigned lb = cnt * BB * sizeof(BT), vb = cnt * B * sizeof(BT);
    bar_expect(bar, bulk_bytes(up, lb) + bulk_bytes(iv, lb) + bulk_bytes(vv, vb));
    bulk_copy(d, up, lb, bar);
    bulk_copy(d + R::BLK, iv, lb, bar);
    bulk_copy(d + 2 * R::BLK, vv, vb, bar);
  };
  for (int c = 0; c < S - 1; c++) ask_bwd(c);
  BT yv = 0;
  {
    BT vq[B];
#pragma unroll
    for (int q = 0; q < B; q++) vq[q] = __shfl_sync(0xffffffffu, v, q, LG);
    if (has) {
      const BT* I = &Linv[(size_t)(p0 + n - 1) * BB + B * rr];
#pragma unroll
      for (int q = 0; q < B; q++) yv += I[q] * vq[q];
      if (row) x[r * N + L.cv[p0 + n - 1]] = yv;
    }
  }
  for (int c = 0; c < chunks; c++) {
    const int q0 = chunks + c, hi = n - 2 - c * K, l0 = max(0, hi - K + 1);
    int cell[K];
#pragma unroll
    for (int t = 0; t < K; t++) cell[t] = hi - t >= 0 ? L.cv[p0 + hi - t] : 0;
    const bool ok = bar_wait(&bars[q0 % S], (q0 / S) & 1, tries);
    const unsigned char* d = ring[q0 % S][g];
    const BT* up = reinterpret_cast<const BT*>(d + shift16(Lup + (size_t)(p0 + l0 + 1) * BB)) + B * rr;
    const BT* iv = reinterpret_cast<const BT*>(d + R::BLK + shift16(Linv + (size_t)(p0 + l0) * BB)) + B * rr;
    const BT* vv = reinterpret_cast<const BT*>(d + 2 * R::BLK + shift16(Lv + (size_t)(p0 + l0) * B)) + rr;
#pragma unroll
    for (int t = 0; t < K; t++) {
      const int i = hi - t, k = max(i - l0, 0);  // past the line's front: any loaded record, unused
      BT a[B], e[B];
      load_row<BT, B>(a, up + k * BB);
      load_row<BT, B>(e, iv + k * BB);
      const BT vi = vv[k * B];
      BT s2 = 0;
#pragma unroll
      for (int q = 0; q < B; q++) s2 += a[q] * __shfl_sync(0xffffffffu, yv, q, LG);
      const BT a1 = vi - s2;
      BT s = 0;
#pragma unroll
      for (int q = 0; q < B; q++) s += e[q] * __shfl_sync(0xffffffffu, a1, q, LG);
      if (i >= 0) {
        yv = s;
        if (row) x[r * N + cell[t]] = yv;
      }
    }
    __syncwarp();
    if (!__all_sync(0xffffffffu, ok)) return give_up(q0, chunks + min(c + S - 1, chunks));
    ask_bwd(c + S - 1);
  }
}

template <typename BT, int B>
void line_relax(const Mesh& m, State& st, const Lines& L, int sweeps, cudaStream_t s, int wait_tries) {
  const int lb = (L.nlines + LW - 1) / LW;
  if (L.nlines) k_lfactor<BT, B><<<lb, 32 * LW, 0, s>>>(m, st, L);
  for (int it = 0; it < sweeps; it++) {
    BT* xin = (BT*)((it % 2 == 0) ? st.x1 : st.x0);
    BT* xout = (BT*)((it % 2 == 0) ? st.x0 : st.x1);
    // two columns at a time: most line cells have three or four couplings off their line.  FP32 resident
    // blocks by measurement (us a pass): 5x5 8 / 9 / 10 8.6 / 8.6 / 7.5 (32 registers, 8 bytes of spills,
    // and one wave of the 49k-cell plate), 6x6 6 / 8 23.2 / 21.1, 7x7 5 / 6 / 7 21.7 / 21.1 / 22.0.  The passes
    // and substitutions are plain launches: as programmatic dependents they measured 4-5% slower
    // (a pass's early blocks take the SMs of the substitutions, which are a chain of latencies)
    constexpr int blocks = sizeof(BT) == 8 ? 1 : B == 5 ? 10 : B == 6 ? 8 : 6;
    k_sweep<BT, B, SWEEP_LINE, 2, blocks><<<m.nslices, B * SLICE, 0, s>>>(
        m, st, xin, xout, it == 0, -1, nullptr, L.line_pos, L.noff, L.off_end, (BT*)L.bv);
    if (L.nlines) k_lsolve<BT, B><<<(L.nlines + LPW - 1) / LPW, 32, 0, s>>>(m, L, xout, st.err, wait_tries);
  }
}

}  // namespace

void launch_line_relax(const Mesh& m, const Params& p, State& st, const Lines& L, int bs, int sweeps,
                       cudaStream_t s, int wait_tries) {
  sweeps = sweeps < 1 ? 1 : sweeps;
  auto run = bs == 5   ? (p.fp32 ? line_relax<float, 5> : line_relax<double, 5>)
             : bs == 6 ? (p.fp32 ? line_relax<float, 6> : line_relax<double, 6>)
                       : (p.fp32 ? line_relax<float, 7> : line_relax<double, 7>);
  run(m, st, L, sweeps, s, wait_tries);
}

}  // namespace jg
