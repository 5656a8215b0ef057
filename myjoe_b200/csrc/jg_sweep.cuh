// jg_sweep.cuh -- one pass of block point relaxation, shared by the 5x5 path, the coupled
// (6x6, 7x7) path and the LINE relaxation's right-hand sides, FP64 or FP32.
//
// A block of B x 32 threads handles one 32-cell slice, warp i the row i of its 32 block rows:
//   acc_i = b_i - sum over the ELL columns of O(i, :) x(neighbour),   x_i = Dinv(i, :) acc.
//
// What bounds a pass: on meshes above L2 the matrix stream (it runs at the copy rate); below, the
// latency of the chain offset -> neighbour id -> x -> barrier, since a 8k-cell colour pass is only
// a block or two per SM.  So
//  * SWEEP_COLS columns are taken at a time: their neighbour ids, then their matrix rows (which no
//    other pass writes) are requested before x is touched;
//  * warp k gathers only component k of x and shares it through shared memory (each component was
//    gathered by all B warps before);
//  * the passes of one solve are programmatic dependents of one another (launch_pass):
//    the next pass's blocks start while this one drains and have everything but x in registers
//    when it ends.  x therefore goes through L2 only (__ldcg): an L1 line read by an earlier pass
//    may not be seen by a later one that started before the boundary.
// Measured, us per solve of 10 sweeps, a kernel taking one column at a time by plain launches -> this one
// (two-layer bumps in colour order): FP64 Jacobi 8k cells 70 -> 29, 50k 84 -> 86, 250k 567 -> 528, 700k
// 1454 -> 1376 (6.3 TB/s of matrix); FP32 Gauss-Seidel, two colours and so 11 passes instead of 20: 8k
// 104 -> 25, 50k 111 -> 45, 250k 467 -> 266, 700k 1239 -> 696.
//
// Every sum keeps its order (k within a column, column by column), so the results are bit for bit
// those of the thread-per-cell kernel (k_jacobi).
#pragma once
#include <cuda_runtime.h>

#include "jg_internal.h"

namespace jg {

constexpr int SWEEP_COLS = 6;  // a hexahedron's row in one chunk

// programmatic dependent launch: wait for the launches this one follows / let the next one start
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// JACOBI: x_out from x_in; GS: in place, the cells of one colour; LINE: x_out from x_in without
// the couplings along the lines, Dinv applied off the lines only
enum { SWEEP_JACOBI = 0, SWEEP_GS = 1, SWEEP_LINE = 2 };

// first: x is zero (the pass is Dinv b).  GS: slices (may be null: every slice) lists the slices
// holding a cell of this colour.  LINE: line_pos the cell's position in the lines (-1:
// on none), where its row goes into line_rhs; off the cell's number of couplings off its line (its
// first columns), off_end per slice one past their last ELL row.
template <typename BT, int B, int KIND, int COLS, int MINB>
__global__ void __launch_bounds__(B * SLICE, MINB) k_sweep(Mesh m, State st, const BT* xin, BT* xout, int first, int color,
                                                     const int* __restrict__ slices,
                                                     const int* __restrict__ line_pos, const int* __restrict__ off,
                                                     const int* __restrict__ off_end, BT* line_rhs) {
  __shared__ BT xs[COLS][B][SLICE];
  __shared__ BT sacc[B][SLICE];
  pdl_trigger();
  const int row = threadIdx.x / SLICE, lane = threadIdx.x % SLICE;
  const int slice = slices ? slices[blockIdx.x] : blockIdx.x;
  const int c = slice * SLICE + lane;
  const int N = m.ncv;
  bool active = c < N;
  if (KIND == SWEEP_GS) active = active && m.color[c] == color;
  if (KIND != SWEEP_LINE) active = active && st.case_active[m.case_of[c]];  // a frozen case does no work
  const int lp = KIND == SWEEP_LINE && active ? line_pos[c] : -1;
  const bool line = KIND == SWEEP_LINE && lp >= 0;
  BT acc = active ? (BT)st.b[(size_t)B * c + row] : (BT)0;
  constexpr bool PRE = COLS > 3;  // Dinv's row in registers before x is there
  BT di[B];
  if (PRE && active && !line) {
    const BT* Di = (const BT*)st.Dinv;
#pragma unroll
    for (int k = 0; k < B; k++) di[k] = Di[(size_t)(B * row + k) * N + c];
  }
  const BT* O = (const BT*)st.O;
  const int j0 = first ? 0 : m.ell_off[slice];
  const int j1 = first ? 0 : KIND == SWEEP_LINE ? off_end[slice] : m.ell_off[slice + 1];
  const int jl = KIND == SWEEP_LINE ? j0 + (active ? off[c] : 0) : j1;  // this cell's last column
  for (int jc = j0; jc < j1; jc += COLS) {
    int nb[COLS];
    BT o[COLS][B];
#pragma unroll
    for (int t = 0; t < COLS; t++) {
      nb[t] = (active && jc + t < jl) ? m.ell_nb[(size_t)(jc + t) * SLICE + lane] : -1;
    }
#pragma unroll
    for (int t = 0; t < COLS; t++)
      if (nb[t] >= 0) {
        const BT* Ob = O + ((size_t)(jc + t) * B * B + B * row) * SLICE + lane;
#pragma unroll
        for (int k = 0; k < B; k++) o[t][k] = Ob[k * SLICE];
      }
    if (jc == j0) pdl_wait();
    else __syncthreads();  // the previous chunk's x is used up
#pragma unroll
    for (int t = 0; t < COLS; t++)
      if (nb[t] >= 0) xs[t][row][lane] = __ldcg(xin + (size_t)row * N + nb[t]);
    __syncthreads();
#pragma unroll
    for (int t = 0; t < COLS; t++)
      if (nb[t] >= 0) {
        BT s = 0;
#pragma unroll
        for (int k = 0; k < B; k++) s += o[t][k] * xs[t][k][lane];
        acc -= s;
      }
  }
  if (j0 == j1) pdl_wait();
  sacc[row][lane] = acc;
  __syncthreads();
  if (active) {
    if (!line) {
      BT s = 0;
#pragma unroll
      for (int k = 0; k < B; k++) s += (PRE ? di[k] : ((const BT*)st.Dinv)[(size_t)(B * row + k) * N + c]) * sacc[k][lane];
      acc = s;
    }
    if (line) line_rhs[(size_t)B * lp + row] = acc;
    else xout[(size_t)row * N + c] = acc;
  }
}

// after_pass: the launch before this one on the stream is a pass of the same solve, so this one may
// start while that one drains (it waits for it before it reads or writes x)
template <typename... P, typename... A>
void launch_pass(void (*kernel)(P...), int grid, int block, bool after_pass, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = after_pass ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// resident blocks of a kernel on the whole GPU
template <typename... P>
int resident_blocks(void (*kernel)(P...), int block) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, block, 0);
  return sms * per;
}

// One pass.  A grid that fits the GPU in one wave takes the widest chunk of columns (the shortest
// dependent chain); a larger FP64 grid lives on resident blocks instead, so it takes three columns
// while those blocks fit one wave and one column with up to 1,920 threads of an SM above.  FP32 rows
// are half as wide in registers and take the whole row at any size, above one wave capped at the
// registers of 960 threads per SM (left to itself the compiler takes 80 a thread).  us per solve of 10
// sweeps, two-layer bumps in colour order (the 8k cells in four layers), 8k / 35k / 50k / 250k / 700k
// cells.  FP64 Jacobi: six columns 29 / 74 / 100 / 633 / 1722, three 41 / 55 / 98 / 545 / 1430, one 49 /
// 78 / 86 / 528 / 1376.  FP32 Gauss-Seidel: six 25 / 37 / 61 / 324 / 873, six capped 29 / 39 / 45 / 266 /
// 696, three 35 / 41 / 51 / 281 / 711, one 57 / 55 / 70 / 297 / 719.
template <typename BT, int B, int KIND>
void launch_sweep(const Mesh& m, const State& st, int grid, const BT* xin, BT* xout, bool first, int color,
                  const int* slices, bool after_pass, cudaStream_t s) {
  constexpr int T = B * SLICE;
  auto wide = k_sweep<BT, B, KIND, SWEEP_COLS, 1>;
  auto packed = k_sweep<BT, B, KIND, SWEEP_COLS, sizeof(BT) == 4 ? 960 / T : 1>;
  auto mid = k_sweep<BT, B, KIND, 3, 1280 / T>;
  auto narrow = k_sweep<BT, B, KIND, 1, 1920 / T>;
  static const int fit_wide = resident_blocks(wide, T), fit_mid = resident_blocks(mid, T);
  auto kernel = grid <= fit_wide ? wide : sizeof(BT) == 4 ? packed : grid <= fit_mid ? mid : narrow;
  if (first) kernel = narrow;  // no matrix rows to request: Dinv b
  launch_pass(kernel, grid, T, after_pass, s, m, st, xin, xout, (int)first, color, slices, nullptr, nullptr, nullptr,
              nullptr);
}

// `sweeps` block Jacobi sweeps from zero: the result is in x0 (odd sweeps) or x1 (even)
template <typename BT, int B>
void sweep_jacobi(const Mesh& m, const State& st, int sweeps, cudaStream_t s) {
  for (int it = 0; it < sweeps; it++) {
    const BT* xin = (const BT*)((it % 2 == 0) ? st.x1 : st.x0);
    BT* xout = (BT*)((it % 2 == 0) ? st.x0 : st.x1);
    launch_sweep<BT, B, SWEEP_JACOBI>(m, st, m.nslices, xin, xout, it == 0, -1, nullptr, it > 0, s);
  }
}

// multicolour Gauss-Seidel from zero, colours forward then backward in turn: the result is in x0.
// A sweep begins with the colour the sweep before it ended with, and nothing else has changed in
// between: that pass would form the same x from the same operands, so it is not launched (with two
// colours 11 passes for 10 sweeps instead of 20).  m.color_proper: no cell is coupled to one of its
// own colour (itself included), the condition for that.
template <typename BT, int B>
void sweep_sgs(const Mesh& m, const State& st, int sweeps, cudaStream_t s) {
  cudaMemsetAsync(st.x0, 0, B * (size_t)m.ncv * sizeof(BT), s);
  int last = -1;
  for (int it = 0; it < sweeps; it++)
    for (int q = 0; q < m.ncolors; q++) {
      const int col = (it % 2 == 0) ? q : m.ncolors - 1 - q;
      if (col == last && m.color_proper) continue;
      const bool lists = m.color_slices != nullptr;
      const int* sl = lists ? m.color_slices + m.color_slice_off[col] : nullptr;
      const int g = lists ? m.color_slice_off[col + 1] - m.color_slice_off[col] : m.nslices;
      if (g == 0) continue;
      launch_sweep<BT, B, SWEEP_GS>(m, st, g, (const BT*)st.x0, (BT*)st.x0, false, col, sl, last >= 0, s);
      last = col;
    }
}

}  // namespace jg
