// jg_bicgstab.cu -- BiCGSTAB with the block-diagonal or the line preconditioner,
// solveCvVectorR5Bcgstab / solveCvVectorR5BcgstabLine (UgpWithCv.cpp:2660-2876, 3627-3992), FP64,
// vectors [5][N].
//
// The scalars of the iteration (rho, alpha, omega, the norms, the stopping rule) live on the
// device: the last block of each reduction finishes it and the step of the recurrence that needs
// it, and every kernel returns at once when the rule has stopped the solve.  The host only
// enqueues, an iteration ahead, and reads the stop flag of the iteration before, so the GPU never
// waits for it: read back one by one the scalars cost six round trips an iteration (49k cells, four
// iterations a step, the call with its state copies: 1,180 -> 612 us a step).
//
// The matrix products take a slice of 32 block rows per block, a warp per row, like the relaxation
// passes (jg_sweep.cuh), the diagonal block's row requested while the vector update before them drains
// and the other blocks' two columns at a time;
// the vector updates form their preconditioned vector in the same pass; the residual's product
// subtracts from the right-hand side and takes the maximum norm on the way.  Reductions keep the
// order of a grid of at most 1,024 blocks with a tree in each and over them.
#include <cuda_runtime.h>
#include <math.h>

#include "jg_internal.h"
#include "jg_sweep.cuh"

namespace jg {

namespace {
constexpr int TB = 128, RT = 256;

// scalars, and after them the words of the running maximum and the block counter
enum { S_RHO, S_ALPHA, S_OMEGA, S_BETA, S_RES0MAX, S_RESMAX, S_DONE, S_ITER, S_MAXBITS, S_COUNT };

// the block sum of v in a fixed tree (RT threads), valid in thread 0
__device__ __forceinline__ double tree_sum(double v, double* s) {
  s[threadIdx.x] = v;
  __syncthreads();
  for (int w = RT / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  const double r = s[0];
  __syncthreads();
  return r;
}

// is this the last block to get here (all threads get the answer); the counter returns to zero
__device__ __forceinline__ bool last_block(double* sc) {
  __shared__ unsigned last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc((unsigned*)&sc[S_COUNT], gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}
}  // namespace

// DOT_RHO: rho = a.b and beta; DOT_ALPHA: gamma = a.b and alpha; DOT_OMEGA: a.b and b.b and omega
enum { DOT_RHO, DOT_ALPHA, DOT_OMEGA };
template <int OP>
__global__ void __launch_bounds__(RT) k_bicg_dot(int n, const double* a, const double* b, double* part, double* sc) {
  __shared__ double s[RT];
  pdl_trigger();
  pdl_wait();
  if (sc[S_DONE] != 0.0) return;
  double v = 0.0, w = 0.0;
  for (long i = blockIdx.x * (long)RT + threadIdx.x; i < n; i += (long)gridDim.x * RT) {
    v += a[i] * b[i];
    if (OP == DOT_OMEGA) w += b[i] * b[i];
  }
  v = tree_sum(v, s);
  if (OP == DOT_OMEGA) w = tree_sum(w, s);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v;
    if (OP == DOT_OMEGA) part[gridDim.x + blockIdx.x] = w;
  }
  if (!last_block(sc)) return;
  v = w = 0.0;
  for (int i = threadIdx.x; i < gridDim.x; i += RT) {
    v += __ldcg(part + i);
    if (OP == DOT_OMEGA) w += __ldcg(part + gridDim.x + i);
  }
  v = tree_sum(v, s);
  if (OP == DOT_OMEGA) w = tree_sum(w, s);
  if (threadIdx.x != 0) return;
  if (OP == DOT_RHO) {
    double rho_prime = -sc[S_OMEGA] * sc[S_RHO];
    if (fabs(rho_prime) < 1.0E-20) rho_prime = 1.0E-20;
    sc[S_RHO] = v;
    sc[S_BETA] = sc[S_ALPHA] * v / rho_prime;
  } else if (OP == DOT_ALPHA) {
    if (fabs(v) < 1.0E-20) v = 1.0E-20;
    sc[S_ALPHA] = sc[S_RHO] / v;
  } else {
    sc[S_OMEGA] = v / (w + 1.0E-20);
  }
}

// a x + b y (+ c z), the vector updates' one expression
__device__ __forceinline__ double lin2(double a, double x, double b, double y) { return a * x + b * y; }

// VEC_P: p = res - beta (p - omega v), y = Dinv p; VEC_S: s = res - alpha v, y = Dinv s;
// VEC_PHI: phi = phi + alpha phat + omega shat.  pre: form y (the block-diagonal preconditioner)
enum { VEC_P, VEC_S, VEC_PHI };
template <int OP>
__global__ void __launch_bounds__(TB) k_bicg_vec(Mesh m, State st, const double* sc, double one, double* out,
                                                 const double* a, const double* b, double* y, int pre) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * TB + threadIdx.x;
  if (c >= m.ncv || sc[S_DONE] != 0.0) return;
  const size_t N = m.ncv;
  const double beta = sc[S_BETA], omega = sc[S_OMEGA], alpha = sc[S_ALPHA];
  double v[5];
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const size_t i = k * N + c;
    if (OP == VEC_P) {         // out p, a res, b v
      v[k] = lin2(one, a[i], -beta, out[i]);
      v[k] += (beta * omega) * b[i];
    } else if (OP == VEC_S) {  // out s, a res, b v
      v[k] = lin2(one, a[i], -alpha, b[i]);
    } else {                   // out phi, a phat, b shat
      v[k] = lin2(one, out[i], alpha, a[i]);
      v[k] += omega * b[i];
    }
    out[i] = v[k];
  }
  if (OP == VEC_PHI || !pre) return;
  const double* Di = (const double*)st.Dinv;
#pragma unroll
  for (int i = 0; i < 5; i++) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 5; k++) s += Di[(size_t)(5 * i + k) * N + c] * v[k];
    y[i * N + c] = s;
  }
}

// y = A x; RES: y = rhs - A x (also into y2 when given), the maximum over the cells of |Dinv y|,
// and the stopping rule (first: the initial residual's norm, no rule)
template <bool RES>
__global__ void __launch_bounds__(5 * SLICE, 8) k_bicg_spmv(Mesh m, State st, const double* x, double* y,
                                                            const double* rhs, double* y2, double* sc,
                                                            int first, double zabs, double zrel, int maxiter,
                                                            volatile unsigned long long* word) {
  constexpr int COLS = 2;
  __shared__ double xs[COLS][5][SLICE];
  __shared__ double wmax[5];
  pdl_trigger();
  const int row = threadIdx.x / SLICE, lane = threadIdx.x % SLICE;
  const int slice = blockIdx.x, c = slice * SLICE + lane;
  const size_t N = m.ncv;
  const bool active = c < m.ncv;
  const double* D = (const double*)st.D;
  const double* O = (const double*)st.O;
  const int j0 = m.ell_off[slice], j1 = m.ell_off[slice + 1];
  double d[5], acc = 0.0;
#pragma unroll
  for (int k = 0; k < 5; k++) d[k] = active ? D[(size_t)(5 * row + k) * N + c] : 0.0;
  pdl_wait();
  if (!first && sc[S_DONE] != 0.0) return;
  xs[0][row][lane] = active ? __ldcg(x + row * N + c) : 0.0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 5; k++) acc += d[k] * xs[0][k][lane];
  for (int jc = j0; jc < j1; jc += COLS) {
    int nb[COLS];
    double o[COLS][5];
#pragma unroll
    for (int t = 0; t < COLS; t++) nb[t] = (active && jc + t < j1) ? m.ell_nb[(size_t)(jc + t) * SLICE + lane] : -1;
#pragma unroll
    for (int t = 0; t < COLS; t++)
      if (nb[t] >= 0)
#pragma unroll
        for (int k = 0; k < 5; k++) o[t][k] = O[((size_t)(jc + t) * 25 + 5 * row + k) * SLICE + lane];
    __syncthreads();
#pragma unroll
    for (int t = 0; t < COLS; t++)
      if (nb[t] >= 0) xs[t][row][lane] = __ldcg(x + row * N + nb[t]);
    __syncthreads();
#pragma unroll
    for (int t = 0; t < COLS; t++)
      if (nb[t] >= 0) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 5; k++) s += o[t][k] * xs[t][k][lane];
        acc += s;
      }
  }
  if (!RES) {
    if (active) y[row * N + c] = acc;
    return;
  }
  acc = active ? rhs[row * N + c] - acc : 0.0;
  if (active) {
    y[row * N + c] = acc;
    if (y2) y2[row * N + c] = acc;
  }
  __syncthreads();
  xs[0][row][lane] = acc;
  __syncthreads();
  double v = 0.0;
  if (active) {
    const double* Di = (const double*)st.Dinv;
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < 5; k++) t += Di[(size_t)(5 * row + k) * N + c] * xs[0][k][lane];
    v = fmax(v, fabs(t));
  }
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) wmax[row] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int r = 1; r < 5; r++) v = fmax(v, wmax[r]);
    // non-negative doubles order as their bit patterns
    atomicMax((unsigned long long*)&sc[S_MAXBITS], (unsigned long long)__double_as_longlong(v));
  }
  if (!last_block(sc) || threadIdx.x != 0) return;
  const double r = __longlong_as_double((long long)atomicExch((unsigned long long*)&sc[S_MAXBITS], 0ull));
  if (first) {
    sc[S_RES0MAX] = r;
    return;
  }
  sc[S_RESMAX] = r;
  const double iter = sc[S_ITER] + 1.0;
  sc[S_ITER] = iter;
  const bool stop = (r <= zabs) || (r / (sc[S_RES0MAX] + 1.0E-12) <= zrel) || iter > maxiter;
  if (stop) sc[S_DONE] = 1.0;
  *word = (unsigned long long)stop << 32 | (unsigned)iter;
  __threadfence_system();
}

__global__ void k_bicg_start(double* sc) {
  for (int i = 0; i < 16; i++) sc[i] = 0.0;
  sc[S_RHO] = sc[S_ALPHA] = sc[S_OMEGA] = 1.0;
}

void launch_bicg_start(const Mesh& m, const State& st, const Bicg& q, cudaStream_t s) {
  k_bicg_start<<<1, 1, 0, s>>>(q.sc);
  k_bicg_spmv<true><<<m.nslices, 5 * SLICE, 0, s>>>(m, st, q.phi, q.res, q.rhs, q.res0, q.sc, 1, 0.0, 0.0, 0, nullptr);
}

// one iteration enqueued
void launch_bicg_iteration(const Mesh& m, const State& st, const Bicg& q, const Lines* lines, cudaStream_t s) {
  const int n5 = 5 * m.ncv, g = grid_for(m.ncv, TB), B = 5 * SLICE, pre = lines == nullptr;
  const int gd = grid_for(n5, RT) < 1024 ? grid_for(n5, RT) : 1024;
  auto spmv = [&](const double* x, double* y, bool after) {
    launch_pass(k_bicg_spmv<false>, m.nslices, B, after, s, m, st, x, y, nullptr, nullptr, q.sc, 0, 0.0, 0.0, 0, nullptr);
  };
  // every kernel waits for the one before it, so each may be launched while that one drains
  launch_pass(k_bicg_dot<DOT_RHO>, gd, RT, true, s, n5, q.res, q.res0, q.part, q.sc);
  launch_pass(k_bicg_vec<VEC_P>, g, TB, true, s, m, st, q.sc, 1.0, q.p, q.res, q.v, q.phat, pre);
  if (lines) launch_line_precond(m, st, *lines, q.p, q.phat, s);
  spmv(q.phat, q.v, pre);
  launch_pass(k_bicg_dot<DOT_ALPHA>, gd, RT, true, s, n5, q.v, q.res0, q.part, q.sc);
  launch_pass(k_bicg_vec<VEC_S>, g, TB, true, s, m, st, q.sc, 1.0, q.s, q.res, q.v, q.shat, pre);
  if (lines) launch_line_precond(m, st, *lines, q.s, q.shat, s);
  spmv(q.shat, q.t, pre);
  launch_pass(k_bicg_dot<DOT_OMEGA>, gd, RT, true, s, n5, q.s, q.t, q.part, q.sc);
  launch_pass(k_bicg_vec<VEC_PHI>, g, TB, true, s, m, st, q.sc, 1.0, q.phi, q.phat, q.shat, nullptr, 0);
  launch_pass(k_bicg_spmv<true>, m.nslices, B, true, s, m, st, q.phi, q.res, q.rhs, nullptr, q.sc, 0, q.zabs, q.zrel,
              q.maxiter, q.word);
}

}  // namespace jg
