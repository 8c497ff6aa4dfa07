// Line engine: compact (tridiagonal) line operators with a whole line group resident in one block.
//
// A thread block takes G neighbouring lines of n points; a thread holds kLineL consecutive points of one
// line in registers (thread = chunk * G + line, so the threads of a warp sit on neighbouring lines: along
// y and z their loads are coalesced; along x the block stages its lines through shared memory).  The
// tridiagonal solve runs chunk by chunk in parallel: every thread sweeps its own points with a zero
// incoming value, the chunk ends go through shared memory, and the missing first-order term is added
// with the products of the sweep's multipliers (LU without row interchanges: y_i = v_i - l_i y_{i-1},
// x_i = y_i / u_i - c_i x_{i+1}; a chunk's result depends on its incoming value y through Pf_i y).  The
// incoming value is folded from the last kf chunk ends only: the multipliers decay, and the host picks kf so
// that the part left out is below 1e-20 of a chunk end (all chunks where they do not decay).  A block that meets
// an infinity or NaN folds every chunk, so that it reaches the whole line as in a sequential solve.
#pragma once

#include "ops_common.cuh"

namespace cruna {

// lines of a block for C chunks a line: at most kLineThreads threads (two blocks of 168 registers a thread
// fit an SM); a warp then covers 32 / 16 / 8 / ... neighbouring lines
constexpr int kLineThreads = 192;
inline int line_group(int chunks) {
  int G = 32;
  while (G > 1 && chunks * G > kLineThreads) G >>= 1;
  return G;
}
inline int line_chunks(int n) { return (n + kLineL - 1) / kLineL; }

// shared memory of one block in doubles: row table, carries of NB simultaneous solves, first / last values
inline size_t line_smem_doubles(int C, int G, int NB) {
  return (size_t)6 * kLineL * C + (size_t)2 * NB * C * G + (size_t)2 * NB * G;
}

struct LineBlock {
  const double2 *tab;   // [rows][3]: (l, Pf), (inv, c), (Qb, fb)
  double *fwd, *bwd, *ends;
  int G, C, c, g, i0;   // chunk and line of this thread, first row of its chunk
};

// the block's shared-memory carve-up and the row table staged from global memory (caller synchronises)
template <int NB>
__device__ __forceinline__ LineBlock line_block(const LineOp &op, double *smem, int G, int C) {
  LineBlock b;
  b.G = G;
  b.C = C;
  b.c = threadIdx.x / G;
  b.g = threadIdx.x - b.c * G;
  b.i0 = b.c * kLineL;
  double2 *t = reinterpret_cast<double2 *>(smem);
  if (op.tab) {
    const double2 *src = reinterpret_cast<const double2 *>(op.tab);
    for (int i = threadIdx.x; i < 3 * kLineL * C; i += blockDim.x) t[i] = src[i];
  }
  b.tab = t;
  b.fwd = smem + 6 * kLineL * C;
  b.bwd = b.fwd + NB * C * G;
  b.ends = b.bwd + NB * C * G;
  return b;
}

// barrier; true where any thread's chunk ends x[q] hold an infinity or NaN
template <int NB>
__device__ __forceinline__ bool line_sync_nonfinite(const double (&x)[NB]) {
  bool bad = false;
#pragma unroll
  for (int q = 0; q < NB; ++q) bad = bad || !isfinite(x[q]);
  return __syncthreads_or(bad);
}

// solves B x = v for NB right-hand sides at once; every thread of the block calls it
template <int NB>
__device__ __forceinline__ void line_solve(const LineOp &op, const LineBlock &b, double (&v)[NB][kLineL]) {
  const double2 *t = b.tab + 3 * b.i0;
#pragma unroll
  for (int k = 1; k < kLineL; ++k) {
    const double l = t[3 * k].x;
#pragma unroll
    for (int q = 0; q < NB; ++q) v[q][k] = v[q][k] - l * v[q][k - 1];
  }
  double in[NB];
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    in[q] = v[q][kLineL - 1];
    b.fwd[(q * b.C + b.c) * b.G + b.g] = in[q];
  }
  const int kf = line_sync_nonfinite<NB>(in) ? b.C : op.kf;
#pragma unroll
  for (int q = 0; q < NB; ++q) in[q] = 0.0;
  for (int j = max(0, b.c - kf); j < b.c; ++j) {
    const double pf = b.tab[3 * (j * kLineL + kLineL - 1)].y;
#pragma unroll
    for (int q = 0; q < NB; ++q) in[q] = b.fwd[(q * b.C + j) * b.G + b.g] + pf * in[q];
  }
#pragma unroll
  for (int k = kLineL - 1; k >= 0; --k) {
    const double pf = t[3 * k].y;
    const double2 ic = t[3 * k + 1];
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const double d = (v[q][k] + pf * in[q]) * ic.x;
      v[q][k] = k == kLineL - 1 ? d : d - ic.y * v[q][k + 1 < kLineL ? k + 1 : k];
    }
  }
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    in[q] = v[q][0];
    b.bwd[(q * b.C + b.c) * b.G + b.g] = in[q];
  }
  const int kb = line_sync_nonfinite<NB>(in) ? b.C : op.kb;
#pragma unroll
  for (int q = 0; q < NB; ++q) in[q] = 0.0;
  for (int j = min(b.C - 1, b.c + kb); j > b.c; --j) {
    const double qb = b.tab[3 * (j * kLineL) + 2].x;
#pragma unroll
    for (int q = 0; q < NB; ++q) in[q] = b.bwd[(q * b.C + j) * b.G + b.g] + qb * in[q];
  }
#pragma unroll
  for (int k = 0; k < kLineL; ++k) {
    const double qb = t[3 * k + 2].x;
#pragma unroll
    for (int q = 0; q < NB; ++q) v[q][k] = v[q][k] + qb * in[q];
  }
  if (op.cyclic) {  // Sherman-Morrison from the solution's first and last values
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      if (b.c == 0) b.ends[2 * q * b.G + b.g] = v[q][0];
      if (b.c == b.C - 1) {
#pragma unroll
        for (int k = 0; k < kLineL; ++k)
          if (b.i0 + k == op.n - 1) b.ends[(2 * q + 1) * b.G + b.g] = v[q][k];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NB; ++q) in[q] = b.ends[2 * q * b.G + b.g] + op.fbrat * b.ends[(2 * q + 1) * b.G + b.g];
#pragma unroll
    for (int k = 0; k < kLineL; ++k) {
      const double fb = t[3 * k + 2].y;
#pragma unroll
      for (int q = 0; q < NB; ++q) v[q][k] = v[q][k] - fb * in[q];
    }
  }
}

// closure row i of an open operator from values f(row); antisymmetric rows mirror with a sign
template <class F>
__device__ __forceinline__ double line_end_row(const LineOp &op, int i, F f) {
  const int n = op.n;
  const bool start = i < op.nb;
  const int row = start ? i : n - 1 - i;
  if (op.keep_ends && row == 0) return f(i);
  double t = 0.0;
#pragma unroll 1
  for (int m = 0; m < op.bw; ++m) {
    const int j = start ? m : n - 1 - m;
    t = (m == 0) ? op.brow[row][0] * f(j) : t + op.brow[row][m] * f(j);
  }
  return (op.antisym && !start) ? -t : t;
}

// explicit part of the thread's rows from the window w[m] = f(i0 - R + m) (unscaled); f serves the few
// closure rows of open lines.  R = 0: the values themselves.  Rows past the line's end become zero.
template <int R, bool ANTI, class F>
__device__ __forceinline__ void line_explicit(const LineOp &op, int i0, const double (&w)[kLineL + 2 * R], F f,
                                              double (&v)[kLineL]) {
#pragma unroll
  for (int k = 0; k < kLineL; ++k) {
    if constexpr (R == 0) {
      v[k] = w[k];
    } else if constexpr (ANTI) {
      double t = op.c[1] * (w[k + R + 1] - w[k + R - 1]);
#pragma unroll
      for (int m = 2; m <= R; ++m)
        if (m <= op.r) t = t + op.c[m] * (w[k + R + m] - w[k + R - m]);
      v[k] = t;
    } else {
      double t = op.c[0] * w[k + R];
#pragma unroll
      for (int m = 1; m <= R; ++m) t = t + op.c[m] * (w[k + R + m] + w[k + R - m]);
      v[k] = t;
    }
  }
  if (R > 0 && !op.periodic && (i0 < op.nb || i0 + kLineL > op.n - op.nb)) {
    // one small loop over the chunk's closure rows: the code of the passes has to stay in the instruction cache
#pragma unroll 1
    for (int e = 0; e < 2 * op.nb; ++e) {
      const int i = e < op.nb ? e : op.n - 1 - (e - op.nb);
      if (i < i0 || i >= i0 + kLineL) continue;
      const double t = line_end_row(op, i, f);
#pragma unroll
      for (int k = 0; k < kLineL; ++k)
        if (i0 + k == i) v[k] = t;
    }
  }
  if (i0 + kLineL > op.n) {
#pragma unroll
    for (int k = 0; k < kLineL; ++k)
      if (i0 + k >= op.n) v[k] = 0.0;
  }
}

// row of window entry i = i0 - R + m: wrapped on periodic lines; past the ends of open ones, and past the
// wrapped part, some row of the line whose value no valid row uses (n >= R for every scheme)
__device__ __forceinline__ int line_row(const LineOp &op, int i) {
  const int n = op.n;
  if (op.periodic) i += i < 0 ? n : (i >= n ? -n : 0);
  return min(max(i, 0), n - 1);
}

template <int R, class F>
__device__ __forceinline__ void line_window(const LineOp &op, int i0, F f, double (&w)[kLineL + 2 * R]) {
#pragma unroll
  for (int m = 0; m < kLineL + 2 * R; ++m) w[m] = f(line_row(op, i0 - R + m));
}

// first point and stride of line l along dir (lines numbered with x fastest); 32-bit, so that an address is one
// multiply-add: grids of up to 2^31 - 1 points (line_grid_ok)
__device__ __forceinline__ void line_base(const Grid &g, int dir, int l, int &base, int &s) {
  if (dir == 0) {
    base = l * g.n1;
    s = 1;
  } else if (dir == 1) {
    const int k = l / g.n1;
    base = (l - k * g.n1) + k * (g.n1 * g.n2);
    s = g.n1;
  } else {
    base = l;
    s = g.n1 * g.n2;
  }
}

inline bool line_grid_ok(const Grid &g) { return g.N < (1LL << 31) - 1; }

}  // namespace cruna
