// Direct RHS passes per direction for schemes with compact (tridiagonal) line operators, which the z-marching
// passes do not take: right_hand_side_direct_3d (src/equations/ns_rho_rhou_p.f90:31-253) as a few kernels on the
// line engine (lines.cuh).
//
// One pass per direction d forms the ten quantities of :95-186 that are differentiated along d -- u, v, w, T,
// rho u_d, rho u_d u_v, p, p u_d -- from the state, differentiates them with the whole line resident in the block,
// writes the four gradients and adds the convective terms to five accumulators (14 field accesses in place of 31);
// a pointwise pass turns gradients into stresses, heat fluxes and friction work; one pass per direction adds the
// divergences of three stresses and the heat flux; a pointwise pass finishes the RHS and makes the RK4 stage update.
// The adjoint RHS keeps its sequence of derivatives (rhs_adjoint_generic): the same kind of pass over its seven
// quantities took 1.2 to 2 times as long as they do (5.9 against 4.5 ms an RK4 step on 256 x 128 x 128).
#include <algorithm>
#include <cmath>

#include "cruna_internal.cuh"
#include "lines.cuh"

namespace cruna {

namespace {

constexpr int L = kLineL;

// what the last pass does with the finished RHS (rk_o4_e.f90:45-50, :92-97)
struct Finish {
  int stage;            // 0: write rhs; 1..4: RK4 stage update
  double dt;
  const double *add;    // forcing or null
  double *rhs;
  const double *q0;
  double *acc, *qnext;
  const double *qref;   // type-400 sponge of the direct RHS: rhs -= shape (q - qref); null: none
  SpongeDev sponge;
};

struct DirArgs {
  LineOp op;
  Grid g;
  int dir, G, C;
  double scale, scale_h;       // 1 / (h div) of the flow's and of the heat flux's derivatives
  double WoR, gamma;
  int first;                   // the accumulators are written, not added to
  const double *q;
  double *t;                   // gradients u_d, v_d, w_d, T_d (flux pass)
  const double *s[4];          // stresses tau_1d, tau_2d, tau_3d and the heat flux along d (viscous pass)
  double *r;                   // five accumulators
};

// A quantity to be differentiated: a, a / rho (ir), or a b / rho.
struct Quant {
  const double *a, *b;
  bool ir;
};

// One block's lines: two quantities at a time are differentiated and handed on.
//   pre(p, at): what is read at p before the stores of kSub points' results (a store may alias the next point's read
//               as far as the compiler knows, so reads and stores point by point would expose every latency)
//   post(p, at, pre's value, d0, d1): takes the derivatives at p
template <int R, bool SOLVE, bool X, bool IR>
struct DirBlock {
  static constexpr int kSub = 4;
  const DirArgs &a;
  LineBlock b;
  int base, s, line, nlines, l0, pitch;
  // X: [2][G][pitch] quantities, then [G][pitch] 1 / rho.  Otherwise (IR): 1 / rho of the block's lines with R wrapped
  // rows at both ends, [rows + 2 R][G]
  double *tile;

  __device__ __forceinline__ DirBlock(const DirArgs &a_, double *sm) : a(a_) {
    b = line_block<2>(a.op, sm, a.G, a.C);
    nlines = (int)(a.g.N / a.op.n);
    l0 = blockIdx.x * a.G;
    line = l0 + b.g;
    pitch = a.op.n | 1;
    tile = b.ends + 4 * a.G;
    line_base(a.g, X ? 0 : a.dir, min(line, nlines - 1), base, s);
    if constexpr (IR) {
      if constexpr (X) {
        double *ir = tile + 2 * a.G * pitch;
        each([&](int p, int at) { ir[at] = 1.0 / a.q[p]; });
      } else {
        const int n = a.op.n;
        double rho[L];
#pragma unroll
        for (int j = 0; j < L; ++j) rho[j] = a.q[base + min(b.i0 + j, n - 1) * s];
#pragma unroll
        for (int j = 0; j < L; ++j) {
          const int i = b.i0 + j;
          const double x = 1.0 / rho[j];
          if (i < n) tile[(i + R) * a.G + b.g] = x;
          if (i < R && i < n) tile[(i + R + n) * a.G + b.g] = x;
          if (i < n && i >= n - R) tile[(i + R - n) * a.G + b.g] = x;
        }
      }
    }
    __syncthreads();           // the row table
  }

  template <class F>
  __device__ __forceinline__ void each(F fn) {   // X: the block's points in memory order, their tile places
    const int n = a.op.n;
    const int first = l0 * n, count = min(a.G, nlines - l0) * n;
    int l = threadIdx.x / n, x = threadIdx.x - l * n;
    for (int p = threadIdx.x; p < count; p += blockDim.x) {
      fn(first + p, l * pitch + x);
      x += blockDim.x;
      while (x >= n) {
        x -= n;
        ++l;
      }
    }
  }

  // as each, kSub points at a time: pre(p, at) reads memory for all of them, then post(p, at, pre's value)
  template <class Old, class Pre, class Post>
  __device__ __forceinline__ void each_sub(Pre pre, Post post) {
    const int n = a.op.n;
    const int first = l0 * n, count = min(a.G, nlines - l0) * n;
    int l = threadIdx.x / n, x = threadIdx.x - l * n;
    for (int p0 = threadIdx.x; p0 < count; p0 += kSub * blockDim.x) {
      int at[kSub];
      Old old[kSub];
#pragma unroll
      for (int j = 0; j < kSub; ++j) {
        at[j] = l * pitch + x;
        x += blockDim.x;
        while (x >= n) {
          x -= n;
          ++l;
        }
        const int p = p0 + j * blockDim.x;
        if (p < count) old[j] = pre(first + p, at[j]);
      }
#pragma unroll
      for (int j = 0; j < kSub; ++j) {
        const int p = p0 + j * blockDim.x;
        if (p < count) post(first + p, at[j], old[j]);
      }
    }
  }

  // 1 / rho at the point that pre and post know as `at` (IR)
  __device__ __forceinline__ double inv(int at) const {
    return X ? tile[2 * a.G * pitch + at] : tile[(b.i0 + at + R) * a.G + b.g];
  }

  // quantity c at point p (ir: 1 / rho there)
  __device__ __forceinline__ double value(const Quant &c, int p, double ir) const {
    double v = c.a[p];
    if (c.b) v = v * (c.b[p] * ir);
    else if (c.ir) v = v * ir;
    return v;
  }

  template <class Old, class Pre, class Post>
  __device__ __forceinline__ void run(const Quant &c0, const Quant &c1, double s0, double s1, Pre pre, Post post) {
    const int n = a.op.n;
    double v[2][L];
    if constexpr (X) {
      const double *ir = tile + 2 * a.G * pitch;
      each_sub<double2>(
          [&](int p, int at) {
            const double i = IR ? ir[at] : 0.0;
            return make_double2(value(c0, p, i), value(c1, p, i));
          },
          [&](long long, int at, double2 f) {
            tile[at] = f.x;
            tile[a.G * pitch + at] = f.y;
          });
      __syncthreads();
    }
    // one copy of the window and stencil code for both quantities (their results move by register copies)
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      double w[L + 2 * R], u[L];
      if constexpr (X) {
        const double *row = tile + (k * a.G + b.g) * pitch;
        auto f = [=](int i) { return row[i]; };
        line_window<R>(a.op, b.i0, f, w);
        line_explicit<R, true>(a.op, b.i0, w, f, u);
      } else {
        const Quant c = k == 0 ? c0 : c1;
        const double *rho = a.q;
        int off[L + 2 * R];
#pragma unroll
        for (int m = 0; m < L + 2 * R; ++m) off[m] = base + line_row(a.op, b.i0 - R + m) * s;
#pragma unroll
        for (int m = 0; m < L + 2 * R; ++m) w[m] = c.a[off[m]];
        const double *irt = tile + b.i0 * a.G + b.g;
        if (IR && c.b) {
#pragma unroll
          for (int m = 0; m < L + 2 * R; ++m) w[m] = w[m] * (c.b[off[m]] * irt[m * a.G]);
        } else if (IR && c.ir) {
#pragma unroll
          for (int m = 0; m < L + 2 * R; ++m) w[m] = w[m] * irt[m * a.G];
        }
        const int st = s, b0 = base;
        auto f = [=](int i) {  // closure rows
          const int o = b0 + i * st;
          double x = c.a[o];
          if (c.b) x = x * (c.b[o] / rho[o]);
          else if (c.ir) x = x / rho[o];
          return x;
        };
        line_explicit<R, true>(a.op, b.i0, w, f, u);
      }
      const double sk = k == 0 ? s0 : s1;
#pragma unroll
      for (int j = 0; j < L; ++j) {
        const double x = u[j] * sk;
        if (k == 0) v[0][j] = x;
        else v[1][j] = x;
      }
    }
    if constexpr (SOLVE) line_solve<2>(a.op, b, v);
    else if constexpr (X) __syncthreads();
    if constexpr (X) {
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < L; ++j)
          if (b.i0 + j < n) tile[(k * a.G + b.g) * pitch + b.i0 + j] = v[k][j];
      __syncthreads();
      each_sub<Old>(pre, [&](int p, int at, const Old &old) { post(p, at, old, tile[at], tile[a.G * pitch + at]); });
    } else if (line < nlines) {
#pragma unroll
      for (int j0 = 0; j0 < L; j0 += kSub) {
        Old old[kSub];
#pragma unroll
        for (int j = 0; j < kSub; ++j)
          if (b.i0 + j0 + j < n) old[j] = pre(base + (b.i0 + j0 + j) * s, j0 + j);
#pragma unroll
        for (int j = 0; j < kSub; ++j)
          if (b.i0 + j0 + j < n) post(base + (b.i0 + j0 + j) * s, j0 + j, old[j], v[0][j0 + j], v[1][j0 + j]);
      }
    }
  }
};

// The batches of a pass run as one loop over the same code with run-time operands: written out one after
// another they outgrew the instruction cache (flux pass on 256 x 192 x 128 along y: 1.29 ms, "no instruction"
// the largest stall).
struct FluxBatch {
  Quant c0, c1;
  double s0, s1;                     // scales of the derivatives
  double *o0, *o1;                   // outputs: o = (add ? o : 0) + their derivative
  bool add0, add1;
};

// gradients along d and convective terms of the direct RHS
template <int R, bool SOLVE, bool X>
__global__ void __launch_bounds__(kLineThreads, 2) k_dir_flux(const __grid_constant__ DirArgs a) {
  extern __shared__ double dir_sm[];
  DirBlock<R, SOLVE, X, true> B(a, dir_sm);
  const long long N = a.g.N;
  const int d = a.dir;
  const double *q = a.q, *md = q + (1 + d) * N, *p5 = q + 4 * N;
  double *t = a.t, *r = a.r;
  const bool more = a.first == 0;
  const double s = a.scale, gt = a.gamma / (a.gamma - 1.0);
#pragma unroll 1
  for (int k = 0; k < 5; ++k) {
    FluxBatch f;
    if (k == 0)        // u, v (:95-112)
      f = {{q + N, nullptr, true}, {q + 2 * N, nullptr, true}, s, s, t + (F_UX + d) * N, t + (F_VX + d) * N, false, false};
    else if (k == 1)   // w, T (:95-116, :189-191)
      f = {{q + 3 * N, nullptr, true}, {p5, nullptr, true}, s, a.scale_h * a.WoR, t + (F_WX + d) * N, t + (F_TX + d) * N, false, false};
    else if (k == 2)   // mass and the first momentum flux (:131-149)
      f = {{md, nullptr, false}, {md, q + N, false}, -s, -s, r, r + N, more, more};
    else if (k == 3)   // the other momentum fluxes (:152-177)
      f = {{md, q + 2 * N, false}, {md, q + 3 * N, false}, -s, -s, r + 2 * N, r + 3 * N, more, more};
    else               // pressure gradient and pressure flux (:145-187)
      f = {{p5, nullptr, false}, {p5, md, false}, -s, -gt * s, r + (1 + d) * N, r + 4 * N, true, more};
    B.template run<double3>(
        f.c0, f.c1, f.s0, f.s1,
        [=](int p, int) {
          double3 o = make_double3(0.0, 0.0, 0.0);
          if (f.add0) o.x = f.o0[p];
          if (f.add1) o.y = f.o1[p];
          if (k == 4) o.z = md[p];
          return o;
        },
        [&, f](int p, int at, const double3 &o, double x, double y) {
          f.o0[p] = o.x + x;
          f.o1[p] = o.y + (k == 4 ? y - o.z * B.inv(at) * x : y);   // u_d dp/dx_d with the pressure flux
        });
  }
}

// viscosity, stresses, heat fluxes and friction work (:115-128, :193-206) in place of the gradients
__global__ void __launch_bounds__(256) k_dir_visc(Grid g, const double *__restrict__ q, double *__restrict__ t,
                                                  double *__restrict__ r, double WoR, double mu0, double T0,
                                                  double cp_over_pr) {
  const long long N = g.N;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
    const double T = WoR * q[p + 4 * N] / q[p];
    const double tr = T / T0;
    const double mu = mu0 * (tr * sqrt(tr)) * ((T0 + 110.4) / (T + 110.4));
    const double ux = t[p + F_UX * N], uy = t[p + F_UY * N], uz = t[p + F_UZ * N];
    const double vx = t[p + F_VX * N], vy = t[p + F_VY * N], vz = t[p + F_VZ * N];
    const double wx = t[p + F_WX * N], wy = t[p + F_WY * N], wz = t[p + F_WZ * N];
    const double div = -(2.0 / 3.0 * mu * (ux + vy + wz)), lam = mu * cp_over_pr;
    const double t11 = div + 2 * mu * ux, t22 = div + 2 * mu * vy, t33 = div + 2 * mu * wz;
    const double t12 = mu * (uy + vx), t13 = mu * (uz + wx), t23 = mu * (vz + wy);
    t[p + F_T11 * N] = t11;
    t[p + F_T22 * N] = t22;
    t[p + F_T33 * N] = t33;
    t[p + F_T12 * N] = t12;
    t[p + F_T13 * N] = t13;
    t[p + F_T23 * N] = t23;
    t[p + F_HX * N] = lam * t[p + F_TX * N];
    t[p + F_HY * N] = lam * t[p + F_TY * N];
    t[p + F_HZ * N] = lam * t[p + F_TZ * N];
    r[p + 4 * N] += t11 * ux + t12 * uy + t13 * uz + t12 * vx + t22 * vy + t23 * vz + t13 * wx + t23 * wy + t33 * wz;
  }
}

// divergence of the stresses and of the heat flux along d (:138-177, :195-200)
template <int R, bool SOLVE, bool X>
__global__ void __launch_bounds__(kLineThreads, 2) k_dir_visc_div(const __grid_constant__ DirArgs a) {
  extern __shared__ double dir_sm[];
  DirBlock<R, SOLVE, X, false> B(a, dir_sm);
  const long long N = a.g.N;
  double *__restrict__ r = a.r;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    const double *__restrict__ s0 = a.s[2 * h], *__restrict__ s1 = a.s[2 * h + 1];
    const int v = 1 + 2 * h;
    B.template run<double2>({s0, nullptr, false}, {s1, nullptr, false}, a.scale, h ? a.scale_h : a.scale,
                               [=](int p, int) { return make_double2(r[p + v * N], r[p + (v + 1) * N]); },
                               [&](int p, int, double2 o, double x, double y) {
                                 r[p + v * N] = o.x + x;
                                 r[p + (v + 1) * N] = o.y + y;
                               });
  }
}

// the finished RHS from the accumulators (scale5 on the energy equation), forcing or source, the type-400
// sponge, and the RK4 stage update
__global__ void __launch_bounds__(256) k_dir_finish(const __grid_constant__ Finish f, Grid g, const double *__restrict__ q,
                                                    const double *__restrict__ r, double scale5) {
  const long long N = g.N;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
    double k[5], q0[5], acc[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const long long o = p + v * N;
      k[v] = v == 4 ? scale5 * r[o] : r[o];
      q0[v] = f.stage != 0 ? f.q0[o] : 0.0;
      acc[v] = f.stage >= 2 ? f.acc[o] : 0.0;
      if (f.add) k[v] = k[v] + f.add[o];
    }
    if (f.qref) {
      const double sh = sponge_at(f.sponge, g, p);
      if (sh != 0.0) {
#pragma unroll
        for (int v = 0; v < 5; ++v) k[v] = k[v] - sh * (q[p + v * N] - f.qref[p + v * N]);
      }
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const long long o = p + v * N;
      if (f.stage == 0) f.rhs[o] = k[v];
      else if (f.stage == 4) f.qnext[o] = q0[v] + f.dt / 6.0 * (acc[v] + k[v]);
      else {
        f.acc[o] = f.stage == 1 ? k[v] : acc[v] + 2.0 * k[v];
        f.qnext[o] = q0[v] + (f.stage == 3 ? f.dt : 0.5 * f.dt) * k[v];
      }
    }
  }
}

enum DirPass { PASS_FLUX, PASS_VISC };

template <int R, bool SOLVE, bool X>
void launch_dir(cruna_ctx *c, DirPass pass, DirArgs &a) {
  a.C = line_chunks(a.op.n);
  a.G = line_group(a.C);
  const long long lines = a.g.N / a.op.n;
  // tiles: two quantities (X), 1 / rho
  const size_t rows = X ? (size_t)(a.op.n | 1) : (size_t)a.C * L + 3 * R;
  const size_t tiles = (X ? 2 : 0) + (pass == PASS_VISC ? 0 : 1);
  const size_t sm = sizeof(double) * (line_smem_doubles(a.C, a.G, 2) + tiles * rows * a.G);
  auto go = [&](auto kernel) {
    if (sm > 48 * 1024)
      CRUNA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    kernel<<<(unsigned)((lines + a.G - 1) / a.G), a.C * a.G, sm, c->stream>>>(a);
  };
  if (pass == PASS_FLUX) go(k_dir_flux<R, SOLVE, X>);
  else go(k_dir_visc_div<R, SOLVE, X>);
  CRUNA_LAUNCH_CHECK(c);
}

template <int R, bool SOLVE>
void launch_dir_x(cruna_ctx *c, DirPass pass, DirArgs &a) {
  if (a.dir == 0) launch_dir<R, SOLVE, true>(c, pass, a);
  else launch_dir<R, SOLVE, false>(c, pass, a);
}

// compact schemes (radius 1 or 2) run the radius-2 kernels (coefficients past the radius are skipped), explicit
// ones of radius 4 the radius-4 kernels
void launch_dir_pass(cruna_ctx *c, DirPass pass, DirArgs &a) {
  static const char *names[2][3] = {{"dir_flux_x", "dir_flux_y", "dir_flux_z"},
                                    {"dir_visc_x", "dir_visc_y", "dir_visc_z"}};
  ProfScope ps(c, names[pass][a.dir]);
  if (a.op.solve) launch_dir_x<2, true>(c, pass, a);
  else launch_dir_x<4, false>(c, pass, a);
}

DirArgs dir_args(const cruna_ctx *c, int d) {
  DirArgs a{};
  a.op = c->dop[d];
  a.g = c->g;
  a.dir = d;
  a.scale = 1.0 / (c->dx[d] * a.op.div);
  a.scale_h = 1.0 / ((c->cfg.heat_flux_dx ? c->dx[d] : 1.0) * a.op.div);
  a.WoR = c->cfg.W / c->cfg.R;
  a.gamma = c->cfg.gamma;
  return a;
}

Finish finish_args(const cruna_ctx *c, int stage, double dt, const double *add, double *rhs, const double *q0, double *acc,
                   double *qnext) {
  Finish f{};
  f.stage = stage;
  f.dt = dt;
  f.add = add;
  f.rhs = rhs;
  f.q0 = q0;
  f.acc = acc;
  f.qnext = qnext;
  f.sponge = c->sponge;
  return f;
}

void finish(cruna_ctx *c, const Finish &f, const double *q, const double *r, double scale5) {
  ProfScope ps(c, "dir_finish");
  k_dir_finish<<<(int)std::min<long long>(nblocks(c->g.N), 148LL * 32), kThreads, 0, c->stream>>>(f, c->g, q, r, scale5);
  CRUNA_LAUNCH_CHECK(c);
}

// workspace field of tau_vd
int visc_field(int v, int d) {
  static const int f[3][3] = {{F_T11, F_T12, F_T13}, {F_T12, F_T22, F_T23}, {F_T13, F_T23, F_T33}};
  return f[v][d];
}

}  // namespace

bool only_sponge(const cruna_ctx *c) {   // the RHS boundary table is one type-400 row
  int rows = 0;
  for (const BCRow &r : c->bc) {
    if (r.type == 100 || (r.type >= 204 && r.type <= 206)) return false;
    rows += r.type == 400;
  }
  return rows == 1;
}

// the passes of one direction, for rhs_direct_dir and for the z-marching passes that take their y
// derivatives from here (fused.cu)
void dir_flux(cruna_ctx *c, int d, const double *q, double *t, double *r, bool first) {
  DirArgs a = dir_args(c, d);
  a.q = q;
  a.t = t;
  a.r = r;
  a.first = first;
  launch_dir_pass(c, PASS_FLUX, a);
}

void dir_viscous(cruna_ctx *c, int d, const double *t1, const double *t2, const double *t3, const double *h, double *r) {
  DirArgs a = dir_args(c, d);
  a.s[0] = t1;
  a.s[1] = t2;
  a.s[2] = t3;
  a.s[3] = h;
  a.r = r;
  launch_dir_pass(c, PASS_VISC, a);
}

// The direct RHS on these passes where they are the better path: at least one compact direction (row table) or, on
// grids of 2^20 points or more, none; explicit directions periodic o8.  RK4 steps in ms, passes against the
// sequence of single derivatives (rhs_direct_generic): compact in every direction 128 x 120 x 96 periodic 2.48 / 2.80, 512^2 open
// 0.99 / 1.37; o8 in every direction 256 x 128 x 128 6.40 / 6.83, but 1024 x 64 x 64 7.42 / 6.65 (a block holds few
// long lines) and 32^3 0.74 / 0.67; explicit schemes of radius 1 and 2 run the radius-4 kernels and lose everywhere (open
// o4 160^3 9.09 / 5.77, with a compact y 8.86 / 6.08).
bool dir_passes_supported(const cruna_ctx *c) {
  if (!line_grid_ok(c->g)) return false;
  bool compact = false, o8 = false;
  for (const LineOp &op : c->dop) {
    if (op.kind == OP_ZERO) continue;
    if (op.solve ? !(op.tab && op.r <= 2) : op.r != 4) return false;
    (op.solve ? compact : o8) = true;
  }
  const int longest[3] = {compact ? 512 : 256, compact ? 1024 : 512, compact ? 1024 : 512};
  for (int d = 0; d < 3; ++d)
    if (c->dop[d].kind != OP_ZERO && !c->dop[d].solve && c->dop[d].n > longest[d]) return false;
  return compact || (o8 && c->g.N >= 1LL << 20);
}

// direct RHS (stage 0) or RK stage of the state q_in; bc_mask as rhs_direct_generic
void rhs_direct_dir(cruna_ctx *c, const double *q_in, double *rhs, double *qbc, int bc_mask, int stage, const double *q0,
                    double *acc, double *qnext, double dt) {
  const long long N = c->g.N;
  double *t = c->tmp;
  auto F = [&](int f) { return t + (long long)f * N; };
  double *r = F(F_M1);
  const double *q = q_in;
  if (c->has_q_bc && (bc_mask & 1)) {                     // ns_rho_rhou_p.f90:89-92
    copy_state(c, qbc, q_in, 5);
    bc_q(c, qbc, 0);
    q = qbc;
  }
  bool first = true;
  for (int d = 0; d < 3; ++d) {
    if (c->dop[d].kind == OP_ZERO) {                      // an empty direction's derivatives are zero
      for (int f : {F_UX + d, F_VX + d, F_WX + d, F_TX + d})
        CRUNA_CUDA_CHECK(cudaMemsetAsync(F(f), 0, sizeof(double) * N, c->stream));
      continue;
    }
    dir_flux(c, d, q, t, r, first);
    first = false;
  }
  {
    ProfScope ps(c, "dir_visc");
    k_dir_visc<<<(int)std::min<long long>(nblocks(N), 148LL * 32), kThreads, 0, c->stream>>>(
        c->g, q, t, r, c->cfg.W / c->cfg.R, c->cfg.mu0, c->cfg.T0,
        c->cfg.gamma * (c->cfg.R / c->cfg.W) / (c->cfg.gamma - 1.0) / c->cfg.Pr);
    CRUNA_LAUNCH_CHECK(c);
  }
  for (int d = 0; d < 3; ++d)
    if (c->dop[d].kind != OP_ZERO) dir_viscous(c, d, F(visc_field(0, d)), F(visc_field(1, d)), F(visc_field(2, d)), F(F_HX + d), r);
  const bool bcs = c->has_rhs_bc && (bc_mask & 2);
  const bool split = bcs && !only_sponge(c);              // other RHS boundary types act on the finished RHS
  Finish f = finish_args(c, split ? 0 : stage, dt, c->force, rhs, q0, acc, qnext);
  if (bcs && !split) f.qref = c->qref;
  finish(c, f, q, r, c->cfg.gamma - 1.0);
  if (split) {
    bc_rhs(c, rhs, q);                                    // :218
    if (stage) rk_stage(c, stage, dt, rhs, q0, acc, qnext);
  }
}

}  // namespace cruna
