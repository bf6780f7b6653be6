// hx_filter.cu -- Helmholtz PDE density filter on the structured node grid.
//
// The reference (src/Optimization/GPUHelmholtz.jl:39-229) assembles
// Ae = r^2 Ke + Me element by element with atomics.  On a full structured
// grid of identical box elements the assembled operator is exactly
//   A = r^2 (Sx(x)My(x)Mz + Mx(x)Sy(x)Mz + Mx(x)My(x)Sz) + Mx(x)My(x)Mz
// with S/M the assembled 1D stiffness/mass (tridiagonal; boundary rows carry
// one element).
// ref_compat=1 reproduces the reference element whose top face is at z=+dz
// (src/Core/Element.jl:106-107), i.e. a box 1.5*dz tall.
//
// Jacobi-CG on it is two kernels per iteration.  The step (k_filter_step) forms
// the new direction while it stages it, advances x with the old one, and applies
// A plane by plane: with the z-direction split off,
//   A = Mz (x) [r^2 (Sx My + Mx Sy) + Mx My] + Sz (x) [r^2 Mx My],
// each plane needs two 9-point sums a, b (26 operations on a shared-memory tile)
// and each node 6 more over three planes.  The Jacobi diagonal takes 27 values (row
// types), so no vector holds it.  The update (k_filter_update) is the rest.  At
// a million nodes the vectors fit the L2 and latency bounds both kernels: an
// iteration at 161 x 81 x 81 nodes took 56 us (plain product from 27 global
// loads per node, then two passes over five vectors) and takes 30 us.
#include "hx_internal.h"

namespace hx {

FilterCoef make_filter_coef(double dx, double dy, double dz, double radius, int ref_compat) {
  FilterCoef F{};
  const double h[3] = {dx, dy, ref_compat ? 1.5 * dz : dz};
  for (int a = 0; a < 3; ++a) {
    const double s = 1.0 / h[a], m = h[a] / 6.0;
    // row type 0: first node (one element on its +side)
    F.S[a][0][0] = 0;  F.S[a][0][1] = s;       F.S[a][0][2] = -s;
    F.M[a][0][0] = 0;  F.M[a][0][1] = 2 * m;   F.M[a][0][2] = m;
    // row type 1: interior
    F.S[a][1][0] = -s; F.S[a][1][1] = 2 * s;   F.S[a][1][2] = -s;
    F.M[a][1][0] = m;  F.M[a][1][1] = 4 * m;   F.M[a][1][2] = m;
    // row type 2: last node
    F.S[a][2][0] = -s; F.S[a][2][1] = s;       F.S[a][2][2] = 0;
    F.M[a][2][0] = m;  F.M[a][2][1] = 2 * m;   F.M[a][2][2] = 0;
  }
  F.r2 = radius * radius;
  for (int x = 0; x < 3; ++x)
    for (int y = 0; y < 3; ++y)
      for (int z = 0; z < 3; ++z) {
        const double sx = F.S[0][x][1], mx = F.M[0][x][1], sy = F.S[1][y][1], my = F.M[1][y][1],
                     sz = F.S[2][z][1], mz = F.M[2][z][1];
        F.inv[x][y][z] =
            1.0 / (F.r2 * (sx * my * mz + mx * sy * mz + mx * my * sz) + mx * my * mz);
      }
  F.vol8 = dx * dy * dz / 8.0;  // the RHS uses the true volume (GPUHelmholtz.jl:175-176)
  return F;
}

namespace {

__device__ __forceinline__ int row_type(int i, int n) {
  return i == 0 ? 0 : (i == n - 1 ? 2 : 1);
}

constexpr int FB_X = 32, FB_Y = 8, FB_NT = FB_X * FB_Y;
constexpr int FS_X = FB_X + 2, FS_Y = FB_Y + 2;  // staged tile with its halo
constexpr int FS_R = 2, FS_NT = FB_NT / FS_R;    // node rows and threads of the step
constexpr int FB_RESIDENT = 4;
constexpr int FB_ROW_RESIDENT = 6;  // CTAs per SM of the row kernels (40 registers)

// One CTA owns a 32 x 8 node column over planes [k0, k1) and marches along z:
// plane kp's new direction p = D^-1 r + beta p_in goes to shared memory (tile
// and halo; the owner also stores it and x + alpha p_in), its sums a, b to
// registers, and q of plane kp - 1 follows from three planes' sums.  r, p_in and
// x are loaded two planes ahead.  A thread has two adjacent rows: they share
// two of their four staged rows' x sums, and the index and bounds arithmetic,
// most of the instructions of a plane (a filter of 30 iterations at 161 x 81 x 81
// nodes 0.985 -> 0.947 ms; one row per thread issued 214 instructions per plane and
// warp, 65% of the issue slots).
__global__ void __launch_bounds__(FS_NT, FB_RESIDENT)
    k_filter_step(const double* __restrict__ pin, double* __restrict__ pout,
                  const double* __restrict__ r, double* __restrict__ x, double* __restrict__ q,
                  Grid g, const __grid_constant__ FilterCoef F, int kchunk, CgState* st,
                  double* partials) {
  pdl_wait();
  pdl_trigger();
  if (st->status != HX_RUNNING) return;
  const bool first = st->iter == 0;  // x = p_in = 0
  const double alpha = first ? 0.0 : st->alpha, beta = first ? 0.0 : st->beta;
  __shared__ double tile[2][FS_Y][FS_X];
  const int tx = threadIdx.x, ty = FS_R * threadIdx.y, tid = tx + FB_X * threadIdx.y;
  const int i = blockIdx.x * FB_X + tx, j = blockIdx.y * FB_Y + ty;
  const int k0 = blockIdx.z * kchunk, k1 = min(k0 + kchunk, g.nzn);
  const bool act[FS_R] = {i < g.nxn && j < g.nyn, i < g.nxn && j + 1 < g.nyn};
  const int64_t pl = (int64_t)g.nxn * g.nyn;
  const int rx = row_type(min(i, g.nxn - 1), g.nxn);
  // Nodes outside the grid are staged as 0, so that only the diagonal entries
  // depend on the row; the off-diagonal ones are m and -s everywhere.
  const double mx1 = F.M[0][rx][1], sx1 = F.S[0][rx][1];
  int ry[FS_R];
  double my1[FS_R], sy1[FS_R];
#pragma unroll
  for (int b = 0; b < FS_R; ++b) {
    ry[b] = row_type(min(j + b, g.nyn - 1), g.nyn);
    my1[b] = F.M[1][ry[b]][1];
    sy1[b] = F.S[1][ry[b]][1];
  }
  // halo node of the staged tile that this thread fills besides its own: two
  // rows of 34, then two columns of 8
  static_assert(2 * FS_X + 2 * FB_Y <= FS_NT, "one halo node per thread");
  const bool halo = tid < 2 * FS_X + 2 * FB_Y;
  int hx, hy;
  if (tid < 2 * FS_X) {
    hx = tid % FS_X;
    hy = tid < FS_X ? 0 : FS_Y - 1;
  } else {
    hx = ((tid - 2 * FS_X) & 1) ? FS_X - 1 : 0;
    hy = 1 + min((tid - 2 * FS_X) >> 1, FB_Y - 1);
  }
  const int hi = blockIdx.x * FB_X - 1 + hx, hj = blockIdx.y * FB_Y - 1 + hy;
  const bool hact = halo && hi >= 0 && hj >= 0 && hi < g.nxn && hj < g.nyn;
  const int hrx = row_type(min(max(hi, 0), g.nxn - 1), g.nxn),
            hry = row_type(min(max(hj, 0), g.nyn - 1), g.nyn);
  const int64_t own = (int64_t)j * g.nxn + i, hown = (int64_t)hj * g.nxn + hi;
  // values of the next plane and of the one after it: one plane's work does not
  // cover the latency of its loads
  struct In {
    double r[FS_R], p[FS_R], x[FS_R], hr, hp;
  };
  auto load = [&](int kp, int64_t o) {
    In v{};
    if (kp < 0 || kp >= g.nzn || kp > k1) return v;
    const double *rp = r + (o + own), *pp = pin + (o + own), *xp = x + (o + own);
    const bool kown = kp >= k0 && kp < k1;
#pragma unroll
    for (int b = 0; b < FS_R; ++b)
      if (act[b]) {
        v.r[b] = rp[b * g.nxn];
        if (!first) {
          v.p[b] = pp[b * g.nxn];
          if (kown) v.x[b] = xp[b * g.nxn];
        }
      }
    if (hact) {
      v.hr = r[o + hown];
      if (!first) v.hp = pin[o + hown];
    }
    return v;
  };
  In n0 = load(k0 - 1, (k0 - 1) * pl), n1 = load(k0, k0 * pl);
  double a0[FS_R] = {}, a1[FS_R] = {}, b0[FS_R] = {}, b1[FS_R] = {};  // planes kp - 2, kp - 1
  double p1[FS_R] = {}, dsum = 0.0;
  const int rz0 = row_type(max(k0 - 1, 0), g.nzn);
  double iv[FS_R], ivh = F.inv[hrx][hry][rz0];  // of plane kp
#pragma unroll
  for (int b = 0; b < FS_R; ++b) iv[b] = F.inv[rx][ry[b]][rz0];
  int64_t o = (k0 - 1) * pl;  // first node of plane kp
  for (int kp = k0 - 1; kp <= k1; ++kp) {
    double(*t)[FS_X] = tile[kp & 1];
    if (kp == 1 || kp == g.nzn - 1) {
      const int rz = row_type(kp, g.nzn);
#pragma unroll
      for (int b = 0; b < FS_R; ++b) iv[b] = F.inv[rx][ry[b]][rz];
      ivh = F.inv[hrx][hry][rz];
    }
    const bool kown = kp >= k0 && kp < k1;
    double *po = pout + (o + own), *xo = x + (o + own);
    double pn[FS_R];
#pragma unroll
    for (int b = 0; b < FS_R; ++b) {
      pn[b] = iv[b] * n0.r[b] + beta * n0.p[b];
      t[ty + b + 1][tx + 1] = pn[b];
      if (act[b] && kown) {
        po[b * g.nxn] = pn[b];
        xo[b * g.nxn] = n0.x[b] + alpha * n0.p[b];
      }
    }
    if (halo) t[hy][hx] = ivh * n0.hr + beta * n0.hp;
    n0 = n1;
    n1 = load(kp + 2, o + 2 * pl);
    __syncthreads();  // plane kp staged (its buffer was last read two planes ago)
    double a2[FS_R] = {}, b2[FS_R] = {};
    if (kp >= 0 && kp < g.nzn) {
      double xm[FS_R + 2], xs[FS_R + 2];
#pragma unroll
      for (int b = 0; b < FS_R + 2; ++b) {
        const double v = t[ty + b][tx + 1], w = t[ty + b][tx] + t[ty + b][tx + 2];
        xm[b] = fma(mx1, v, F.M[0][1][0] * w);
        xs[b] = fma(sx1, v, F.S[0][1][0] * w);
      }
#pragma unroll
      for (int b = 0; b < FS_R; ++b) {
        const double wm = xm[b] + xm[b + 2];
        const double mm = fma(my1[b], xm[b + 1], F.M[1][1][0] * wm),
                     ms = fma(sy1[b], xm[b + 1], F.S[1][1][0] * wm);
        const double sm = fma(my1[b], xs[b + 1], F.M[1][1][0] * (xs[b] + xs[b + 2]));
        a2[b] = fma(F.r2, sm + ms, mm);
        b2[b] = F.r2 * mm;
      }
    }
    if (kp > k0) {
      const int zt = row_type(kp - 1, g.nzn);
      const double mz = F.M[2][zt][1], sz = F.S[2][zt][1];
      double* qo = q + (o - pl + own);
#pragma unroll
      for (int b = 0; b < FS_R; ++b)
        if (act[b]) {
          const double v = fma(mz, a1[b], F.M[2][1][0] * (a0[b] + a2[b])) +
                           fma(sz, b1[b], F.S[2][1][0] * (b0[b] + b2[b]));
          qo[b * g.nxn] = v;
          dsum += p1[b] * v;
        }
    }
#pragma unroll
    for (int b = 0; b < FS_R; ++b) {
      a0[b] = a1[b];
      a1[b] = a2[b];
      b0[b] = b1[b];
      b1[b] = b2[b];
      p1[b] = pn[b];
    }
    o += pl;
  }
  double vv[1] = {dsum};
  if (grid_reduce<1>(vv, partials, &st->ticket[TK_MATVEC]) && tid == 0) {
    const double pq = vv[0];
    st->pq = pq;
    if (!(pq > 0.0) || !isfinite(pq))
      st->status = HX_ST_BREAKDOWN;
    else
      st->alpha = st->rz / pq;
  }
}

// The kernels below take node (element) rows by warp: no division per entry.
// Few long rows are cut into segments of `len` entries (blockIdx.y; see
// row_grid).
__device__ __forceinline__ int seg_begin(int len) { return blockIdx.y * len + threadIdx.x; }
__device__ __forceinline__ int seg_end(int len, int n) { return min((int)(blockIdx.y + 1) * len, n); }

// r -= alpha q, r.D^-1 r and r.r, tests, beta.
__global__ void __launch_bounds__(FB_NT, FB_ROW_RESIDENT)
    k_filter_update(double* __restrict__ r, const double* __restrict__ q, Grid g,
                    const __grid_constant__ FilterCoef F, int len, CgState* st, double* partials) {
  pdl_wait();
  pdl_trigger();
  if (st->status != HX_RUNNING) return;
  const double alpha = st->alpha;
  __shared__ CgState s0;  // read after grid_reduce's barriers
  load_state(&s0, st);
  double rz = 0, rr = 0;
  const int i0 = seg_begin(len), i1 = seg_end(len, g.nxn);
  const unsigned rows = (unsigned)g.nyn * (unsigned)g.nzn;
  for (unsigned row = blockIdx.x * FB_Y + threadIdx.y; row < rows; row += gridDim.x * FB_Y) {
    const int k = row / (unsigned)g.nyn, j = row - k * (unsigned)g.nyn;
    const int ty = row_type(j, g.nyn), tz = row_type(k, g.nzn);
    const double in = F.inv[1][ty][tz], lo = F.inv[0][ty][tz], hi = F.inv[2][ty][tz];
    const int64_t o = (int64_t)row * g.nxn;
#pragma unroll 4
    for (int i = i0; i < i1; i += FB_X) {
      const double ri = r[o + i] - alpha * q[o + i];
      r[o + i] = ri;
      const double d = i == 0 ? lo : (i == g.nxn - 1 ? hi : in);
      rz += ri * (d * ri);
      rr += ri * ri;
    }
  }
  double v[2] = {rz, rr};
  if (grid_reduce<2>(v, partials, &st->ticket[TK_UPDATE]) && threadIdx.x + threadIdx.y == 0)
    cg_finish_iteration(st, s0, v[0], v[1]);
}

// r_n = vol/8 * sum of rho over the (up to 8) elements around node n
// (GPUHelmholtz.jl:39-50 scatters the same sums with atomics), and the CG
// state of x = 0.
__global__ void __launch_bounds__(FB_NT)
    k_filter_init(const double* __restrict__ rho, double* __restrict__ r, Grid g,
                  const __grid_constant__ FilterCoef F, int len, CgState* st, double* partials) {
  double rz = 0, rr = 0;
  const int i0 = seg_begin(len), i1 = seg_end(len, g.nxn);
  const unsigned rows = (unsigned)g.nyn * (unsigned)g.nzn;
  for (unsigned row = blockIdx.x * FB_Y + threadIdx.y; row < rows; row += gridDim.x * FB_Y) {
    const int k = row / (unsigned)g.nyn, j = row - k * (unsigned)g.nyn;
    const int ty = row_type(j, g.nyn), tz = row_type(k, g.nzn);
    for (int i = i0; i < i1; i += FB_X) {
      double s = 0.0;
#pragma unroll
      for (int dk = -1; dk <= 0; ++dk)
#pragma unroll
        for (int dj = -1; dj <= 0; ++dj)
#pragma unroll
          for (int di = -1; di <= 0; ++di) {
            const int ei = i + di, ej = j + dj, ek = k + dk;
            if (ei >= 0 && ej >= 0 && ek >= 0 && ei < g.nxe && ej < g.nye && ek < g.nze)
              s += rho[((int64_t)ek * g.nye + ej) * g.nxe + ei];
          }
      const double ri = s * F.vol8;
      r[(int64_t)row * g.nxn + i] = ri;
      rz += ri * (F.inv[row_type(i, g.nxn)][ty][tz] * ri);
      rr += ri * ri;
    }
  }
  double v[2] = {rz, rr};
  if (grid_reduce<2>(v, partials, &st->ticket[TK_INIT]) && threadIdx.x + threadIdx.y == 0) {
    st->rz = v[0];
    st->rr = v[1];
    st->bnorm = sqrt(v[1]);
    st->iter = 0;
    st->best_rel = INFINITY;
    st->snap = 0;
    st->rel_res = v[1] == 0.0 ? 0.0 : 1.0;
    st->status = v[1] == 0.0 ? HX_ST_ZERO_RHS : (isfinite(v[1]) ? HX_RUNNING : HX_ST_NONFINITE);
  }
}

// element value = mean of its 8 nodal values (GPUHelmholtz.jl:78-89) of x + alpha p,
// of x alone without p
__global__ void __launch_bounds__(FB_NT, FB_ROW_RESIDENT)
    k_filter_extract(const double* __restrict__ x, const double* __restrict__ p, double alpha,
                     double* __restrict__ out, Grid g, int len) {
  const int i0 = seg_begin(len), i1 = seg_end(len, g.nxe);
  const unsigned rows = (unsigned)g.nye * (unsigned)g.nze;
  const int64_t pl = (int64_t)g.nxn * g.nyn;
  for (unsigned row = blockIdx.x * FB_Y + threadIdx.y; row < rows; row += gridDim.x * FB_Y) {
    const int k = row / (unsigned)g.nye, j = row - k * (unsigned)g.nye;
    for (int i = i0; i < i1; i += FB_X) {
      const int64_t n0 = (int64_t)k * pl + (int64_t)j * g.nxn + i;
      auto at = [&](int64_t n) { return p ? x[n] + alpha * p[n] : x[n]; };
      const double s = at(n0) + at(n0 + 1) + at(n0 + g.nxn + 1) + at(n0 + g.nxn) + at(n0 + pl) +
                       at(n0 + pl + 1) + at(n0 + pl + g.nxn + 1) + at(n0 + pl + g.nxn);
      out[(int64_t)row * g.nxe + i] = s / 8.0;
    }
  }
}

// CTAs for `rows` rows of n entries (at most one wave of resident ones), and the
// entries of a segment.  A warp that owns a row takes n / 32 steps; where the rows
// fill less than four CTAs per SM they are cut, down to 128 entries (four loads in
// flight per lane), until they do.  By whole rows a filter (radius 4) took 45 ms on
// 100000 x 1 x 1 elements and 1.5 ms on 2000 x 40 x 2, where most SMs had no row;
// now 1.9 and 0.7 ms.
dim3 row_grid(int64_t rows, int n, int* len) {
  const unsigned bx = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(cdiv(rows, FB_Y), (int64_t)FB_ROW_RESIDENT * sm_count()));
  const int64_t want = std::max<int64_t>(1, 4LL * sm_count() / bx);
  const unsigned seg = (unsigned)std::min<int64_t>(want, cdiv(n, 4 * FB_X));
  *len = (int)cdiv(cdiv(n, seg), FB_X) * FB_X;
  return dim3(bx, cdiv(n, *len));
}

// Planes per CTA of the step: one wave of resident CTAs (two halo planes are
// staged per chunk), but at least 4 planes.
dim3 step_grid(const Grid& g, int* kchunk) {
  const int64_t cols = (int64_t)cdiv(g.nxn, FB_X) * cdiv(g.nyn, FB_Y);
  const int64_t nch = std::max<int64_t>(1, (int64_t)FB_RESIDENT * sm_count() / cols);
  const int kc = std::min(g.nzn, std::max(4, (int)cdiv(g.nzn, nch)));
  *kchunk = kc;
  return dim3(cdiv(g.nxn, FB_X), cdiv(g.nyn, FB_Y), cdiv(g.nzn, kc));
}

}  // namespace

size_t filter_blocks(const Grid& g) {
  int kc, len;
  const dim3 a = step_grid(g, &kc), b = row_grid((int64_t)g.nyn * g.nzn, g.nxn, &len);
  return std::max((size_t)a.x * a.y * a.z, (size_t)b.x * b.y);
}

void launch_filter_init(cudaStream_t s, const double* rho, double* r, const Grid& g,
                        const FilterCoef& F, CgState* st, double* partials) {
  int len;
  const dim3 grid = row_grid((int64_t)g.nyn * g.nzn, g.nxn, &len);
  k_filter_init<<<grid, dim3(FB_X, FB_Y), 0, s>>>(rho, r, g, F, len, st, partials);
  HX_CHECK_LAUNCH();
}

void launch_filter_step(cudaStream_t s, const double* pin, double* pout, const double* r,
                        double* x, double* q, const Grid& g, const FilterCoef& F, CgState* st,
                        double* partials) {
  int kc;
  const dim3 grid = step_grid(g, &kc);
  launch_dep(one_wave((int64_t)grid.x * grid.y * grid.z, FB_RESIDENT), k_filter_step, grid,
             dim3(FB_X, FB_Y / FS_R), 0, s, pin, pout, r, x, q, g, F, kc, st, partials);
  HX_CHECK_LAUNCH();
}

void launch_filter_update(cudaStream_t s, double* r, const double* q, const Grid& g,
                          const FilterCoef& F, CgState* st, double* partials) {
  int len;
  const dim3 grid = row_grid((int64_t)g.nyn * g.nzn, g.nxn, &len);
  launch_dep(one_wave((int64_t)grid.x * grid.y, FB_ROW_RESIDENT), k_filter_update, grid, dim3(FB_X, FB_Y), 0, s,
             r, q, g, F, len, st, partials);
  HX_CHECK_LAUNCH();
}

void launch_filter_extract(cudaStream_t s, const double* x, const double* p, double alpha,
                           double* out, const Grid& g) {
  int len;
  const dim3 grid = row_grid((int64_t)g.nye * g.nze, g.nxe, &len);
  k_filter_extract<<<grid, dim3(FB_X, FB_Y), 0, s>>>(x, p, alpha, out, g, len);
  HX_CHECK_LAUNCH();
}

}  // namespace hx
