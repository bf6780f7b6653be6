// hx_operator.cu -- structured-grid Hex8 stiffness operator K(f) x, alone or
// fused with the CG direction/solution updates.
//
// Layout in HBM: node n = i + NXn*(j + NYn*k) (i fastest, src/Mesh/Mesh.jl:
// 13-15), vectors interleaved 3 per node (dof = 3n + c), element
// e = i + NXe*(j + NYe*k) (the element loop of Mesh.jl:44-55), one factor
// per element, one byte of free-DOF bits per node.
//
// Kernel design (replaces the one-thread-per-element, 24-atomics kernel of
// src/Solvers/GPUSolver.jl:37-79 and the broadcast kernels around it):
//  * a CTA of w warps owns a 31 x (w R - 1) column of output nodes and marches
//    along z over a chunk of node planes; each thread owns R element columns
//    adjacent in y, the one-element halo in x and y is recomputed (atomic-free
//    and deterministic).  FP32: R = 2, and the two elements are the two halves
//    of packed FP32 operations; FP64: R = 1 (see Tile);
//  * node planes (tile + one-node halo) are staged into shared memory with
//    16-byte cp.async, several planes ahead (see Stage, Smem);
//  * the element product runs in the per-axis sum/difference (Haar) basis,
//    where Ke is eight 3 x 3 blocks (lambda_pair); a plane's face
//    coefficients are formed once and carried to the layer above, and so are
//    a layer's top-face outputs;
//  * the element columns around a node are summed in the thread (the two
//    elements of a pair), with one warp shuffle (x) and one shared-memory
//    exchange with the next warp (y).  That exchange is read after the next
//    plane's barrier, so a plane costs one barrier: the node plane ke is
//    finished while element layer ke + 1 is computed;
//  * FUSED (the PCG step): the staged planes hold p_old, r, M^-1 and x (the
//    FCG step: p_old, z and x).  Each thread forms p = M^-1 r + beta p_old
//    (p = z + beta p_old) on the chunks that it copied itself, stores it to
//    a small ring that the element products read and, for owned nodes,
//    to p, and updates x += alpha_old p_old.  p ping-pongs between two
//    buffers so neighbouring CTAs never read a value another CTA rewrote.
//    The epilogue adds the shift and reduces p.q deterministically into the
//    CG state (alpha = rz / pq); q stays unmasked on the fixed DOFs, where p is
//    0 and the residual update does not read it.
// What bounds it: instruction issue and the latency between dependent
// instructions (12 warps per SM, 50-62% of the issue slots used), not memory
// (the FP32 flexible-CG step moves 0.64 GB at 3.8 TB/s, the FP64 PCG step 1.47
// GB at 4.6 TB/s).  A warp issues about 520 instructions per plane and pair of
// element rows in FP32 and 370 per row in FP64.
// Measured at 320 x 160 x 160 (B200), before (one element column per thread in
// both precisions, 45-term product, two barriers per plane) and now: FP64 PCG
// step 402 -> 319 us, FP64 K x 260 -> 205 us, FP32 PCG step 220 -> 182 us, FP32
// flexible-CG step 207 -> 170 us; FP32 Chebyshev step and residual at 192 x 96
// x 96: 55 -> 36 and 50 -> 36 us.  Boxes (sides 1 : 0.8 : 1.25), whose coefficients
// come from the kernel's arguments, in the same order: 402 -> 328, 259 -> 209, 220 ->
// 182, 208 -> 170 us, and a V-cycle 1607 -> 1003 us (cubes 983).
// Measured and dropped (FP32 flexible-CG step, 320 x 160 x 160): one element
// row per thread at 24 warps per SM 188 us; 8 warps x 2 CTAs (128 registers,
// spills) 189-204 us; 12 x 1 201 us; 6 x 2 178 us; the plane loop unrolled
// twice 179-208 us; positions advanced per plane instead of recomputed 176-182
// us.
#include <type_traits>
#include <utility>

#include "hx_internal.h"

namespace hx {

namespace {

constexpr int MV_BX = 32;  // lanes = element columns in x

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// 16-byte asynchronous copy global -> shared; only the first `bytes`
// (0..16) are read, the rest of the 16 are zero-filled.
__device__ __forceinline__ void cp_async16(unsigned sdst, const void* gsrc, unsigned bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sdst), "l"(gsrc),
               "r"(bytes));
}
__device__ __forceinline__ void cp_async16(unsigned sdst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sdst), "l"(gsrc));
}
__device__ __forceinline__ void cp_async8(unsigned sdst, const void* gsrc, unsigned bytes = 8) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sdst), "l"(gsrc),
               "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Elements per thread (R), the type that holds one value of each, warps per
// CTA and CTAs per SM.  The forms want about 160 registers a thread (the face
// coefficients of two planes, the carried outputs and the block in work), so
// 12 warps fit an SM; small CTAs wait less at the barrier of a plane, large
// ones recompute less halo.  FP64 K x fits 128 registers (16 warps: 205 us at
// 320 x 160 x 160 against 219 us in the fused form's shape; the fused form in
// that shape spills: 406 against 319 us).
template <typename T, bool FUSED>
struct Tile;
template <bool FUSED>
struct Tile<float, FUSED> {
  static constexpr int R = 2, WARPS = 4, RESIDENT = 3;
  using V = float2;
};
template <bool FUSED>
struct Tile<double, FUSED> {
  static constexpr int R = 1, WARPS = FUSED ? 6 : 8, RESIDENT = 2;
  using V = double;
};
template <typename T>
using VecOf = typename Tile<T, false>::V;
template <typename T, bool FUSED>
constexpr int mv_by() { return Tile<T, FUSED>::WARPS * Tile<T, FUSED>::R; }  // element rows of a CTA
constexpr bool mode_fused(int mode) { return mode == 3 || mode == 4 || mode == 7; }

__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ double vneg(double a) { return -a; }
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }
template <typename V>
__device__ __forceinline__ V vzero();
template <>
__device__ __forceinline__ double vzero<double>() { return 0.0; }
template <>
__device__ __forceinline__ float2 vzero<float2>() { return make_float2(0.f, 0.f); }
template <typename V>
__device__ __forceinline__ V vone();
template <>
__device__ __forceinline__ double vone<double>() { return 1.0; }
template <>
__device__ __forceinline__ float2 vone<float2>() { return make_float2(1.f, 1.f); }

// a - b as fma(b, m, a) with m = (-1, -1) held in registers
__device__ __forceinline__ float2 vsubm(float2 a, float2 b, float2 m) { return __ffma2_rn(b, m, a); }
__device__ __forceinline__ double vsubm(double a, double b, double) { return a - b; }
// Element coefficients, one per element of the thread (both halves equal):
// the Haar-domain operator of a box element, or (CUBE) the five numbers that
// are left of it for equal sides (see lambda_pair).
template <typename V, bool CUBE>
struct CoefV {
  V dg[3][8], lam[3][2], mu[3][2];
};
template <typename V>
struct CoefV<V, true> {
  V unit, rho, rho3, rho49, third;
};
__host__ inline void put(double& d, double v) { d = v; }
__host__ inline void put(float2& d, double v) { d = make_float2((float)v, (float)v); }
template <typename T, typename V>
void coef_v(const ElemCoef<T>& k, CoefV<V, false>& o) {
  for (int c = 0; c < 3; ++c) {
    for (int s = 0; s < 8; ++s) put(o.dg[c][s], (double)k.dg[c][s]);
    for (int s = 0; s < 2; ++s) {
      put(o.lam[c][s], (double)k.lam[c][s]);
      put(o.mu[c][s], (double)k.mu[c][s]);
    }
  }
}
template <typename T, typename V>
void coef_v(const ElemCoef<T>& k, CoefV<V, true>& o) {
  put(o.unit, (double)k.mu[0][0]);
  put(o.rho, k.rho);
  put(o.rho3, k.rho / 3.0);
  put(o.rho49, (k.rho + 4.0) / 9.0);
  put(o.third, 1.0 / 3.0);
}
// Loop constants that stay in vector registers: read back from shared memory,
// so that the compiler takes them for data.  Straight from the kernel's
// arguments it keeps them in uniform registers, which packed operations cannot
// read: every use then costs moves.  CUBE only (the general coefficients are
// too many for registers).
template <typename V>
__device__ __forceinline__ V from_shared(const volatile V* p);
template <>
__device__ __forceinline__ double from_shared<double>(const volatile double* p) { return *p; }
template <>
__device__ __forceinline__ float2 from_shared<float2>(const volatile float2* p) {
  return make_float2(p->x, p->y);
}
template <typename V>
__device__ __forceinline__ void pin_coef(CoefV<V, true>& k, const volatile V* sh) {
  k.rho = from_shared(sh);
  k.rho3 = from_shared(sh + 1);
  k.rho49 = from_shared(sh + 2);
  k.third = from_shared(sh + 3);
}
template <typename V>
__device__ __forceinline__ void pin_coef(CoefV<V, false>&, const volatile V*) {}
template <typename V>
__device__ __forceinline__ void share_coef(const CoefV<V, true>& k, V* sh) {
  sh[0] = k.rho;
  sh[1] = k.rho3;
  sh[2] = k.rho49;
  sh[3] = k.third;
}
template <typename V>
__device__ __forceinline__ void share_coef(const CoefV<V, false>&, V*) {}
template <typename V>
__device__ __forceinline__ V unit_of(const CoefV<V, true>& k) { return k.unit; }
template <typename V>
__device__ __forceinline__ V unit_of(const CoefV<V, false>&) { return vzero<V>(); }

// Staging geometry.  A staged row is the 33 nodes i0-1 .. i0+31 of one
// node row, 99 contiguous values of an interleaved vector.  It is copied in
// 16-byte chunks (W values) starting at the 16-byte boundary at or below its
// first value, so a row takes CPR chunks and sits in shared memory with a
// lead of (first value's index) mod W values, which depends on the row and
// the plane.  Lanes then read node a, component c of row b at
// b*RS + lead_b + 3a + c: a stride of 3 words (FP32) or 3 doublewords
// (FP64) across a warp, free of bank conflicts.
template <typename T, bool FUSED>
struct Stage {
  static constexpr int W = 16 / (int)sizeof(T);           // values per chunk
  static constexpr int ROWV = 3 * (MV_BX + 1);            // 99 values per row
  static constexpr int CPR = (ROWV + W - 1 + W - 1) / W;  // chunks per row
  static constexpr int RS = CPR * W;                      // row stride (values)
  static constexpr int ROWS = mv_by<T, FUSED>() + 1;
  static constexpr int PLANE = ROWS * RS;                 // values
  static_assert(RS >= ROWV + W - 1, "a row with any lead fits its staged chunks");
  static_assert((PLANE * sizeof(T)) % 16 == 0, "planes keep 16-byte chunk alignment");
};

// Rings of staged planes, by MODE (see k_struct).  FUSED: NS planes of each
// input in flight (a thread transforms the chunks that it copied itself, so
// a slot is free again at once), two or three planes of the new p.  Others: NX planes
// of x, of which NX - 2 are in flight, and NA planes of each of the AUX
// vectors that the epilogue reads.
template <typename T, int MODE>
struct Smem {
  static constexpr bool FUSED = mode_fused(MODE);
  static constexpr int PLANE = Stage<T, FUSED>::PLANE, WARPS = Tile<T, FUSED>::WARPS;
  static constexpr int IN = MODE == 3 ? 4 : 3;  // FUSED: staged inputs
  static constexpr int NS = 3;
  static constexpr int AUX = MODE == 5 ? 3 : (MODE == 6 ? 1 : 0);
  static constexpr int NX = FUSED ? (sizeof(T) == 4 ? 3 : 2) : (AUX ? 4 : 6);
  static constexpr bool KEEP = NX == 2;  // plane ke is gone when its sums are ready
  static constexpr int NA = AUX ? 3 : 0;
  T p[NX][PLANE];
  T in[FUSED ? NS : (AUX ? NA : 1)][FUSED ? IN : (AUX ? AUX : 1)][(FUSED || AUX) ? PLANE : 16 / (int)sizeof(T)];
  T red[2][WARPS][3][MV_BX];  // y-direction partials, of two planes
  VecOf<T> k[6];  // loop constants (see from_shared)
};

template <typename T, bool CUBE>
struct OpArgs {
  const T* pin;   // vector to multiply (MODE 0, 1, 5, 6) or p_old (FUSED)
  const T* r;     // MODE 3: residual; MODE 5, 6: right-hand side b
  const T* minv;  // MODE 3, 5: Jacobi inverse diagonal; MODE 4: preconditioned z
  const float* z32;  // MODE 7: preconditioned z
  T* x;           // FUSED: solution (x += alpha_old p_old on owned nodes); MODE 5:
                  // x_prev in, x_new out
  T* pout;        // FUSED: new direction p
  T* xbest;       // FUSED, FP64: receives x too when the state asks for a snapshot (or null)
  T* q;           // output K x + s x, masked; FUSED: not masked (0 for p, not for q, on
                  // the fixed DOFs); MODE 6: the residual
  const T* fac;
  const uint8_t* nmask;
  Grid g;
  int kchunk;
  int yx;  // 1: blockIdx.x counts the columns in y (see mv_grid)
  CoefV<VecOf<T>, CUBE> K;
  T shift;
  T omega, gamma;  // MODE 5: recurrence coefficients
  int xprev_zero;  // MODE 5: x_prev = 0 (not read)
  CgState* st;
  double* partials;
  double* out;
};

// Lambda in the Haar domain.  Its coefficients couple only where t = sigma xor
// e_c agrees (e_c: the bit of the component's own axis): eight blocks of one
// coefficient per component, through lambda where neither of the two
// components' bits is set in t, through mu where both are.  Blocks Q and Q + 4
// together take the z-sums s and z-differences d of the face coefficients
// (x, Q ^ 1), (y, Q ^ 2) and (z, Q), and give the outputs of the same three,
// so a layer's product needs few values at a time.  The z-sum of coefficient
// 0 is a rigid translation: it is not read and its output is 0.
template <int Q, typename V>
__device__ __forceinline__ void lambda_pair(const CoefV<V, false>& K, V (&s)[3], V (&d)[3]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int t = Q + 4 * h;
    // block t: x and y from s (h = 0) or d, z from d (h = 0) or s
    V u[3] = {h ? d[0] : s[0], h ? d[1] : s[1], h ? s[2] : d[2]}, y[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int sg = t ^ (1 << c);
      if (!sg) {
        y[c] = vzero<V>();
        continue;
      }
      y[c] = vmul(K.dg[c][sg], u[c]);
#pragma unroll
      for (int e = 1; e <= 2; ++e) {
        const int o = (c + e) % 3, k = 3 - c - o;
        const int bc = (t >> c) & 1, bo = (t >> o) & 1, bk = (t >> k) & 1;
        if (bc != bo || !(t ^ (1 << o))) continue;
        y[c] = vfma(bc ? K.mu[k][bk] : K.lam[k][bk], u[o], y[c]);
      }
    }
    (h ? d[0] : s[0]) = y[0];
    (h ? d[1] : s[1]) = y[1];
    (h ? s[2] : d[2]) = y[2];
  }
}
// Equal sides h, in units of mu h / 16 (folded into the element factor), with
// rho = lambda / mu: normal strains (t = 0) 2 u_c + rho (u_x + u_y + u_z);
// t one bit: u_i + rho/3 (u_i + u_j) for the other two components; t two bits:
// u_i + u_j for both of them, (rho + 4)/9 u for the third; t = 7: (u_c + sum)/3.
// 27 operations instead of 45, and no coefficient per entry to load.
template <int Q, typename V>
__device__ __forceinline__ void lambda_pair(const CoefV<V, true>& K, V (&s)[3], V (&d)[3]) {
  auto bit1 = [&](V& a, V& b) {
    const V t = vadd(a, b);
    a = vfma(K.rho3, t, a);
    b = vfma(K.rho3, t, b);
  };
  if constexpr (Q == 0) {
    const V t = vmul(K.rho, vadd(vadd(s[0], s[1]), d[2]));
    s[0] = vadd(vadd(s[0], s[0]), t);
    s[1] = vadd(vadd(s[1], s[1]), t);
    d[2] = vadd(vadd(d[2], d[2]), t);
    bit1(d[0], d[1]);
    s[2] = vzero<V>();
  } else if constexpr (Q == 1) {
    bit1(s[1], d[2]);
    s[0] = vzero<V>();
    d[0] = s[2] = vadd(d[0], s[2]);
    d[1] = vmul(K.rho49, d[1]);
  } else if constexpr (Q == 2) {
    bit1(s[0], d[2]);
    s[1] = vzero<V>();
    d[1] = s[2] = vadd(d[1], s[2]);
    d[0] = vmul(K.rho49, d[0]);
  } else {
    s[0] = s[1] = vadd(s[0], s[1]);
    d[2] = vmul(K.rho49, d[2]);
    const V t = vmul(K.third, vadd(vadd(d[0], d[1]), s[2]));
    d[0] = vfma(K.third, d[0], t);
    d[1] = vfma(K.third, d[1], t);
    s[2] = vfma(K.third, s[2], t);
  }
}

// MODE 0: q = mask(K x + s x);  MODE 1: also out[0] = x.q;
// MODE 3: fused PCG step (see file header): st->pq = p.q, st->alpha = rz / pq,
//         breakdown test;
// MODE 4: flexible-CG step: p = z + beta p_old (z from a variable
//         preconditioner), x += alpha_old p_old, q = K p; alpha = z.r / p.q
//         with z.r from the preconditioner's output pass (st->aux[3]); p.r
//         = z.r + beta p_old.r and the previous step length makes p_old.r
//         vanish, so r is not staged;
// MODE 5: Chebyshev step of the multigrid smoother as a three-term
//         recurrence on x: x_new = x + omega (x - x_prev) + gamma M^-1 (b - A x)
//         with A x = mask(K x + s x); x_prev (A.x) is overwritten by x_new
//         (each node's x_prev is read and written by its owner only; the
//         staged x, read by the neighbours, is not written);
// MODE 6: residual r = mask(b - K x - s x) into A.q;
// MODE 7: MODE 4 of an FP64 solve with z in FP32, as the multigrid cycle leaves
//         it (two z's fill the first half of a 16-byte slot of their plane).
//         With an FP64 copy of z, the copy took 48 us at 320 x 160 x 160, the
//         coefficients 93 (now 81) and this step 307 (now 296).
template <typename T, int MODE, bool CUBE>
__global__ void __launch_bounds__(MV_BX* Tile<T, mode_fused(MODE)>::WARPS,
                                  Tile<T, mode_fused(MODE)>::RESIDENT)
    k_struct(const __grid_constant__ OpArgs<T, CUBE> A) {
  using S = Smem<T, MODE>;
  using G = Stage<T, S::FUSED>;
  using V = VecOf<T>;
  constexpr bool FUSED = S::FUSED;
  constexpr bool DOT = MODE == 1 || FUSED;  // reduces x.q / p.q
  constexpr bool FCG = MODE == 4 || MODE == 7;
  static_assert(MODE != 7 || sizeof(T) == 8, "an FP64 step");
  constexpr int R = Tile<T, FUSED>::R, WARPS = S::WARPS, BY = WARPS * R;
  constexpr int NT = MV_BX * WARPS;
  constexpr int W = G::W, CPR = G::CPR, RS = G::RS, PLANE = G::PLANE;
  // Chunks of a staged plane by thread: FP32 in runs of 32 chunks of a row, run
  // wy, wy + WARPS, ... by warp wy (a row is one run of 26); FP64, whose rows are
  // 50 chunks, one after the other.
  constexpr bool RUNS = CPR <= 32;
  constexpr int NCT = RUNS ? (G::ROWS + WARPS - 1) / WARPS : (G::ROWS * CPR + NT - 1) / NT;
  using VecT = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  extern __shared__ __align__(16) unsigned char smraw[];
  S& sm = *reinterpret_cast<S*>(smraw);
  const Grid& g = A.g;
  const int lx = threadIdx.x, wy = threadIdx.y;
  const int tid = lx + MV_BX * wy;
  const int i0 = (A.yx ? blockIdx.y : blockIdx.x) * (MV_BX - 1);
  const int j0 = (A.yx ? blockIdx.x : blockIdx.y) * (BY - 1);
  const int k0 = blockIdx.z * A.kchunk;
  const int k1 = min(k0 + A.kchunk, g.nzn);
  const int in = i0 - 1 + lx, jn = j0 - 1 + R * wy;  // first element column, first node
  const int nplane = g.nxn * g.nyn;
  const int P3 = 3 * nplane;  // values per node plane (32-bit: the grid extent check bounds it)
  const int kp_last = min(k1, g.nzn - 1);  // last plane staged
  // Rows and nodes outside the grid are never copied: they have to be finite,
  // and are 0.  CTAs inside the grid read only what they copied.
  if (i0 + MV_BX >= g.nxn || j0 == 0 || j0 - 1 + BY >= g.nyn)
    for (int i = tid; i < (int)(sizeof(S) / 16); i += NT)
      reinterpret_cast<uint4*>(smraw)[i] = make_uint4(0u, 0u, 0u, 0u);

  // Chunk assignment, the same for every plane: the chunks that this thread
  // copies (and, in the fused modes, transforms).  rof: a chunk's first value,
  // before rounding down to W, from the plane's first value (32-bit: the grid
  // extent check bounds it).  use / own: chunks inside the grid / in owned rows;
  // a row's owned nodes are the own_len values from 3 past its first, dlo the
  // chunk's offset from them for a lead of 0.
  int rofa[NCT], sba[NCT], dla[NCT];
  bool use[NCT], own[NCT];
  const int own_len = 3 * (min(i0 + MV_BX - 1, g.nxn) - i0);
  const int rstep = 3 * WARPS * g.nxn;
#pragma unroll
  for (int q = 0; q < NCT; ++q) {
    const int ch = tid + q * NT;
    const int b = RUNS ? wy + q * WARPS : ch / CPR, cc = RUNS ? lx : ch - b * CPR;
    const int jj = j0 - 1 + b;
    // a chunk past the row's last node in the grid is not needed
    use[q] = b <= BY && cc < CPR && jj >= 0 && jj < g.nyn && cc * W < 3 * (g.nxn - i0 + 1) + W - 1;
    own[q] = use[q] && b >= 1 && b <= BY - 1;
    rofa[q] = 3 * (jj * g.nxn + i0 - 1) + cc * W;
    sba[q] = b * RS + cc * W;
    dla[q] = cc * W - 3;
  }
  auto rof = [&](int q) { return RUNS ? rofa[0] + q * rstep : rofa[q]; };
  auto sbase = [&](int q) { return RUNS ? sba[0] + q * WARPS * RS : sba[q]; };
  auto dlo = [&](int q) { return RUNS ? dla[0] : dla[q]; };
  __syncthreads();
  if (tid == 0) {
    share_coef(A.K, sm.k);
    sm.k[4] = vneg(vone<V>());
  }
  // everything above may overlap the previous kernel (launch_dep)
  pdl_wait();
  pdl_trigger();
  // MODE 5, 6 inside a solve stop with its state too
  if ((FUSED || (MODE >= 5 && A.st)) && A.st->status != HX_RUNNING) return;
  T alpha_old = T(0), beta_old = T(0);
  if (FUSED) {
    alpha_old = (T)A.st->alpha;
    beta_old = (T)A.st->beta;
  }
  // the iterate that the last iteration flagged as the best so far is complete
  // only here (x + alpha p)
  const bool snap = FUSED && sizeof(T) == 8 && A.xbest && A.st->snap;
  __syncthreads();

  // Node plane kp starts at value pv = kp * P3: a chunk's 16-byte aligned
  // address is the plane's rounded-down base plus a 32-bit offset.
  auto chunk_off = [&](int q, int64_t pv) { return (rof(q) + (int)(pv & (W - 1))) & ~(W - 1); };
  auto plane_ptr = [&](auto* v, int64_t pv) { return v + (pv & ~(int64_t)(W - 1)); };
  // Copies of plane kp of the vectors that the mode stages, chunk by chunk.
  // Only the first and last planes hold chunks that start before the vector
  // or reach past its end: those are cut to the part inside (the rest is 0).
  const bool use_xp = MODE == 5 && !A.xprev_zero && A.omega != T(0);
  const int nzn = g.nzn;
  auto cut = [&](const T* v, T* sdst, int q, int64_t pv) {
    const int64_t at = (pv & ~(int64_t)(W - 1)) + chunk_off(q, pv), left = P3 * (int64_t)nzn - at;
    const unsigned bytes =
        (at >= 0 && left > 0) ? (unsigned)((left < W ? left : (int64_t)W) * sizeof(T)) : 0u;
    cp_async16(smem_u32(sdst + sbase(q)), v + (bytes ? at : 0), bytes);
  };
  auto cut_z32 = [&](T* sdst, int q, int64_t pv) {
    const int64_t at = (pv & ~(int64_t)(W - 1)) + chunk_off(q, pv), left = P3 * (int64_t)nzn - at;
    const unsigned bytes =
        (at >= 0 && left > 0) ? (unsigned)((left < W ? left : (int64_t)W) * sizeof(float)) : 0u;
    cp_async8(smem_u32(sdst + sbase(q)), A.z32 + (bytes ? at : 0), bytes);
  };
  auto issue = [&](int kp, T* p) {
    if ((unsigned)kp > (unsigned)kp_last) return;
    const int64_t pv = (int64_t)kp * P3;
    const bool kown = kp >= k0 && kp < k1;
    if (kp == 0 || kp == nzn - 1) {
#pragma unroll
      for (int q = 0; q < NCT; ++q) {
        if (!use[q]) continue;
        cut(A.pin, p, q, pv);
        if (FUSED) {
          if (MODE == 7)
            cut_z32(p + PLANE, q, pv);
          else
            cut(A.minv, p + PLANE, q, pv);
          if (own[q] && kown) cut(A.x, p + 2 * PLANE, q, pv);
          if (MODE == 3) cut(A.r, p + 3 * PLANE, q, pv);
        }
      }
      return;
    }
    const T* bp = plane_ptr(A.pin, pv);
    const T* bm = FUSED && MODE != 7 ? plane_ptr(A.minv, pv) : nullptr;
    const float* bz = MODE == 7 ? plane_ptr(A.z32, pv) : nullptr;
    const T* bx = FUSED ? plane_ptr((const T*)A.x, pv) : nullptr;
    const T* br = MODE == 3 ? plane_ptr(A.r, pv) : nullptr;
    const unsigned d0 = smem_u32(p);
#pragma unroll
    for (int q = 0; q < NCT; ++q) {
      const int off = chunk_off(q, pv);
      const unsigned d = d0 + sbase(q) * (int)sizeof(T);
      if (use[q]) {
        cp_async16(d, bp + off);
        if (MODE == 7)
          cp_async8(d + PLANE * sizeof(T), bz + off);
        else if (FUSED)
          cp_async16(d + PLANE * sizeof(T), bm + off);
        if (MODE == 3) cp_async16(d + 3 * PLANE * sizeof(T), br + off);
      }
      if (FUSED && own[q] && kown) cp_async16(d + 2 * PLANE * sizeof(T), bx + off);
    }
  };
  auto issue_aux = [&](int kp, T* aux) {
    if (kp < k0 || kp >= k1) return;
    const int64_t pv = (int64_t)kp * P3;
    if (kp == 0 || kp == nzn - 1) {
#pragma unroll
      for (int q = 0; q < NCT; ++q) {
        if (!own[q]) continue;
        cut(A.r, aux, q, pv);
        if (MODE == 5) cut(A.minv, aux + PLANE, q, pv);
        if (MODE == 5 && use_xp) cut(A.x, aux + 2 * PLANE, q, pv);
      }
      return;
    }
    const T* br = plane_ptr(A.r, pv);
    const T* bm = MODE == 5 ? plane_ptr(A.minv, pv) : nullptr;
    const T* bx = MODE == 5 ? plane_ptr((const T*)A.x, pv) : nullptr;
    const unsigned d0 = smem_u32(aux);
#pragma unroll
    for (int q = 0; q < NCT; ++q) {
      const int off = chunk_off(q, pv);
      const unsigned d = d0 + sbase(q) * (int)sizeof(T);
      if (own[q]) {
        cp_async16(d, br + off);
        if (MODE == 5) cp_async16(d + PLANE * sizeof(T), bm + off);
        if (MODE == 5 && use_xp) cp_async16(d + 2 * PLANE * sizeof(T), bx + off);
      }
    }
  };

  // FUSED: p = M^-1 r + beta p_old (MODE 4: z + beta p_old) of this thread's
  // chunks of plane kp into pd; the values of owned nodes of owned planes are
  // stored to p and advance x with the old direction (16-byte stores where a
  // whole chunk is owned).
  auto transform = [&](int kp, const T* src, T* pd) {
    if ((unsigned)kp > (unsigned)kp_last) return;
    const bool kown = kp >= k0 && kp < k1;
    const int64_t pv = (int64_t)kp * P3;
#pragma unroll
    for (int q = 0; q < NCT; ++q) {
      if (!use[q]) continue;
      const T* a = src + sbase(q);
      const VecT po = *reinterpret_cast<const VecT*>(a);
      VecT mv;
      if constexpr (MODE == 7) {
        const float2 zf = *reinterpret_cast<const float2*>(a + PLANE);
        mv = VecT{zf.x, zf.y};
      } else {
        mv = *reinterpret_cast<const VecT*>(a + PLANE);
      }
      const T* pa = reinterpret_cast<const T*>(&po);
      const T* ma = reinterpret_cast<const T*>(&mv);
      VecT rv{};
      if (MODE == 3) rv = *reinterpret_cast<const VecT*>(a + 3 * PLANE);
      const T* ra = reinterpret_cast<const T*>(&rv);
      T pnew[W];
#pragma unroll
      for (int t = 0; t < W; ++t) pnew[t] = (FCG ? ma[t] : ma[t] * ra[t]) + beta_old * pa[t];
      *reinterpret_cast<VecT*>(pd + sbase(q)) = *reinterpret_cast<const VecT*>(pnew);
      if (!kown || !own[q]) continue;
      const VecT xw = *reinterpret_cast<const VecT*>(a + 2 * PLANE);
      const T* xa = reinterpret_cast<const T*>(&xw);
      T xv[W];
#pragma unroll
      for (int t = 0; t < W; ++t) xv[t] = xa[t] + alpha_old * pa[t];
      const int off = chunk_off(q, pv);
      T* pd2 = plane_ptr(A.pout, pv) + off;
      T* xd = plane_ptr(A.x, pv) + off;
      // the chunk's offset from the row's first owned value
      const int d = dlo(q) - ((rof(q) + (int)(pv & (W - 1))) & (W - 1));
      if (d >= 0 && d + W <= own_len) {
        *reinterpret_cast<VecT*>(pd2) = *reinterpret_cast<const VecT*>(pnew);
        *reinterpret_cast<VecT*>(xd) = *reinterpret_cast<const VecT*>(xv);
      } else if (d + W > 0 && d < own_len) {
#pragma unroll
        for (int t = 0; t < W; ++t)
          if (d + t >= 0 && d + t < own_len) {
            pd2[t] = pnew[t];
            xd[t] = xv[t];
          }
      }
      // (as a launch of its own the snapshot cost 1.3 us of 15 per iteration on
      // 60 x 20 x 20 even where none was due)
      if (snap) {
        T* xs = plane_ptr(A.xbest, pv) + off;
#pragma unroll
        for (int t = 0; t < W; ++t)
          if (d + t >= 0 && d + t < own_len) xs[t] = xv[t];
      }
    }
  };

  // This thread's element columns join nodes lx and lx + 1 of R + 1 node
  // rows.  Row b of a plane whose first value has index pl (mod W) starts at
  // b * RS + lead, lead = (pl + lead0[b]) mod W.
  const int row0 = 3 * (jn * g.nxn + i0 - 1);
  const int p3m = P3 & (W - 1);
  unsigned lead0[R + 1];
#pragma unroll
  for (int b = 0; b <= R; ++b) lead0[b] = (unsigned)(row0 + 3 * b * g.nxn) & (W - 1);
  const int basea = R * wy * RS + 3 * lx;
  auto row_at = [&](int b, unsigned pl) {
    return basea + b * RS + (int)((pl + lead0[b]) & (W - 1));
  };
  // face coefficients P[c][sigma_x + 2 sigma_y] of the thread's elements from
  // a staged plane
  T ownn[R][3];  // KEEP: node values of the plane that `face` read last
  auto face = [&](const T* ps, unsigned pl, V (&P)[3][4]) {
    const T* a[R + 1];
#pragma unroll
    for (int b = 0; b <= R; ++b) a[b] = ps + row_at(b, pl);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      T s[R + 1], d[R + 1];
#pragma unroll
      for (int b = 0; b <= R; ++b) {
        const T u = a[b][c], v = a[b][3 + c];
        if (S::KEEP && b < R) ownn[b][c] = u;
        s[b] = u + v;
        d[b] = v - u;
      }
      if constexpr (R == 2) {
        P[c][0] = make_float2(s[0] + s[1], s[1] + s[2]);
        P[c][1] = make_float2(d[0] + d[1], d[1] + d[2]);
        P[c][2] = make_float2(s[1] - s[0], s[2] - s[1]);
        P[c][3] = make_float2(d[1] - d[0], d[2] - d[1]);
      } else {
        P[c][0] = s[0] + s[1];
        P[c][1] = d[0] + d[1];
        P[c][2] = s[1] - s[0];
        P[c][3] = d[1] - d[0];
      }
    }
  };

  // Element factors: columns outside the grid read one inside it and carry a
  // zero scale.  Fetched one layer ahead of their use (a pointer that stays on
  // the first and last layer; layers outside are not computed).
  const int eplane = g.nxe * g.nye;
  const int ie = min(max(in, 0), g.nxe - 1), je = min(max(jn, 0), g.nye - 1);
  const T* fp = A.fac + ((int64_t)max(k0 - 1, 0) * eplane + je * g.nxe + ie);
  const int fstep = R == 2 && jn + 1 < g.nye && jn >= 0 ? g.nxe : 0;
  V fscale;
  {
    const bool cx = in >= 0 && in < g.nxe, cy = jn >= 0 && jn < g.nye;
    if constexpr (R == 2) {
      const bool cy1 = jn + 1 < g.nye;
      const float2 un = CUBE ? unit_of(A.K) : make_float2(1.f, 1.f);
      fscale = make_float2(cx && cy ? un.x : 0.f, cx && cy1 ? un.y : 0.f);
    } else {
      fscale = cx && cy ? (CUBE ? unit_of(A.K) : 1.0) : 0.0;
    }
  }
  auto load_fac = [&]() -> V {
    if constexpr (R == 2)
      return make_float2(fp[0], fp[fstep]);
    else
      return fp[0];
  };
  // Outputs and node masks: pointers that advance with the plane.  The fixed
  // DOFs of q need no mask in the fused steps and none is applied to A x in
  // the Chebyshev step: p and x are 0 there and so is M^-1, which every use
  // of q and A x multiplies by or tests.
  constexpr bool MASK = MODE == 0 || MODE == 1 || MODE == 6;
  bool out_ok[R];
#pragma unroll
  for (int b = 0; b < R; ++b)
    out_ok[b] = lx >= 1 && R * wy + b >= 1 && in < g.nxn && jn + b < g.nyn;
  const int64_t first = (int64_t)k0 * nplane + jn * g.nxn + in;  // node of plane k0
  const bool has_mask = MASK && A.nmask != nullptr;
  const uint8_t* mp = has_mask ? A.nmask + first : nullptr;
  T* qp = (MODE == 5 ? A.x : A.q) + 3 * first;

  double dsum = 0.0;
  T rowS[R][3], ownp[R][3];  // plane ke: sums so far, node values
  unsigned mk[R];
#pragma unroll
  for (int b = 0; b < R; ++b) mk[b] = 7u;
  unsigned plo = (unsigned)((int64_t)(k0 - 1) * p3m) & (W - 1);  // pl of plane ke (then kn)
  // Finishes node plane ke - 1 (owned): the neighbouring warp's partial,
  // shift, mask, output.
  const T wx = MODE == 5 ? T(1) + (use_xp || A.xprev_zero ? A.omega : T(0)) : T(0);
  auto finish = [&](int par, const T* aux, unsigned pl) {
    bool masked = false;
    if (MASK && has_mask) {
      unsigned all = 7u;
      for (int b = 0; b < R; ++b) all &= mk[b];
      masked = __any_sync(0xffffffffu, all != 7u);
    }
#pragma unroll
    for (int b = 0; b < R; ++b) {
      T pdot = T(0);  // this node's p.q in T (3 terms), accumulated in FP64
      T o[3];
      const T* ax = (MODE == 5 || MODE == 6) ? aux + row_at(b, pl) : nullptr;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T v = rowS[b][c];
        if (b == 0) v += sm.red[par][wy][c][lx];
        const T xv = ownp[b][c];
        v = fma(A.shift, xv, v);
        if (MODE == 5) {
          // x_prev: read, or 0 (the step after a start from x = 0), or
          // unused (the first step: omega = 0)
          v = fma(A.gamma * ax[PLANE + c], ax[c] - v, wx * xv);
          if (use_xp) v = fma(-A.omega, ax[2 * PLANE + c], v);
        } else if (MODE == 6) {
          v = ax[c] - v;
        }
        o[c] = v;
        if (DOT) pdot = fma(xv, v, pdot);
      }
      if (MASK && masked)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if (!((mk[b] >> c) & 1u)) o[c] = T(0);
      if (out_ok[b]) {
        T* d = qp + 3 * b * g.nxn;
#pragma unroll
        for (int c = 0; c < 3; ++c) d[c] = o[c];
        if (DOT) dsum += (double)pdot;
      }
    }
    qp += P3;
  };

  const V m1 = from_shared<V>(&sm.k[4]);
  CoefV<V, CUBE> K = A.K;
  pin_coef(K, sm.k);
  V Ytp[3][4], Pb[3][4];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int q = 0; q < 4; ++q) Ytp[c][q] = Pb[c][q] = vzero<V>();

  // Prologue: the first planes requested; planes k0-1 and k0 ready, the face
  // coefficients of plane k0-1 formed.  Slots: plane kp of p in slot (kp -
  // k0 + 1) mod NX, of the fused inputs mod NS; aux plane kp in (kp - k0) mod
  // NA.  One commit group per call of issue, so that the wait counts hold to
  // the end of the chunk.
  auto step = [](int v, int n) { return v + 1 == n ? 0 : v + 1; };
  int sp = 0, sa = 0;  // fused: slot of plane ke + 2; else of plane ke, of aux plane ke + 1
  if constexpr (FUSED) {
#pragma unroll 1
    for (int d = 0; d < S::NS; ++d) {
      issue(k0 - 1 + d, &sm.in[d][0][0]);
      cp_async_commit();
    }
#pragma unroll 1
    for (int d = 0; d < 2; ++d) {
      cp_async_wait<S::NS - 1>();
      transform(k0 - 1 + d, &sm.in[d][0][0], sm.p[d]);
      issue(k0 - 1 + d + S::NS, &sm.in[d][0][0]);
      cp_async_commit();
    }
    sp = 2 % S::NS;
    __syncthreads();
  } else {
#pragma unroll 1
    for (int d = 0; d < S::NX - 1; ++d) {
      issue(k0 - 1 + d, sm.p[d]);
      cp_async_commit();
    }
    cp_async_wait<S::NX - 2>();
    __syncthreads();
  }
#pragma unroll
  for (int b = 0; b < R; ++b)
#pragma unroll
    for (int c = 0; c < 3; ++c) ownn[b][c] = T(0);
  if (k0 > 0) face(sm.p[0], plo, Pb);
  V f_next = load_fac();
  int s0 = 0;  // slot of plane ke

#pragma unroll 1
  for (int ke = k0 - 1; ke < k1; ++ke) {
    const V f = vmul(f_next, fscale);
    fp += ke >= 0 && ke + 1 < g.nze ? eplane : 0;
    f_next = load_fac();
    const int s1 = step(s0, S::NX), s2 = step(s1, S::NX);
    if constexpr (!FUSED) cp_async_wait<(S::AUX ? 1 : S::NX - 3)>();
    __syncthreads();  // plane ke+1 ready; red of plane ke-1 visible; plane ke-1 consumed
    if (ke - 1 >= k0)
      finish((ke - 1) & 1, &sm.in[S::AUX ? step(sa, S::NA) : 0][0][0], plo - p3m);
    if constexpr (!FUSED) {
      issue(ke - 1 + S::NX, sm.p[sp == 0 ? S::NX - 1 : sp - 1]);
      if (S::AUX) {
        issue_aux(ke - 2 + S::NA, &sm.in[sa][0][0]);
        sa = step(sa, S::NA);
      }
      cp_async_commit();
      sp = step(sp, S::NX);
    } else {
      cp_async_wait<S::NS - 1>();
      transform(ke + 2, &sm.in[sp][0][0], sm.p[s2]);
      issue(ke + 2 + S::NS, &sm.in[sp][0][0]);
      cp_async_commit();
      sp = step(sp, S::NS);
    }
    if (has_mask && ke >= k0) {
#pragma unroll
      for (int b = 0; b < R; ++b)
        if (out_ok[b]) mk[b] = mp[b * g.nxn];
      mp += nplane;
    }

    if constexpr (S::KEEP) {
#pragma unroll
      for (int b = 0; b < R; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) ownp[b][c] = ownn[b][c];
    }

    // Element layer ke: bottom face f (Y_s - Y_d) plus the layer below's top
    // face; top face f (Y_s + Y_d), carried to the layer above.
    V F[3][4];
    if (ke >= 0 && ke < g.nze) {
      V Pt[3][4];
      face(sm.p[s1], plo + p3m, Pt);
      const V nf = vneg(f);
      auto blocks = [&](auto qc) {
        constexpr int Q = decltype(qc)::value;
        constexpr int e[3] = {Q ^ 1, Q ^ 2, Q};
        V s[3], d[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (e[c] != 0) s[c] = vadd(Pb[c][e[c]], Pt[c][e[c]]);
          else s[c] = vzero<V>();
          d[c] = vsubm(Pt[c][e[c]], Pb[c][e[c]], m1);
        }
        lambda_pair<Q>(K, s, d);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          V& y = Ytp[c][e[c]];
          if (e[c] == 0) {
            F[c][0] = vfma(nf, d[c], y);
            y = vmul(f, d[c]);
          } else {
            F[c][e[c]] = vfma(nf, d[c], vfma(f, s[c], y));
            y = vfma(f, d[c], vmul(f, s[c]));
          }
        }
      };
      blocks(std::integral_constant<int, 0>{});
      blocks(std::integral_constant<int, 1>{});
      blocks(std::integral_constant<int, 2>{});
      blocks(std::integral_constant<int, 3>{});
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q) Pb[c][q] = Pt[c][q];
    } else {
      // no elements below the first and above the last node plane
      if (ke < 0) face(sm.p[s1], plo + p3m, Pb);
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q) F[c][q] = Ytp[c][q];
    }
    // y and x transforms back to the R + 1 node rows
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const V as = vsubm(F[c][0], F[c][2], m1), ad = vsubm(F[c][1], F[c][3], m1);
      const V bs = vadd(F[c][0], F[c][2]), bd = vadd(F[c][1], F[c][3]);
      T s[R + 1], d[R + 1];
      if constexpr (R == 2) {
        s[0] = as.x;
        d[0] = ad.x;
        s[1] = bs.x + as.y;
        d[1] = bd.x + ad.y;
        s[2] = bs.y;
        d[2] = bd.y;
      } else {
        s[0] = as;
        d[0] = ad;
        s[1] = bs;
        d[1] = bd;
      }
#pragma unroll
      for (int b = 0; b <= R; ++b) {
        const T left = s[b] - d[b], right = s[b] + d[b];
        // element lx-1 contributes its +x corners to this thread's nodes
        const T t = left + __shfl_up_sync(0xffffffffu, right, 1);
        if (b < R)
          rowS[b][c] = t;
        else if (wy + 1 < WARPS)
          sm.red[ke & 1][wy + 1][c][lx] = t;
      }
    }
    if constexpr (!S::KEEP) {  // the node values of plane ke: its slot lives until the next barrier
#pragma unroll
      for (int b = 0; b < R; ++b) {
        const T* a = sm.p[s0] + row_at(b, plo);
#pragma unroll
        for (int c = 0; c < 3; ++c) ownp[b][c] = a[c];
      }
    }
    s0 = s1;
    plo += p3m;
  }
  cp_async_wait<0>();
  __syncthreads();  // red of plane k1-1 visible
  finish((k1 - 1) & 1, &sm.in[S::AUX ? step(sa, S::NA) : 0][0][0], plo - p3m);

  if (DOT) {
    double v[1] = {dsum};
    if (grid_reduce<1>(v, A.partials, &A.st->ticket[TK_MATVEC]) && tid == 0) {
      if (MODE == 1) {
        A.out[0] = v[0];
      } else {
        const double pq = v[0], num = FCG ? A.st->aux[3] : A.st->rz;
        A.st->pq = pq;
        if (!(pq > 0.0) || !isfinite(pq) || (FCG && !isfinite(num)))
          A.st->status = HX_ST_BREAKDOWN;
        else
          A.st->alpha = num / pq;
      }
    }
  }
}

// Factors beyond the range of the FP32 forms, infinite or NaN.
__device__ __forceinline__ bool beyond_range(double f) { return !(fabs(f) <= 3e38); }

// Per-node Jacobi diagonal: diag(n,c) = kd[c] * sum of the factors of the
// (up to 8) elements around n; node mask = free-DOF bits of `bcfree`
// cleared where the node carries no stiffness (or a NaN).  Writes diag into `diag`,
// the mask into `nmask`, and reduces the max diagonal over free DOFs (out[0]) and
// whether any node's sum is beyond_range (out[1]).
template <typename T>
__global__ void k_node_diag(const T* __restrict__ fac, const uint8_t* __restrict__ bcfree,
                            uint8_t* __restrict__ nmask, T* __restrict__ diag, Grid g,
                            ElemCoef<double> K, double* partials, CgState* st, double* out) {
  const int64_t nn = (int64_t)g.nxn * g.nyn * g.nzn;
  double mx = 0.0, wild = 0.0;
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nn;
       n += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(n % g.nxn);
    const int64_t r = n / g.nxn;
    const int j = (int)(r % g.nyn);
    const int k = (int)(r / g.nyn);
    double s = 0.0;
#pragma unroll
    for (int dk = -1; dk <= 0; ++dk)
#pragma unroll
      for (int dj = -1; dj <= 0; ++dj)
#pragma unroll
        for (int di = -1; di <= 0; ++di) {
          const int ei = i + di, ej = j + dj, ek = k + dk;
          if (ei >= 0 && ej >= 0 && ek >= 0 && ei < g.nxe && ej < g.nye && ek < g.nze)
            s += (double)fac[((int64_t)ek * g.nye + ej) * g.nxe + ei];
        }
    if (beyond_range(s)) wild = 1.0;
    const unsigned m = (s > 0.0) ? (bcfree ? bcfree[n] : 7u) : 0u;
    nmask[n] = (uint8_t)m;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double d = K.kd[c] * s;
      diag[3 * n + c] = (T)d;
      if ((m >> c) & 1u) mx = fmax(mx, d);
    }
  }
  double v[2] = {mx, wild};
  if (grid_reduce<2, true>(v, partials, &st->ticket[TK_AUX]) && threadIdx.x == 0) {
    out[0] = v[0];
    out[1] = v[1];
  }
}

// The factors with those beyond_range set to 0 where all nodes of the element are
// fixed: it has no part in any free row, but 0 times such a factor is a NaN.
__global__ void k_bounded_factors(const double* __restrict__ fac,
                                  const uint8_t* __restrict__ nmask, double* __restrict__ out,
                                  Grid g) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < g.elems();
       e += (int64_t)gridDim.x * blockDim.x) {
    double f = fac[e];
    if (beyond_range(f)) {
      const int i = (int)(e % g.nxe);
      const int64_t r = e / g.nxe;
      const int j = (int)(r % g.nye), k = (int)(r / g.nye);
      unsigned free = 0;
      for (int b = 0; b < 8; ++b)
        free |= nmask[((int64_t)(k + (b >> 2)) * g.nyn + j + ((b >> 1) & 1)) * g.nxn + i + (b & 1)];
      if (!free) f = 0.0;
    }
    out[e] = f;
  }
}

// minv = free ? 1/(diag + shift) : 0   (src/Solvers/GPUSolver.jl:402)
template <typename T>
__global__ void k_minv(const uint8_t* __restrict__ nmask, const T* __restrict__ diag,
                       T* __restrict__ minv, int64_t nn, double shift) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 3 * nn;
       i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned m = nmask[i / 3];
    const int c = (int)(i % 3);
    minv[i] = ((m >> c) & 1u) ? (T)(1.0 / ((double)diag[i] + shift)) : T(0);
  }
}

// Node planes per CTA: the chunk length kc that minimises (waves of resident
// CTAs) x (element layers each CTA works on, kc + 1, and one for its start and
// end).  A last wave that fills few SMs costs as much as a full one; ties go
// to the longer chunk.  Short chunks win only where the grid leaves SMs idle.
// For a number of chunks only the shortest length counts, so a grid of n planes has
// about 2 sqrt(n) candidates (1001 planes: 0.75 us instead of 3.5 for all lengths;
// a call asks up to five times).
template <typename T, bool FUSED>
int mv_kchunk(const Grid& g) {
  const int64_t cols = (int64_t)cdiv(g.nxn, MV_BX - 1) * cdiv(g.nyn, mv_by<T, FUSED>() - 1);
  const int64_t slots = (int64_t)Tile<T, FUSED>::RESIDENT * sm_count();
  int best_kc = g.nzn;
  int64_t best = INT64_MAX;
  for (int kc = g.nzn; kc >= 1; --kc) {
    const int chunks = cdiv(g.nzn, kc);
    kc = cdiv(g.nzn, chunks);
    const int64_t cost = (int64_t)cdiv(cols * chunks, slots) * (kc + 2);
    if (cost < best) {
      best = cost;
      best_kc = kc;
    }
  }
  return best_kc;
}

// CTA columns in x, columns in y, chunks.  A grid's y extent ends at 65535, which
// more than 327000 node rows in y reach (the columns in x never do: 2^20 nodes
// are 33826 of them): x and y are exchanged there.
constexpr unsigned MAX_GRID_Y = 65535;
template <typename T, bool FUSED>
dim3 mv_grid(const Grid& g, int kchunk) {
  return dim3(cdiv(g.nxn, MV_BX - 1), cdiv(g.nyn, mv_by<T, FUSED>() - 1), cdiv(g.nzn, kchunk));
}

template <typename T, int MODE, bool CUBE>
void launch_one(cudaStream_t s, OpArgs<T, CUBE>& a, const ElemCoef<T>& K) {
  constexpr size_t smem = sizeof(Smem<T, MODE>);
  static_assert(smem % 16 == 0, "zeroed in 16-byte steps");
  constexpr bool FUSED = mode_fused(MODE);
  using Form = Tile<T, FUSED>;
  static_assert(Form::RESIDENT * (smem + 1024 + 512) <= 228 * 1024, "the CTAs of an SM fit");
  static PerDeviceOnce configured;  // per instantiation and device
  configured.run([&] {
    HX_CUDA(cudaFuncSetAttribute(k_struct<T, MODE, CUBE>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  });
  coef_v(K, a.K);
  a.kchunk = mv_kchunk<T, FUSED>(a.g);
  dim3 grid = mv_grid<T, FUSED>(a.g, a.kchunk);
  a.yx = grid.y > MAX_GRID_Y;
  if (a.yx) std::swap(grid.x, grid.y);
  launch_dep(one_wave((int64_t)grid.x * grid.y * grid.z, Form::RESIDENT), k_struct<T, MODE, CUBE>,
             grid, dim3(MV_BX, Form::WARPS), smem, s, a);
  HX_CHECK_LAUNCH();
}

// `fill` sets the mode's fields of the arguments.
template <typename T, int MODE, typename F>
void launch_struct(cudaStream_t s, const T* fac, const uint8_t* nmask, const Grid& g,
                   const ElemCoef<T>& K, T shift, F&& fill) {
  auto go = [&](auto cube) {
    OpArgs<T, decltype(cube)::value> a{};
    a.fac = fac;
    a.nmask = nmask;
    a.g = g;
    a.shift = shift;
    fill(a);
    launch_one<T, MODE>(s, a, K);
  };
  // equal sides: every axis has the same coefficients
  if (K.mu[0][0] == K.mu[1][0] && K.mu[1][0] == K.mu[2][0])
    go(std::true_type{});
  else
    go(std::false_type{});
}

template <typename T, bool FUSED>
size_t num_blocks(const Grid& g) {
  const dim3 a = mv_grid<T, FUSED>(g, mv_kchunk<T, FUSED>(g));
  return (size_t)a.x * a.y * a.z;
}

}  // namespace

template <typename T>
size_t mv_num_blocks(const Grid& g) {
  return std::max(num_blocks<T, true>(g), num_blocks<T, false>(g));
}
template size_t mv_num_blocks<float>(const Grid&);
template size_t mv_num_blocks<double>(const Grid&);

size_t mv_apply_blocks(const Grid& g) { return num_blocks<double, false>(g); }

template <typename T>
void launch_matvec(cudaStream_t s, int mode, const T* x, T* y, const T* fac, const uint8_t* nmask,
                   const Grid& g, const ElemCoef<T>& K, T shift, CgState* st, double* partials,
                   double* out) {
  auto fill = [&](auto& a) {
    a.pin = x;
    a.q = y;
    a.st = st;
    a.partials = partials;
    a.out = out;
  };
  if (mode == 0)
    launch_struct<T, 0>(s, fac, nmask, g, K, shift, fill);
  else
    launch_struct<T, 1>(s, fac, nmask, g, K, shift, fill);
}
template void launch_matvec<double>(cudaStream_t, int, const double*, double*, const double*,
                                    const uint8_t*, const Grid&, const ElemCoef<double>&, double,
                                    CgState*, double*, double*);

template <typename T>
void launch_cheb_step(cudaStream_t s, const T* x, T* xprev_new, bool xprev_zero, const T* b,
                      const T* minv, T omega, T gamma, const T* fac, const uint8_t* nmask,
                      const Grid& g, const ElemCoef<T>& K, T shift, const CgState* st) {
  launch_struct<T, 5>(s, fac, nmask, g, K, shift, [&](auto& a) {
    a.st = const_cast<CgState*>(st);
    a.pin = x;
    a.x = xprev_new;
    a.xprev_zero = xprev_zero ? 1 : 0;
    a.r = b;
    a.minv = minv;
    a.omega = omega;
    a.gamma = gamma;
  });
}
template void launch_cheb_step<float>(cudaStream_t, const float*, float*, bool, const float*,
                                      const float*, float, float, const float*, const uint8_t*,
                                      const Grid&, const ElemCoef<float>&, float, const CgState*);

template <typename T>
void launch_residual(cudaStream_t s, const T* x, const T* b, T* r, const T* fac,
                     const uint8_t* nmask, const Grid& g, const ElemCoef<T>& K, T shift,
                     const CgState* st) {
  launch_struct<T, 6>(s, fac, nmask, g, K, shift, [&](auto& a) {
    a.st = const_cast<CgState*>(st);
    a.pin = x;
    a.r = b;
    a.q = r;
  });
}
template void launch_residual<float>(cudaStream_t, const float*, const float*, float*,
                                     const float*, const uint8_t*, const Grid&,
                                     const ElemCoef<float>&, float, const CgState*);

template <typename T>
void launch_pcg_step(cudaStream_t s, const T* pin, T* pout, const T* r, const T* minv, T* x, T* q,
                     const T* fac, const uint8_t* nmask, const Grid& g, const ElemCoef<T>& K,
                     T shift, CgState* st, double* partials, T* xbest) {
  launch_struct<T, 3>(s, fac, nmask, g, K, shift, [&](auto& a) {
    a.xbest = xbest;
    a.pin = pin;
    a.pout = pout;
    a.r = r;
    a.minv = minv;
    a.x = x;
    a.q = q;
    a.st = st;
    a.partials = partials;
  });
}
template void launch_pcg_step<double>(cudaStream_t, const double*, double*, const double*,
                                      const double*, double*, double*, const double*,
                                      const uint8_t*, const Grid&, const ElemCoef<double>&,
                                      double, CgState*, double*, double*);
template void launch_pcg_step<float>(cudaStream_t, const float*, float*, const float*,
                                     const float*, float*, float*, const float*, const uint8_t*,
                                     const Grid&, const ElemCoef<float>&, float, CgState*,
                                     double*, float*);

template <typename T, typename TZ>
void launch_fcg_step(cudaStream_t s, const T* pin, T* pout, const TZ* z, T* x, T* q, const T* fac,
                     const uint8_t* nmask, const Grid& g, const ElemCoef<T>& K, T shift,
                     CgState* st, double* partials, T* xbest) {
  constexpr bool SAME = std::is_same<T, TZ>::value;
  launch_struct<T, SAME ? 4 : 7>(s, fac, nmask, g, K, shift, [&](auto& a) {
    a.xbest = xbest;
    a.pin = pin;
    a.pout = pout;
    if constexpr (SAME)
      a.minv = z;
    else
      a.z32 = z;
    a.x = x;
    a.q = q;
    a.st = st;
    a.partials = partials;
  });
}
template void launch_fcg_step<double>(cudaStream_t, const double*, double*, const double*,
                                      double*, double*, const double*, const uint8_t*,
                                      const Grid&, const ElemCoef<double>&, double, CgState*,
                                      double*, double*);
template void launch_fcg_step<double, float>(cudaStream_t, const double*, double*, const float*,
                                             double*, double*, const double*, const uint8_t*,
                                             const Grid&, const ElemCoef<double>&, double,
                                             CgState*, double*, double*);
template void launch_fcg_step<float>(cudaStream_t, const float*, float*, const float*, float*,
                                     float*, const float*, const uint8_t*, const Grid&,
                                     const ElemCoef<float>&, float, CgState*, double*,
                                     float*);

template <typename T>
void launch_node_diag(cudaStream_t s, const T* fac, const uint8_t* bcfree, uint8_t* nmask, T* diag,
                      const Grid& g, const ElemCoef<double>& K, double* partials, CgState* st,
                      double* out) {
  const int64_t nn = (int64_t)g.nxn * g.nyn * g.nzn;
  const unsigned blocks = std::min<int64_t>(cdiv(nn, 256), 8LL * sm_count());
  k_node_diag<T><<<blocks, 256, 0, s>>>(fac, bcfree, nmask, diag, g, K, partials, st, out);
  HX_CHECK_LAUNCH();
}
template void launch_node_diag<double>(cudaStream_t, const double*, const uint8_t*, uint8_t*,
                                       double*, const Grid&, const ElemCoef<double>&, double*,
                                       CgState*, double*);
template void launch_node_diag<float>(cudaStream_t, const float*, const uint8_t*, uint8_t*, float*,
                                      const Grid&, const ElemCoef<double>&, double*, CgState*,
                                      double*);

void launch_bounded_factors(cudaStream_t s, const double* fac, const uint8_t* nmask, double* out,
                            const Grid& g) {
  const unsigned blocks = std::min<int64_t>(cdiv(g.elems(), 256), 8LL * sm_count());
  k_bounded_factors<<<blocks, 256, 0, s>>>(fac, nmask, out, g);
  HX_CHECK_LAUNCH();
}

template <typename T>
void launch_minv(cudaStream_t s, const uint8_t* nmask, const T* diag, T* minv, int64_t nn,
                 double shift) {
  const unsigned blocks = std::min<int64_t>(cdiv(3 * nn, 256), 16LL * sm_count());
  k_minv<T><<<blocks, 256, 0, s>>>(nmask, diag, minv, nn, shift);
  HX_CHECK_LAUNCH();
}
template void launch_minv<double>(cudaStream_t, const uint8_t*, const double*, double*, int64_t,
                                  double);
template void launch_minv<float>(cudaStream_t, const uint8_t*, const float*, float*, int64_t,
                                 double);

}  // namespace hx
