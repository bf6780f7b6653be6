// hx_vector.cu -- fused Krylov vector kernels with device-side scalars.
//
// One CG iteration of the reference (src/Solvers/GPUSolver.jl:452-526) is
// ~8 broadcast kernels plus 3 cuBLAS dots, each dot a host round trip.  Here
// it is two kernels and no host round trip:
//   PCG step (hx_operator.cu):  p = M^-1 r + beta p_old; x += alpha_old p_old;
//                  q = A p; pq = p.q; alpha = rz/pq
//   k_cg_update2:  r -= alpha q; z = M^-1 r (not stored); rz' = r.z,
//                  rr = r.r; convergence / divergence tests; beta = rz'/rz
// x lags one step behind (x += alpha p happens in the next PCG step); the
// host applies the last step with k_axpy_state once the loop stops.
// All reductions are FP64 and deterministic (fixed-order block partials).
#include "hx_internal.h"

namespace hx {

namespace {

// 16 bytes of T, loaded and stored as one vector (W entries)
template <typename T>
struct Vec16;
template <>
struct Vec16<double> {
  using type = double2;
  static constexpr int W = 2;
  __device__ static void get(const double2& v, double (&a)[2]) { a[0] = v.x; a[1] = v.y; }
  __device__ static double2 make(const double (&a)[2]) { return make_double2(a[0], a[1]); }
};
template <>
struct Vec16<float> {
  using type = float4;
  static constexpr int W = 4;
  __device__ static void get(const float4& v, float (&a)[4]) {
    a[0] = v.x;
    a[1] = v.y;
    a[2] = v.z;
    a[3] = v.w;
  }
  __device__ static float4 make(const float (&a)[4]) { return make_float4(a[0], a[1], a[2], a[3]); }
};

// M^-1 entry of a free DOF (the fixed ones' is 0); the integer test of the
// upper half keeps FP64 comparisons off the FP64 pipe
__device__ __forceinline__ bool is_free(double m) { return __double2hiint(m) != 0; }
__device__ __forceinline__ bool is_free(float m) { return m != 0.f; }

__device__ __forceinline__ uint32_t bf16x2_bits(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ int64_t gtid() {
  return (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
}
__device__ __forceinline__ int64_t gstride() { return (int64_t)gridDim.x * blockDim.x; }

// r = b - q (q may be null), z = M^-1 r, p = z; reduces rz, rr, bb.
template <typename T>
__global__ void k_cg_init(const T* __restrict__ b, const T* __restrict__ q,
                          const T* __restrict__ minv, T* __restrict__ r, T* __restrict__ p,
                          int64_t n, CgState* st, double* partials) {
  double rz = 0, rr = 0, bb = 0;
  for (int64_t i = gtid(); i < n; i += gstride()) {
    const T bi = b[i];
    const T ri = q ? bi - q[i] : bi;
    const T zi = minv[i] * ri;
    r[i] = ri;
    p[i] = zi;
    rz += (double)ri * (double)zi;
    rr += (double)ri * (double)ri;
    bb += (double)bi * (double)bi;
  }
  double v[3] = {rz, rr, bb};
  if (grid_reduce<3>(v, partials, &st->ticket[TK_INIT]) && threadIdx.x == 0) {
    st->rz = v[0];
    st->rr = v[1];
    st->bnorm = sqrt(v[2]);
    st->iter = 0;
    st->best_rel = INFINITY;
    st->snap = 0;
    if (st->bnorm == 0.0) {
      st->rel_res = 0.0;
      st->status = HX_ST_ZERO_RHS;
    } else {
      st->rel_res = sqrt(v[1]) / st->bnorm;
      st->status = isfinite(st->rel_res) ? HX_RUNNING : HX_ST_NONFINITE;
    }
  }
}

// Second half of a fused PCG iteration: r -= alpha q on the free DOFs (M^-1
// is 0 on the fixed ones, where the operator leaves q unmasked), dots, tests.  With
// ys: also ys = BF16(D^-1/2 r) of the new residual (the learned
// preconditioner's input, D^-1/2 = sqrt(minv)).  16-byte vector accesses
// (4 FP32 or 2 FP64 entries per thread and step), then a scalar tail.
template <typename T>
__global__ void k_cg_update2(T* __restrict__ r, const T* __restrict__ q,
                             const T* __restrict__ minv, int64_t n, CgState* st,
                             double* partials, __nv_bfloat16* __restrict__ ys) {
  pdl_wait();
  pdl_trigger();
  if (st->status != HX_RUNNING) return;
  const T alpha = (T)st->alpha;
  __shared__ CgState s0;  // read after grid_reduce's barriers
  load_state(&s0, st);
  double rz = 0, rr = 0;
  using VT = Vec16<T>;
  using V = typename VT::type;
  constexpr int W = VT::W;
  const int64_t nv = n / W;
  V* rV = reinterpret_cast<V*>(r);
  const V* qV = reinterpret_cast<const V*>(q);
  const V* mV = reinterpret_cast<const V*>(minv);
  for (int64_t i = gtid(); i < nv; i += gstride()) {
    T ra[W], qa[W], ma[W];
    VT::get(rV[i], ra);
    VT::get(qV[i], qa);
    VT::get(mV[i], ma);
    float ya[W];
#pragma unroll
    for (int e = 0; e < W; ++e) {
      ra[e] = is_free(ma[e]) ? ra[e] - alpha * qa[e] : T(0);
      ya[e] = dinv_sqrt((float)ma[e]) * (float)ra[e];
      rz += (double)ra[e] * (double)(ma[e] * ra[e]);
      rr += (double)ra[e] * (double)ra[e];
    }
    rV[i] = VT::make(ra);
    if (ys) {
      if constexpr (W == 4)
        reinterpret_cast<uint2*>(ys)[i] =
            make_uint2(bf16x2_bits(ya[0], ya[1]), bf16x2_bits(ya[2], ya[3]));
      else
        reinterpret_cast<uint32_t*>(ys)[i] = bf16x2_bits(ya[0], ya[1]);
    }
  }
  for (int64_t i = nv * W + gtid(); i < n; i += gstride()) {
    const T ri = is_free(minv[i]) ? r[i] - alpha * q[i] : T(0);
    r[i] = ri;
    if (ys) ys[i] = __float2bfloat16_rn(dinv_sqrt((float)minv[i]) * (float)ri);
    rz += (double)ri * (double)(minv[i] * ri);
    rr += (double)ri * (double)ri;
  }
  double v[2] = {rz, rr};
  if (grid_reduce<2>(v, partials, &st->ticket[TK_UPDATE]) && threadIdx.x == 0)
    cg_finish_iteration(st, s0, v[0], v[1]);
}

// k_cg_update2 of the multigrid solve (see launch_fcg_update).  Bound by its 28
// bytes per DOF: reading M^-1 for the mask, and a copy of r to FP32 as a
// launch of its own, made it 44 (320 x 160 x 160: 119 us instead of 126 + 39).
__global__ void k_fcg_update(double* __restrict__ r, const double* __restrict__ q,
                             const uint8_t* __restrict__ nmask, int64_t n, CgState* st,
                             double* partials, float* __restrict__ r32) {
  pdl_wait();
  pdl_trigger();
  if (st->status != HX_RUNNING) return;
  const double alpha = st->alpha;
  __shared__ CgState s0;  // read after grid_reduce's barriers
  load_state(&s0, st);
  double rr = 0;
  auto upd = [&](unsigned free, double ri, double qi) {
    const double v = free ? ri - alpha * qi : 0.0;
    rr += v * v;
    return v;
  };
  const int64_t nv = n / 2;
  double2* rV = reinterpret_cast<double2*>(r);
  const double2* qV = reinterpret_cast<const double2*>(q);
  float2* sV = reinterpret_cast<float2*>(r32);
  // entry 2 i is component c of `node`; both advance with i (no division)
  int64_t node = 2 * gtid() / 3;
  int c = (int)(2 * gtid() - 3 * node);
  const int64_t dn = 2 * gstride() / 3;
  const int dc = (int)(2 * gstride() - 3 * dn);
#pragma unroll 2
  for (int64_t i = gtid(); i < nv; i += gstride()) {
    double2 a = rV[i];
    const double2 b = qV[i];
    const unsigned m0 = nmask[node], m1 = nmask[node + (c == 2)];
    a.x = upd((m0 >> c) & 1u, a.x, b.x);
    a.y = upd((m1 >> (c == 2 ? 0 : c + 1)) & 1u, a.y, b.y);
    rV[i] = a;
    sV[i] = make_float2((float)a.x, (float)a.y);
    node += dn;
    c += dc;
    if (c >= 3) {
      c -= 3;
      ++node;
    }
  }
  for (int64_t i = 2 * nv + gtid(); i < n; i += gstride()) {
    r[i] = upd(((unsigned)nmask[i / 3] >> (int)(i % 3)) & 1u, r[i], q[i]);
    r32[i] = (float)r[i];
  }
  // (r.z = r.r: the flexible step sets its own coefficients before they are used)
  double v[1] = {rr};
  if (grid_reduce<1>(v, partials, &st->ticket[TK_UPDATE]) && threadIdx.x == 0)
    cg_finish_iteration(st, s0, v[0], v[0]);
}

// ys = BF16(D^-1/2 r), as k_cg_update2 writes it (for a residual that
// another kernel produced).
template <typename T>
__global__ void k_dinv_bf16(const T* __restrict__ r, const T* __restrict__ minv,
                            __nv_bfloat16* __restrict__ ys, int64_t n) {
  for (int64_t i = gtid(); i < n; i += gstride())
    ys[i] = __float2bfloat16_rn(dinv_sqrt((float)minv[i]) * (float)r[i]);
}

// dst = x + alpha p, with alpha from the state; with when_snap only if the last
// iteration was flagged as the best so far.
template <typename T>
__global__ void k_axpy_state(T* __restrict__ dst, const T* __restrict__ x,
                             const T* __restrict__ p, int64_t n, const CgState* st,
                             int when_snap) {
  pdl_wait();
  pdl_trigger();
  if (when_snap && !st->snap) return;
  const T a = (T)st->alpha;
  for (int64_t i = gtid(); i < n; i += gstride()) dst[i] = x[i] + a * p[i];
}

__global__ void k_resid_norm(const double* __restrict__ b, const double* __restrict__ q,
                             int64_t n, CgState* st, double* partials, double* out2) {
  double rr = 0, bb = 0;
  for (int64_t i = gtid(); i < n; i += gstride()) {
    const double bi = b[i], ri = bi - q[i];
    rr += ri * ri;
    bb += bi * bi;
  }
  double v[2] = {rr, bb};
  if (grid_reduce<2>(v, partials, &st->ticket[TK_AUX2]) && threadIdx.x == 0) {
    out2[0] = v[0];
    out2[1] = v[1];
  }
}

template <typename T>
__global__ void k_mask_rhs(const double* __restrict__ f, const T* __restrict__ minv,
                           double* __restrict__ b, int64_t n) {
  for (int64_t i = gtid(); i < n; i += gstride()) b[i] = (minv[i] != T(0)) ? f[i] : 0.0;
}

__global__ void k_dot(const double* __restrict__ a, const double* __restrict__ b, int64_t n,
                      CgState* st, double* partials, double* out) {
  double s = 0;
  for (int64_t i = gtid(); i < n; i += gstride()) s += a[i] * b[i];
  double v[1] = {s};
  if (grid_reduce<1>(v, partials, &st->ticket[TK_AUX2]) && threadIdx.x == 0) out[0] = v[0];
}

// Outer step of mixed-precision refinement: r = b - q in FP64, r32 = r/||b||,
// ||r|| reduced; convergence of the outer loop decided on the true residual.
__global__ void k_ir_residual(const double* __restrict__ b, const double* __restrict__ q,
                              float* __restrict__ r32, int64_t n, CgState* st,
                              double* partials) {
  if (st->status != HX_RUNNING) return;
  const double inv_b = 1.0 / st->bnorm;
  double rr = 0;
  for (int64_t i = gtid(); i < n; i += gstride()) {
    const double ri = b[i] - q[i];
    r32[i] = (float)(ri * inv_b);
    rr += ri * ri;
  }
  double v[1] = {rr};
  if (grid_reduce<1>(v, partials, &st->ticket[TK_UPDATE]) && threadIdx.x == 0) {
    const double rel = sqrt(v[0]) / st->bnorm;
    st->rr = v[0];
    st->rel_res = rel;
    if (!isfinite(rel))
      st->status = HX_ST_NONFINITE;
    else if (rel < st->tol)
      st->status = HX_ST_CONVERGED;
    else if (st->iter >= st->max_iter)
      st->status = HX_ST_MAXITER;
    st->iter += 1;
  }
}

__global__ void k_ir_correct(double* __restrict__ x, const float* __restrict__ d32, int64_t n,
                             const CgState* st) {
  const double sb = st->bnorm;
  for (int64_t i = gtid(); i < n; i += gstride()) x[i] += sb * (double)d32[i];
}

template <typename TD, typename TS>
__global__ void k_convert(TD* __restrict__ dst, const TS* __restrict__ src, int64_t n) {
  for (int64_t i = gtid(); i < n; i += gstride()) dst[i] = (TD)src[i];
}

}  // namespace

unsigned vec_blocks(int64_t n) {
  const int64_t want = cdiv(std::max<int64_t>(n / 2, 1), VEC_THREADS);
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, 8LL * sm_count()));
}

// vector kernels of fewer CTAs than a wave
bool small_vec(int64_t n) { return vec_blocks(n) < 8u * sm_count(); }

template <typename T>
void launch_cg_init(cudaStream_t s, const T* b, const T* q, const T* minv, T* r, T* p, int64_t n,
                    CgState* st, double* partials) {
  k_cg_init<T><<<vec_blocks(n), VEC_THREADS, 0, s>>>(b, q, minv, r, p, n, st, partials);
  HX_CHECK_LAUNCH();
}

template <typename T>
void launch_cg_update2(cudaStream_t s, T* r, const T* q, const T* minv, int64_t n, CgState* st,
                       double* partials, __nv_bfloat16* ys) {
  launch_dep(small_vec(n), k_cg_update2<T>, vec_blocks(n), VEC_THREADS, 0, s, r, q, minv, n, st,
             partials, ys);
  HX_CHECK_LAUNCH();
}

void launch_fcg_update(cudaStream_t s, double* r, const double* q, const uint8_t* nmask, int64_t n,
                       CgState* st, double* partials, float* r32) {
  launch_dep(small_vec(n), k_fcg_update, vec_blocks(n), VEC_THREADS, 0, s, r, q, nmask, n, st,
             partials, r32);
  HX_CHECK_LAUNCH();
}

template <typename T>
void launch_dinv_bf16(cudaStream_t s, const T* r, const T* minv, __nv_bfloat16* ys, int64_t n) {
  k_dinv_bf16<T><<<vec_blocks(n), VEC_THREADS, 0, s>>>(r, minv, ys, n);
  HX_CHECK_LAUNCH();
}

template <typename T>
void launch_axpy_state(cudaStream_t s, T* dst, const T* x, const T* p, int64_t n,
                       const CgState* st, int when_snap) {
  launch_dep(small_vec(n), k_axpy_state<T>, vec_blocks(n), VEC_THREADS, 0, s, dst, x, p, n, st,
             when_snap);
  HX_CHECK_LAUNCH();
}

#define HX_INST_CG(T)                                                                         \
  template void launch_cg_init<T>(cudaStream_t, const T*, const T*, const T*, T*, T*, int64_t, \
                                  CgState*, double*);                                         \
  template void launch_cg_update2<T>(cudaStream_t, T*, const T*, const T*, int64_t, CgState*,  \
                                     double*, __nv_bfloat16*);                                 \
  template void launch_dinv_bf16<T>(cudaStream_t, const T*, const T*, __nv_bfloat16*,         \
                                    int64_t);                                                  \
  template void launch_axpy_state<T>(cudaStream_t, T*, const T*, const T*, int64_t,            \
                                     const CgState*, int);
HX_INST_CG(double)
HX_INST_CG(float)

void launch_resid_norm(cudaStream_t s, const double* b, const double* q, int64_t n, CgState* st,
                       double* partials, double* out2) {
  k_resid_norm<<<vec_blocks(n), VEC_THREADS, 0, s>>>(b, q, n, st, partials, out2);
  HX_CHECK_LAUNCH();
}

template <typename T>
void launch_mask_rhs(cudaStream_t s, const double* f, const T* minv, double* b, int64_t n) {
  k_mask_rhs<T><<<vec_blocks(n), VEC_THREADS, 0, s>>>(f, minv, b, n);
  HX_CHECK_LAUNCH();
}
template void launch_mask_rhs<double>(cudaStream_t, const double*, const double*, double*,
                                      int64_t);
template void launch_mask_rhs<float>(cudaStream_t, const double*, const float*, double*, int64_t);

void launch_dot(cudaStream_t s, const double* a, const double* b, int64_t n, CgState* st,
                double* partials, double* out) {
  k_dot<<<vec_blocks(n), VEC_THREADS, 0, s>>>(a, b, n, st, partials, out);
  HX_CHECK_LAUNCH();
}

void launch_ir_residual(cudaStream_t s, const double* b, const double* q, float* r32, int64_t n,
                        CgState* st, double* partials) {
  k_ir_residual<<<vec_blocks(n), VEC_THREADS, 0, s>>>(b, q, r32, n, st, partials);
  HX_CHECK_LAUNCH();
}

void launch_ir_correct(cudaStream_t s, double* x, const float* d32, int64_t n,
                       const CgState* st) {
  k_ir_correct<<<vec_blocks(n), VEC_THREADS, 0, s>>>(x, d32, n, st);
  HX_CHECK_LAUNCH();
}

template <typename TD, typename TS>
void launch_convert(cudaStream_t s, TD* dst, const TS* src, int64_t n) {
  k_convert<TD, TS><<<vec_blocks(n), VEC_THREADS, 0, s>>>(dst, src, n);
  HX_CHECK_LAUNCH();
}
template void launch_convert<float, double>(cudaStream_t, float*, const double*, int64_t);
template void launch_convert<double, float>(cudaStream_t, double*, const float*, int64_t);
template void launch_convert<double, double>(cudaStream_t, double*, const double*, int64_t);

__global__ void k_sub(double* __restrict__ r, const double* __restrict__ a,
                      const double* __restrict__ b, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    r[i] = a[i] - b[i];
}
void launch_axpby(cudaStream_t s, double* r, const double* a, const double* b, int64_t n) {
  k_sub<<<vec_blocks(n), VEC_THREADS, 0, s>>>(r, a, b, n);
  HX_CHECK_LAUNCH();
}

// Device-side pruning of the reference's solve entry (src/Solvers/Solver.jl:
// 60-91 with src/Mesh/MeshPruner.jl:18-112): element factor E * density
// where density >= thr (GPUSolver.jl:128,147), else 0; nodes left without
// stiffness are then held at 0 by the node mask, which is what the
// reference's prune-solve-reconstruct returns for them.
__global__ void k_threshold_factor(const float* __restrict__ dens, float thr, float E,
                                   double* __restrict__ fac, int64_t n) {
  for (int64_t e = gtid(); e < n; e += gstride()) {
    const float d = dens[e];
    fac[e] = d >= thr ? (double)(E * d) : 0.0;
  }
}

// Free-DOF bits per node from the reference's bc_indicator (nN x 3 Float32,
// column-major, > 0 = fixed; src/Core/Boundary.jl:135-160).
__global__ void k_bc_bits(const float* __restrict__ bc, uint8_t* __restrict__ free_bits,
                          int64_t nn) {
  for (int64_t i = gtid(); i < nn; i += gstride()) {
    unsigned m = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (!(bc[d * nn + i] > 0.0f)) m |= 1u << d;
    free_bits[i] = (uint8_t)m;
  }
}

void launch_threshold_factor(cudaStream_t s, const float* dens, float thr, float E, double* fac,
                             int64_t n) {
  k_threshold_factor<<<vec_blocks(n), VEC_THREADS, 0, s>>>(dens, thr, E, fac, n);
  HX_CHECK_LAUNCH();
}

void launch_bc_bits(cudaStream_t s, const float* bc, uint8_t* free_bits, int64_t nn) {
  k_bc_bits<<<vec_blocks(nn), VEC_THREADS, 0, s>>>(bc, free_bits, nn);
  HX_CHECK_LAUNCH();
}

void launch_fill_zero(cudaStream_t s, void* p, size_t bytes) {
  HX_CUDA(cudaMemsetAsync(p, 0, bytes, s));
}

}  // namespace hx
