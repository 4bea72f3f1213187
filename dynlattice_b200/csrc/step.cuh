// Device code of one explicit step, shared by the ahead-of-time build
// (kernels.cu, nvcc) and the runtime-compiled elastoplastic kernels (NVRTC,
// jit.cpp); contains no host code and no standard headers.
//
// One explicit step (LeapFrogModule::solve, LeapFrogModule.cpp:44-84, with
// ExplicitModule::getForce/getAcce/updateVec, ExplicitModule.cpp:339-419) is
// two phases over HBM-resident structure-of-arrays data:
//   element phase: per element, gather the two node states, evaluate the rod
//     kinematics, strains, stress resultants (elastic or cutting-plane return
//     map with history commit) and write the two end-force vectors;
//   node phase: per node, sum its incident end forces in a fixed order (CSR),
//     add loads, solve the node-block mass (translational scalar, rotational
//     R P D P^T R^T) with acceleration constraints, and update v, x and the
//     rotation quaternion by the exponential map.
// The persistent kernel runs many steps in one cooperative launch with a
// bounded grid barrier between the phases; k_element/k_node launch one phase
// each (stream mode).  Kernels are templated on the element precision T and on
// the yield-function policy Y.
#pragma once

#include "contact.cuh"
#include "devtypes.cuh"
#include "rodkin.cuh"

namespace dl {

constexpr double kDblEpsilon = 2.220446049250313e-16;  // DBL_EPSILON

// Gauss points/weights of Gauss1..Gauss3 on [-1, 1] (ascending)
__constant__ double c_gxi[3][3] = {{0.0, 0.0, 0.0},
                                   {-0.57735026918962576451, 0.57735026918962576451, 0.0},
                                   {-0.77459666924148337704, 0.0, 0.77459666924148337704}};
__constant__ double c_gw[3][3] = {{2.0, 0.0, 0.0},
                                  {1.0, 1.0, 0.0},
                                  {0.55555555555555555556, 0.88888888888888888889,
                                   0.55555555555555555556}};

// ---------------------------------------------------------------------------
// expression interpreter (programs from expr.cpp; uniform control flow)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float x_pow(float a, float b) { return powf(a, b); }
__device__ __forceinline__ double x_pow(double a, double b) { return pow(a, b); }
__device__ __forceinline__ float x_fmod(float a, float b) { return fmodf(a, b); }
__device__ __forceinline__ double x_fmod(double a, double b) { return fmod(a, b); }

template <class T>
__device__ __forceinline__ void run_prog(const DevProg<T> &p, const T *args, T *r) {
  for (int i = 0; i < p.n_ops; ++i) {
    const ExprOp o = p.ops[i];
    const T a = r[o.a], b = r[o.b], c = r[o.c];
    T v;
    switch (o.op) {
      case XO_CONST: v = p.consts[o.a | (o.b << 8)]; break;
      case XO_ARG: v = args[o.a]; break;
      case XO_ADD: v = a + b; break;
      case XO_SUB: v = a - b; break;
      case XO_MUL: v = a * b; break;
      case XO_DIV: v = a / b; break;
      case XO_POW: v = x_pow(a, b); break;
      case XO_SQUARE: v = a * a; break;
      case XO_NEG: v = -a; break;
      case XO_ABS: v = fabs(a); break;
      case XO_SQRT: v = sqrt(a); break;
      case XO_EXP: v = exp(a); break;
      case XO_LOG: v = log(a); break;
      case XO_SIN: v = sin(a); break;
      case XO_COS: v = cos(a); break;
      case XO_TAN: v = tan(a); break;
      case XO_ATAN: v = atan(a); break;
      case XO_FLOOR: v = floor(a); break;
      case XO_CEIL: v = ceil(a); break;
      case XO_SIGN: v = T((a > T(0)) - (a < T(0))); break;
      case XO_MIN: v = a < b ? a : b; break;
      case XO_MAX: v = a > b ? a : b; break;
      case XO_MOD: v = x_fmod(a, b); break;
      case XO_LT: v = a < b ? T(1) : T(0); break;
      case XO_LE: v = a <= b ? T(1) : T(0); break;
      case XO_GT: v = a > b ? T(1) : T(0); break;
      case XO_GE: v = a >= b ? T(1) : T(0); break;
      case XO_EQ: v = a == b ? T(1) : T(0); break;
      case XO_NE: v = a != b ? T(1) : T(0); break;
      case XO_AND: v = (a != T(0) && b != T(0)) ? T(1) : T(0); break;
      case XO_OR: v = (a != T(0) || b != T(0)) ? T(1) : T(0); break;
      case XO_NOT: v = a == T(0) ? T(1) : T(0); break;
      case XO_SELECT: v = a != T(0) ? b : c; break;
      default: v = T(0); break;
    }
    r[o.dst] = v;
  }
}


// Yield-function policy of the ahead-of-time build: interprets the compiled
// register program (expr.cpp).  The runtime-compiled build replaces it with
// straight-line code generated from the same expressions (YieldJit).
struct YieldInterp {
  static constexpr bool kPlastic = true;
  static constexpr int kNh = -1;  // hardening count known only at run time
  static constexpr int kMinBlocks = 1;
  static constexpr int kInv = 0, kGradInv = 0;  // values of an element's own variables that prep() and
                                                // prep_grad() compute for f and grad
  static constexpr int kRegs = kMaxExprRegs;
  template <class T>
  __device__ static __forceinline__ void prep(const T *, T *) {}
  template <class T>
  __device__ static __forceinline__ void prep_grad(const T *, T *) {}
  template <class T>
  __device__ static __forceinline__ T f(const DevModel<T> &m, const T *args, const T *, T *regs) {
    run_prog(m.yield, args, regs);
    return regs[m.yield.out0];
  }
  template <class T>
  __device__ static __forceinline__ void grad(const DevModel<T> &m, const T *args, const T *, T *gr, T *regs) {
    run_prog(m.grad, args, regs);
    for (int k = 0; k < 6 + m.nh; ++k) gr[k] = regs[m.grad.outs[k]];
  }
};

// Policy of elastic lattices: no return map is compiled in.
struct ElasticOnly {
  static constexpr bool kPlastic = false;
  static constexpr int kNh = 0;
  static constexpr int kMinBlocks = 2;
  static constexpr int kInv = 0, kGradInv = 0;
  static constexpr int kRegs = 1;
  template <class T>
  __device__ static __forceinline__ void prep(const T *, T *) {}
  template <class T>
  __device__ static __forceinline__ void prep_grad(const T *, T *) {}
  template <class T>
  __device__ static __forceinline__ T f(const DevModel<T> &, const T *, const T *, T *) {
    return T(0);
  }
  template <class T>
  __device__ static __forceinline__ void grad(const DevModel<T> &, const T *, const T *, T *, T *) {}
};

// ---------------------------------------------------------------------------
// loads/stores
// ---------------------------------------------------------------------------
// Node state and end forces written in the other phase of the same persistent
// launch are read with plain (L1-cacheable) loads: the grid barrier's
// gpu-scope acquire makes the other blocks' writes visible, as for a
// cooperative-groups grid synchronisation.
// One node's position or rotation is one 32-byte access where the assembler
// knows it (PTX 8.8; a process may bring an older runtime compiler along).
#if !defined(__CUDACC_VER_MAJOR__) || __CUDACC_VER_MAJOR__ > 12 || (__CUDACC_VER_MAJOR__ == 12 && __CUDACC_VER_MINOR__ >= 9)
__device__ __forceinline__ double4 ld32(const double4 *p) {
  double4 v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st32(double4 *p, double x, double y, double z, double w) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x), "d"(y), "d"(z), "d"(w) : "memory");
}
#else
__device__ __forceinline__ double4 ld32(const double4 *p) { return *p; }
__device__ __forceinline__ void st32(double4 *p, double x, double y, double z, double w) {
  *p = make_double4(x, y, z, w);
}
#endif
__device__ __forceinline__ Q4<double> ldq(const double4 *p) {
  const double4 v = ld32(p);
  return Q4<double>{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ V3<double> ldx(const double4 *p) {
  const double4 v = ld32(p);
  return V3<double>{v.x, v.y, v.z};
}
// A record in global memory goes through the read-only path (NC); one that may
// lie in shared memory does not.
template <bool NC, class V>
__device__ __forceinline__ V rec_get(const V *p) {
  if constexpr (NC) return __ldg(p);
  else return *p;
}
// scalars [S, S + N) of a record whose first vector is at r (vectors 32 apart)
template <int S, int N, bool NC = true>
__device__ __forceinline__ void rec_load(const float4 *r, float *o) {
#pragma unroll
  for (int v = S / 4; v <= (S + N - 1) / 4; ++v) {
    const float4 q = rec_get<NC>(r + v * 32);
    const float c[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (v * 4 + k >= S && v * 4 + k < S + N) o[v * 4 + k - S] = c[k];
  }
}
template <int S, int N, bool NC = true>
__device__ __forceinline__ void rec_load(const double2 *r, double *o) {
#pragma unroll
  for (int v = S / 2; v <= (S + N - 1) / 2; ++v) {
    const double2 q = rec_get<NC>(r + v * 32);
    if (v * 2 >= S) o[v * 2 - S] = q.x;
    if (v * 2 + 1 < S + N) o[v * 2 + 1 - S] = q.y;
  }
}
template <bool NC = true, class V>
__device__ __forceinline__ int4 rec_ints(const V *r) {
  return rec_get<NC>(reinterpret_cast<const int4 *>(r));
}
// a double stored over the record's scalars from v[0] on
__device__ __forceinline__ double rec_double(const float *v) {
  return __hiloint2double(__float_as_int(v[1]), __float_as_int(v[0]));
}
__device__ __forceinline__ double rec_double(const double *v) { return v[0]; }
__device__ __forceinline__ Q4<double> toq(float4 v) { return Q4<double>{v.x, v.y, v.z, v.w}; }
__device__ __forceinline__ Q4<double> toq(double4 v) { return Q4<double>{v.x, v.y, v.z, v.w}; }

template <class T>
struct Pair {
  using type = double2;
};
template <>
struct Pair<float> {
  using type = float2;
};
// one end-force record (6 values) into its node-ordered slot
__device__ __forceinline__ void store_end(float *p, const float *f) {
  float2 *q = reinterpret_cast<float2 *>(p);
  q[0] = make_float2(f[0], f[1]);
  q[1] = make_float2(f[2], f[3]);
  q[2] = make_float2(f[4], f[5]);
}
__device__ __forceinline__ void store_end(double *p, const double *f) {
  double2 *q = reinterpret_cast<double2 *>(p);
  q[0] = make_double2(f[0], f[1]);
  q[1] = make_double2(f[2], f[3]);
  q[2] = make_double2(f[4], f[5]);
}
__device__ __forceinline__ void load_end(const float *p, double f[6]) {
  const float2 *q = reinterpret_cast<const float2 *>(p);
  const float2 a = q[0], b = q[1], c = q[2];
  f[0] += a.x; f[1] += a.y; f[2] += b.x; f[3] += b.y; f[4] += c.x; f[5] += c.y;
}
__device__ __forceinline__ void load_end(const double *p, double f[6]) {
  const double2 *q = reinterpret_cast<const double2 *>(p);
  const double2 a = q[0], b = q[1], c = q[2];
  f[0] += a.x; f[1] += a.y; f[2] += b.x; f[3] += b.y; f[4] += c.x; f[5] += c.y;
}

// Sum of the end forces in slots [i0, i1), in their order: the loads of R slots
// (beyond the last one: the last again) are issued before the first is used, so
// that a node waits for memory once per R slots and not once per slot.
template <int R, class T>
__device__ __forceinline__ void sum_ends(const T *ef, int i0, int i1, double f[6]) {
  using V = typename Pair<T>::type;
  for (int i = i0; i < i1; i += R) {
    V r[R][3];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const V *q = reinterpret_cast<const V *>(ef + static_cast<size_t>(i + k < i1 ? i + k : i1 - 1) * 6);
      r[k][0] = q[0];
      r[k][1] = q[1];
      r[k][2] = q[2];
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const bool in = i + k < i1;
      f[0] += in ? double(r[k][0].x) : 0.0;
      f[1] += in ? double(r[k][0].y) : 0.0;
      f[2] += in ? double(r[k][1].x) : 0.0;
      f[3] += in ? double(r[k][1].y) : 0.0;
      f[4] += in ? double(r[k][2].x) : 0.0;
      f[5] += in ? double(r[k][2].y) : 0.0;
    }
  }
}

template <class T>
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double s_part[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) s_part[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x < 32) {
    r = (threadIdx.x < (blockDim.x + 31) / 32) ? s_part[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  return r;  // valid in thread 0
}

// ---------------------------------------------------------------------------
// element phase
// ---------------------------------------------------------------------------
struct ElemEnergy {
  double pot = 0.0, diss = 0.0;
};

// Out-of-line paths that plain runs do not take (contact, plates, group
// output): kept out of the step kernels' register budget.

struct NodeExtra {
  double f[3];
  double energy;
};

// rod--rod contact force of this step (then cleared for the next one) and
// the rigid plates' node--plane penalty
template <class T>
__device__ __noinline__ NodeExtra node_contact(const DevModel<T> &m, int n, int64_t step, double xx, double xy,
                                               double xz, bool energy, bool last, bool walk) {
  NodeExtra o{{0.0, 0.0, 0.0}, 0.0};
  // the node's ends of closed pairs, in the index's fixed order; walked only
  // when a pair of the node closed in this step (walk: its stamp)
  if (walk && m.c_ptr)
    for (uint32_t i = m.c_ptr[n]; i < m.c_ptr[n + 1]; ++i) {
      const int v = m.c_ent[i];
      if (!m.pclosed[v >> 2]) continue;
      const double *f = m.pforce + static_cast<size_t>(v >> 2) * 12 + (v & 3) * 3;
      o.f[0] += f[0];
      o.f[1] += f[1];
      o.f[2] += f[2];
    }
  if (walk && m.j_ptr)
    for (uint32_t i = m.j_ptr[n]; i < m.j_ptr[n + 1]; ++i) {
      const int v = m.j_ent[i];
      if (!m.jclosed[v >> 1]) continue;
      const double *f = m.jforce + static_cast<size_t>(v >> 1) * 6 + (v & 1) * 3;
      o.f[0] += f[0];
      o.f[1] += f[1];
      o.f[2] += f[2];
    }
  for (int pl = 0; pl < m.n_plates; ++pl) {
    const double tk = m.t0 + static_cast<double>(step - m.tstep0) * m.dt;
    const double g = (xx - (m.plate_p0[pl][0] + m.plate_v[pl][0] * tk)) * m.plate_n[pl][0] +
                     (xy - (m.plate_p0[pl][1] + m.plate_v[pl][1] * tk)) * m.plate_n[pl][1] +
                     (xz - (m.plate_p0[pl][2] + m.plate_v[pl][2] * tk)) * m.plate_n[pl][2] - m.c_radius;
    if (g < 0.0) {
      const double kg = m.plate_k[pl] * g;
      for (int c2 = 0; c2 < 3; ++c2) o.f[c2] += kg * m.plate_n[pl][c2];
      if (energy) o.energy += 0.5 * kg * g;
      if (last)
        for (int c2 = 0; c2 < 3; ++c2) atomicAdd(m.plate_force + pl * 3 + c2, kg * m.plate_n[pl][c2]);
    }
  }
  return o;
}

template <class T>
__device__ __noinline__ void store_fint_last(const DevModel<T> &m, int n, double f0, double f1, double f2, double f3,
                                             double f4, double f5) {
  const int N = m.N;
  m.fint_last[n] = f0;
  m.fint_last[N + n] = f1;
  m.fint_last[2 * N + n] = f2;
  m.fint_last[3 * N + n] = f3;
  m.fint_last[4 * N + n] = f4;
  m.fint_last[5 * N + n] = f5;
}

// The element's variables of yield expressions (radius, area) and what the
// yield function makes of them alone, the same at all its points.
template <class T, class Y>
struct YieldElem {
  T ec[2];
  T inv[Y::kInv > 0 ? Y::kInv : 1];
};
template <class T, class Y>
__device__ __forceinline__ void yield_elem(const DevModel<T> &m, T radius, T area, YieldElem<T, Y> &y) {
  y.ec[0] = radius;
  y.ec[1] = area;
  if (Y::kInv > 0) {
    constexpr int nh = Y::kNh > 0 ? Y::kNh : 0;
    T a[8 + nh];
    a[6 + nh] = y.ec[0];
    a[7 + nh] = y.ec[1];
    Y::prep(a, y.inv);
  }
}

// The plastic flow of one Gauss point whose trial stress is outside the yield
// surface: the cutting-plane iterations of ElastoPlasticRodMaterial::getStress
// (ElastoPlasticRodMaterial.cpp:198-269) from the yield value fv of the trial
// stress on.  Inline: as a call (the points that flow are few) its saved
// registers cost the points that stay elastic more, 48.0 against 40.8 us per
// step on the 20^3 BCC lattice in FP64.
template <class T, int NHA>
struct FlowState {
  T ep[6], al[NHA], sig[6];
  T dflow;
  int it;
};
template <class T, class Y, bool X>
__device__ __forceinline__ void plastic_flow(const DevModel<T> &m, const T *eps, const T *Cd, const YieldElem<T, Y> &ye,
                                          T fv, int it_imposed,
                                          FlowState<T, Y::kNh == 0 ? 1 : (Y::kNh > 0 ? Y::kNh : 7)> &s) {
  constexpr int NHC = Y::kNh;
  const int nh = NHC >= 0 ? NHC : m.nh;
  constexpr int NHMAX = NHC >= 0 ? NHC : 7;
  T ep[6], al[NHMAX > 0 ? NHMAX : 1], sig[6], C[6], e6[6], args[16];
  T regs[Y::kRegs];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    ep[k] = s.ep[k];
    sig[k] = s.sig[k];
    C[k] = Cd[k];
    e6[k] = eps[k];
  }
#pragma unroll
  for (int a = 0; a < NHMAX; ++a)
    if (a < nh) al[a] = s.al[a];
  args[6 + nh] = ye.ec[0];
  args[7 + nh] = ye.ec[1];
  auto set_args = [&]() {
#pragma unroll
    for (int a = 0; a < NHMAX; ++a) {
      if (a >= nh) break;
      T h = T(0);
#pragma unroll
      for (int b = 0; b < NHMAX; ++b)
        if (b < nh) h = fma_rn(m.H[a][b], al[b], h);
      args[6 + a] = -h;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) args[k] = sig[k];
  };
  set_args();
  T ginv[Y::kGradInv > 0 ? Y::kGradInv : 1];
  Y::prep_grad(args, ginv);
  T dflow = T(0);
  int it = 0;
  for (;;) {
    T gr[13];
    Y::grad(m, args, ginv, gr, regs);
    T den = T(0);
#pragma unroll
    for (int k = 0; k < 6; ++k) den = fma_rn(mul_rn(gr[k], C[k]), gr[k], den);
#pragma unroll
    for (int a = 0; a < NHMAX; ++a) {
      if (a >= nh) break;
      T h = T(0);
#pragma unroll
      for (int b = 0; b < NHMAX; ++b)
        if (b < nh) h = fma_rn(m.H[a][b], gr[6 + b], h);
      den = fma_rn(gr[6 + a], h, den);
    }
    const T ddf = fv / den;
#pragma unroll
    for (int k = 0; k < 6; ++k) ep[k] = fma_rn(ddf, gr[k], ep[k]);
#pragma unroll
    for (int a = 0; a < NHMAX; ++a)
      if (a < nh) al[a] = fma_rn(ddf, gr[6 + a], al[a]);
    dflow += ddf;
    ++it;
#pragma unroll
    for (int k = 0; k < 6; ++k) sig[k] = C[k] * (e6[k] - ep[k]);
    set_args();
    fv = Y::f(m, args, ye.inv, regs);
    if (!(it < m.max_iter)) {
      atomicOr(m.err, 0x1u);
      break;
    }
    if (X && it_imposed >= 0 ? it >= it_imposed : fv < m.prec) break;
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    s.ep[k] = ep[k];
    s.sig[k] = sig[k];
  }
#pragma unroll
  for (int a = 0; a < NHMAX; ++a)
    if (a < nh) s.al[a] = al[a];
  s.dflow = dflow;
  s.it = it;
}

// Stress resultants at one Gauss point: ElasticRodMaterial::getStress
// (ElasticRodMaterial.cpp:369-373) or the cutting-plane return map of
// ElastoPlasticRodMaterial::getStress (ElastoPlasticRodMaterial.cpp:198-269)
// followed by the commit of ElastoPlasticRodMaterial::applyDeform (:271-307).
// History modes of the material update: HM_COMMIT (explicit step: return map,
// history committed in place; with commit = false the elastic predictor
// only), HM_TRIAL (return map from the committed history, nothing written)
// and HM_STORE (return map, the resulting history written to HistOut: the
// predictor-corrector's trial that is committed once its step is accepted).
enum { HM_COMMIT = 0, HM_TRIAL = 1, HM_STORE = 2 };
template <class T>
struct HistOut {
  T *hist, *epsc;  // layouts of DevModel::hist, epsc
  double *ediss;
};

// A point's history record at p (vectors 32 apart); NHC: the hardening count
// where it is known at compile time (else -1, and nh).
template <class T, int NHC>
__device__ __forceinline__ void hist_load(const T *p, int nh, T ep[6], T *al) {
  constexpr int n = Vec16<T>::n, cnt = 6 + (NHC >= 0 ? NHC : 7);
#pragma unroll
  for (int v = 0; v < (cnt + n - 1) / n; ++v) {
    if (NHC < 0 && v * n >= 6 + nh) break;
    const auto q = *reinterpret_cast<const typename Vec16<T>::type *>(p + v * 32 * n);
    const T *c = reinterpret_cast<const T *>(&q);
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const int i = v * n + k;
      if (i < 6) ep[i] = c[k];
      else if (i < cnt && i - 6 < nh) al[i - 6] = c[k];
    }
  }
}
template <class T, int NHC>
__device__ __forceinline__ void hist_store(T *p, int nh, const T ep[6], const T *al) {
  constexpr int n = Vec16<T>::n, cnt = 6 + (NHC >= 0 ? NHC : 7);
#pragma unroll
  for (int v = 0; v < (cnt + n - 1) / n; ++v) {
    if (NHC < 0 && v * n >= 6 + nh) break;
    typename Vec16<T>::type q;
    T *c = reinterpret_cast<T *>(&q);
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const int i = v * n + k;
      c[k] = i < 6 ? ep[i < 6 ? i : 0] : (i < cnt && i - 6 < nh ? al[i - 6] : T(0));
    }
    *reinterpret_cast<typename Vec16<T>::type *>(p + v * 32 * n) = q;
  }
}
// a point's committed plastic strain and hardening parameters
template <class T, class Y>
struct HistIn {
  T ep[6], al[Y::kNh == 0 ? 1 : (Y::kNh > 0 ? Y::kNh : 7)];
};
template <class T, class Y>
__device__ __forceinline__ void hist_in(const DevModel<T> &m, int e, int g, HistIn<T, Y> &h) {
  if (!Y::kPlastic || !m.plastic) return;
  hist_load<T, Y::kNh>(m.hist + hist_ix<T>(m.G, m.hs, e, g, 0), Y::kNh >= 0 ? Y::kNh : m.nh, h.ep, h.al);
}
__device__ __forceinline__ void epsc_store(float *p, const float eps[6]) {
  float2 *q = reinterpret_cast<float2 *>(p);
  q[0] = make_float2(eps[0], eps[1]);
  q[32] = make_float2(eps[2], eps[3]);
  q[64] = make_float2(eps[4], eps[5]);
}
__device__ __forceinline__ void epsc_store(double *p, const double eps[6]) {
  double2 *q = reinterpret_cast<double2 *>(p);
  q[0] = make_double2(eps[0], eps[1]);
  q[32] = make_double2(eps[2], eps[3]);
  q[64] = make_double2(eps[4], eps[5]);
}

// EN: every step of the launch reports energies (known at compile time):
// the point's dissipated energy is then loaded before the iterations, so
// that its latency overlaps them instead of ending the element's chain.
template <class T, class Y, bool X, int HM = HM_COMMIT, bool EN = false>
__device__ __forceinline__ void material(const DevModel<T> &m, int e, int g, const T eps[6],
                                         const T Cd[6], const YieldElem<T, Y> &ye, const HistIn<T, Y> &hi,
                                         T sig[6], bool commit, bool energy,
                                         double wgt, ElemEnergy &en, int64_t tslot = -1,
                                         const HistOut<T> *ho = nullptr, int64_t bslot = -1) {
  const int E = m.E;
  if (!Y::kPlastic || !m.plastic) {
#pragma unroll
    for (int k = 0; k < 6; ++k) sig[k] = Cd[k] * eps[k];
    if (energy) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < 6; ++k) s += double(eps[k]) * double(sig[k]);
      en.pot += wgt * 0.5 * s;
    }
    return;
  }
  // hardening count: a compile-time constant in the specialised kernels, so
  // that all history arrays below live in registers
  constexpr int NHC = Y::kNh;
  const int nh = NHC >= 0 ? NHC : m.nh;
  constexpr int NHMAX = NHC >= 0 ? NHC : 7;
  T ep[6], ep0[6], al[NHMAX > 0 ? NHMAX : 1];
#pragma unroll
  for (int k = 0; k < 6; ++k) ep[k] = ep0[k] = hi.ep[k];
#pragma unroll
  for (int a = 0; a < NHMAX; ++a)
    if (a < nh) al[a] = hi.al[a];
  T args[16];
  args[6 + nh] = ye.ec[0];
  args[7 + nh] = ye.ec[1];
  constexpr bool ed_early = HM == HM_COMMIT && EN;
  const double ed_in = ed_early ? m.ediss[g * E + e] : 0.0;
  T regs[Y::kRegs];
  T dflow = T(0);
  int it = 0;
  // branch tape of a differentiated run: the iteration count to impose
  size_t bidx = 0;
  int it_imposed = -1;
  if (X && HM == HM_COMMIT && m.br && bslot >= 0) {
    bidx = (static_cast<size_t>(bslot) * m.G + g) * E + e;
    if (m.br_mode == 2) it_imposed = m.br[bidx];
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) sig[k] = Cd[k] * (eps[k] - ep[k]);
  if (HM != HM_COMMIT || commit) {
#pragma unroll
    for (int a = 0; a < NHMAX; ++a) {
      if (a >= nh) break;
      T s = T(0);
#pragma unroll
      for (int b = 0; b < NHMAX; ++b)
        if (b < nh) s = fma_rn(m.H[a][b], al[b], s);
      args[6 + a] = -s;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) args[k] = sig[k];
    const T fv = Y::f(m, args, ye.inv, regs);
    if (!(X && it_imposed >= 0 ? it_imposed <= 0 : fv < m.prec)) {
      FlowState<T, Y::kNh == 0 ? 1 : (Y::kNh > 0 ? Y::kNh : 7)> fs;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        fs.ep[k] = ep[k];
        fs.sig[k] = sig[k];
      }
#pragma unroll
      for (int a = 0; a < NHMAX; ++a)
        if (a < nh) fs.al[a] = al[a];
      plastic_flow<T, Y, X>(m, eps, Cd, ye, fv, it_imposed, fs);
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        ep[k] = fs.ep[k];
        sig[k] = fs.sig[k];
      }
#pragma unroll
      for (int a = 0; a < NHMAX; ++a)
        if (a < nh) al[a] = fs.al[a];
      dflow = fs.dflow;
      it = fs.it;
    }
  }
  if (HM == HM_COMMIT && !commit) return;
  if (HM == HM_TRIAL) return;
  if (X && HM == HM_COMMIT && m.br && bslot >= 0 && m.br_mode == 1) m.br[bidx] = static_cast<uint8_t>(it < 255 ? it : 255);
  // applyDeform: dissipation with the previous committed total strain
  double dd = 0.0;
  if (fabs(double(dflow)) > kDblEpsilon) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const T eold = m.epsc[epsc_ix(m.G, e, g, k)];
      const double so = double(Cd[k]) * double(eold - ep0[k]);
      dd += (so + double(sig[k])) / 2.0 * double(ep[k] - ep0[k]);
    }
    if (HM == HM_COMMIT) {
      if (ed_early) m.ediss[g * E + e] = ed_in + dd;
      else m.ediss[g * E + e] += dd;
    }
  }
  const size_t hx = hist_ix<T>(m.G, m.hs, e, g, 0), ex = epsc_ix(m.G, e, g, 0);
  if (HM == HM_STORE) {
    const double ed = m.ediss[g * E + e] + dd;
    ho->ediss[g * E + e] = ed;
    hist_store<T, NHC>(ho->hist + hx, nh, ep, al);
    epsc_store(ho->epsc + ex, eps);
    if (energy) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < 6; ++k) s += double(eps[k] - ep[k]) * double(sig[k]);
      en.pot += wgt * 0.5 * s;
      en.diss += wgt * ed;
    }
    return;
  }
  if (it > 0) hist_store<T, NHC>(m.hist + hx, nh, ep, al);
  epsc_store(m.epsc + ex, eps);
  if (X && m.tp_hist && tslot >= 0) {  // adjoint recomputation: history after this step
    const size_t E32 = static_cast<size_t>(tiles32(E)) * tslot;
    hist_store<T, NHC>(m.tp_hist + E32 * m.G * m.hs + hx, nh, ep, al);
    epsc_store(m.tp_epsc + E32 * m.G * 6 + ex, eps);
  }
  if (energy) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) s += double(eps[k] - ep[k]) * double(sig[k]);
    en.pot += wgt * 0.5 * s;
    en.diss += wgt * (ed_early ? ed_in + dd : m.ediss[g * E + e]);
  }
}

// A plastic point's step where it stays elastic: its stress, committed strain and
// energies.  False (nothing done) where the trial stress lies outside the yield
// surface, or a differentiated run imposes iterations.
template <class T, class Y, bool X, bool EN>
__device__ __forceinline__ bool material_elastic(const DevModel<T> &m, int e, int g, const T eps[6], const T Cd[6],
                                                 const YieldElem<T, Y> &ye, const HistIn<T, Y> &hi, T sig[6],
                                                 bool energy, double wgt, ElemEnergy &en, int64_t tslot,
                                                 int64_t bslot) {
  constexpr int NHC = Y::kNh, NHMAX = NHC >= 0 ? NHC : 7;
  const int nh = NHC >= 0 ? NHC : m.nh;
  T args[16], regs[Y::kRegs];
  args[6 + nh] = ye.ec[0];
  args[7 + nh] = ye.ec[1];
#pragma unroll
  for (int k = 0; k < 6; ++k) args[k] = sig[k] = Cd[k] * (eps[k] - hi.ep[k]);
#pragma unroll
  for (int a = 0; a < NHMAX; ++a) {
    if (a >= nh) break;
    T s = T(0);
#pragma unroll
    for (int b = 0; b < NHMAX; ++b)
      if (b < nh) s = fma_rn(m.H[a][b], hi.al[b], s);
    args[6 + a] = -s;
  }
  const T fv = Y::f(m, args, ye.inv, regs);
  bool stays = fv < m.prec;
  if (X && m.br && bslot >= 0) {
    uint8_t *const br = m.br + (static_cast<size_t>(bslot) * m.G + g) * m.E + e;
    if (m.br_mode == 2) stays = *br == 0;
    else if (m.br_mode == 1 && stays) *br = 0;
  }
  if (!stays) return false;
  const size_t ex = epsc_ix(m.G, e, g, 0);
  epsc_store(m.epsc + ex, eps);
  if (X && m.tp_hist && tslot >= 0) {  // adjoint recomputation: history after this step
    const size_t E32 = static_cast<size_t>(tiles32(m.E)) * tslot;
    hist_store<T, NHC>(m.tp_hist + E32 * m.G * m.hs + hist_ix<T>(m.G, m.hs, e, g, 0), nh, hi.ep, hi.al);
    epsc_store(m.tp_epsc + E32 * m.G * 6 + ex, eps);
  }
  if (energy) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) s += double(eps[k] - hi.ep[k]) * double(sig[k]);
    en.pot += wgt * 0.5 * s;
    en.diss += wgt * m.ediss[g * m.E + e];
  }
  return true;
}

// Internal force of one element (SpecialCosseratRodModel::assemble_,
// SpecialCosseratRodModel.cpp:899-949, with Line3D::getXi, Line3D.cpp:141-162):
//   f_n += w [ N'_n n ; N'_n m - N_n phi' x n ],  n = Lambda sigma_n, m = Lambda sigma_m,
// summed over the Gauss points in the frame of Lambda_r and turned to space
// once: with n_g = R(xi phi/2) sigma_n and m_g likewise (Lambda = Lambda_r
// R(xi phi/2), phi' = Lambda_r d) the element needs S0 = sum W n_g, S1 = sum W xi n_g
// and SM = sum W m_g only:
//   f_J = -f_I = Lambda_r S0/2,
//   moments  Lambda_r (P - Q) at J and -Lambda_r (P + Q) at I,
//   P = SM/2 - L0/4 d x S1,  Q = L0/4 d x S0.
// Symmetric points +-xi share one matrix R(e) - 1, e = exp(-xi phi/2): their
// rotations are each other's transpose.

// R(q) - 1, row-major: a small rotation keeps its relative precision.
template <class T>
__device__ __forceinline__ void qmat_less_one(const Q4<T> &q, T m[3][3]) {
  const T x2 = q.x + q.x, y2 = q.y + q.y, z2 = q.z + q.z;
  const T wx = mul_rn(q.w, x2), wy = mul_rn(q.w, y2), wz = mul_rn(q.w, z2);
  const T xx = mul_rn(q.x, x2), zz = mul_rn(q.z, z2);
  m[0][0] = -fma_rn(q.y, y2, zz);
  m[1][1] = -(xx + zz);
  m[2][2] = -fma_rn(q.y, y2, xx);
  m[0][1] = fma_rn(q.x, y2, -wz);
  m[1][0] = fma_rn(q.x, y2, wz);
  m[0][2] = fma_rn(q.x, z2, wy);
  m[2][0] = fma_rn(q.x, z2, -wy);
  m[1][2] = fma_rn(q.y, z2, -wx);
  m[2][1] = fma_rn(q.y, z2, wx);
}
// v + m v and v + m^T v
template <class T>
__device__ __forceinline__ V3<T> add_mat(const T m[3][3], const V3<T> &v) {
  return V3<T>{v.x + fma_rn(m[0][2], v.z, fma_rn(m[0][1], v.y, mul_rn(m[0][0], v.x))),
               v.y + fma_rn(m[1][2], v.z, fma_rn(m[1][1], v.y, mul_rn(m[1][0], v.x))),
               v.z + fma_rn(m[2][2], v.z, fma_rn(m[2][1], v.y, mul_rn(m[2][0], v.x)))};
}
template <class T>
__device__ __forceinline__ V3<T> add_mat_t(const T m[3][3], const V3<T> &v) {
  return V3<T>{v.x + fma_rn(m[2][0], v.z, fma_rn(m[1][0], v.y, mul_rn(m[0][0], v.x))),
               v.y + fma_rn(m[2][1], v.z, fma_rn(m[1][1], v.y, mul_rn(m[0][1], v.x))),
               v.z + fma_rn(m[2][2], v.z, fma_rn(m[1][2], v.y, mul_rn(m[0][2], v.x)))};
}
// R(e) - 1 of the Gauss point g (m: of the largest abscissa): as it is for
// xi > 0, transposed for xi < 0, zero for xi = 0.
template <class T>
__device__ __forceinline__ void gp_turn(const T m[3][3], T xi, T r[3][3]) {
  const bool pos = xi > T(0), neg = xi < T(0);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) r[i][j] = pos ? m[i][j] : (neg ? m[j][i] : T(0));
}

// Gauss point g of an element: strain, stress resultants (with the history
// update of the history mode), the point's n_g and m_g.  kap: the element's
// curvature strain, the same at every point of a two-node element.  FAST: a
// plastic point that stays elastic only (false where it does not).
template <class T, class Y, bool X, int HM, bool EN, bool TURN, bool NC, bool FAST = false>
__device__ __forceinline__ bool gp_local(const DevModel<T> &m, int e, int g, int G,
                                         const typename Vec16<T>::type *rec, const ElemKin<T> &k,
                                         const T turn[3][3], const V3<T> &kap, double L0, const T Cd[6],
                                         const YieldElem<T, Y> &ye, const HistIn<T, Y> &hi, bool commit,
                                         bool energy, ElemEnergy &en, int64_t tslot, const HistOut<T> *ho,
                                         int64_t bslot, V3<T> &ng, V3<T> &mg) {
  T g0[3];
  const T *rg = reinterpret_cast<const T *>(rec);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int sc = ElemRecIx<T>::g0 + 3 * g + q;
    g0[q] = rec_get<NC>(rg + sc / Vec16<T>::n * 32 * Vec16<T>::n + sc % Vec16<T>::n);
  }
  T eps[6] = {k.dme3.x - g0[0], k.dme3.y - g0[1], k.dme3.z - g0[2], kap.x, kap.y, kap.z};
  if (TURN) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
      eps[i] = fma_rn(turn[i][2], k.d.z, fma_rn(turn[i][1], k.d.y, fma_rn(turn[i][0], k.d.x, eps[i])));
  }
  T sig[6];
  const double wgt = c_gw[G - 1][g] * 0.5 * L0;
  if constexpr (FAST) {
    if (!material_elastic<T, Y, X, EN>(m, e, g, eps, Cd, ye, hi, sig, energy, wgt, en, tslot, bslot)) return false;
  } else {
    material<T, Y, X, HM, EN>(m, e, g, eps, Cd, ye, hi, sig, commit, energy, wgt, en, tslot, ho, bslot);
  }
  ng = V3<T>{sig[0], sig[1], sig[2]};
  mg = V3<T>{sig[3], sig[4], sig[5]};
  if (TURN) {
    ng = add_mat_t(turn, ng);
    mg = add_mat_t(turn, mg);
  }
  return true;
}

// The element's end forces from its sums: F at J (and -F at I), moments
// MP - MQ at J and -(MP + MQ) at I.
template <class T>
struct EndForces {
  V3<T> F, MP, MQ;
};
template <class T>
__device__ __forceinline__ EndForces<T> end_forces(const ElemKin<T> &k, double L0, const V3<T> &S0, const V3<T> &S1,
                                                   const V3<T> &SM) {
  const T h = T(0.25 * L0);
  const V3<T> c1 = cross(k.d, S1);
  const V3<T> P{fma_rn(-h, c1.x, T(0.5) * SM.x), fma_rn(-h, c1.y, T(0.5) * SM.y), fma_rn(-h, c1.z, T(0.5) * SM.z)};
  const V3<T> c0 = cross(k.d, S0);
  const V3<T> Q{mul_rn(h, c0.x), mul_rn(h, c0.y), mul_rn(h, c0.z)};
  T r[3][3];
  qmat_less_one(k.qr, r);
  return EndForces<T>{T(0.5) * add_mat(r, S0), add_mat(r, P), add_mat(r, Q)};
}
template <class T>
__device__ __forceinline__ void end_i(const EndForces<T> &f, T o[6]) {
  o[0] = -f.F.x; o[1] = -f.F.y; o[2] = -f.F.z;
  o[3] = -(f.MP.x + f.MQ.x); o[4] = -(f.MP.y + f.MQ.y); o[5] = -(f.MP.z + f.MQ.z);
}
template <class T>
__device__ __forceinline__ void end_j(const EndForces<T> &f, T o[6]) {
  o[0] = f.F.x; o[1] = f.F.y; o[2] = f.F.z;
  o[3] = f.MP.x - f.MQ.x; o[4] = f.MP.y - f.MQ.y; o[5] = f.MP.z - f.MQ.z;
}

// The gathered end states, kinematics and section constants of element e.
template <class T, class Y>
struct ElemPre {
  const typename Vec16<T>::type *rec;  // the element's record
  int2 slot;
  ElemKin<T> k;
  V3<T> kap;  // curvature strain phi/L0 - K0 (one value per two-node element)
  double L0;
  T Cd[6];
  YieldElem<T, Y> ye;
};
// The states of an element's end nodes: from the global arrays...
struct GlobalEnds {
  static constexpr bool kReadOnly = true;
  const double4 *P, *Q;
  template <class T>
  __device__ __forceinline__ const typename Vec16<T>::type *rec(const DevModel<T> &m, int e, int nv) const {
    return m.erec + static_cast<size_t>(e >> 5) * (nv * 32) + (e & 31);
  }
  __device__ __forceinline__ void get(int, int4 c, V3<double> &xi, V3<double> &xj, Q4<double> &Ri,
                                      Q4<double> &Rj) const {
    xi = ldx(P + c.x);
    xj = ldx(P + c.y);
    Ri = ldq(Q + c.x);
    Rj = ldq(Q + c.y);
  }
};
template <class T, class Y, class S>
__device__ __forceinline__ void elem_pre(const DevModel<T> &m, int e, int G, const S &src, ElemPre<T, Y> &p) {
  using Ix = ElemRecIx<T>;
  p.rec = src.template rec<T>(m, e, Ix::vecs(G));
  const int4 c = rec_ints<S::kReadOnly>(p.rec);
  p.slot = make_int2(c.z, c.w);
  V3<double> xi, xj;
  Q4<double> Ri, Rj;
  src.get(e, c, xi, xj, Ri, Rj);
  T qn[8], r[6 + 2 + 3 + 1 + 8 / sizeof(T)];
  rec_load<Ix::qN, 8, S::kReadOnly>(p.rec, qn);
  rec_load<Ix::C, 6 + 2 + 3 + 1 + 8 / int(sizeof(T)), S::kReadOnly>(p.rec, r);
  const double invL0 = rec_double(r + (Ix::invL0 - Ix::C));
  p.k = elem_kin<T>(xi, xj, Ri, Rj, Q4<double>{double(qn[0]), double(qn[1]), double(qn[2]), double(qn[3])},
                    Q4<double>{double(qn[4]), double(qn[5]), double(qn[6]), double(qn[7])}, invL0);
  const T il = T(invL0);
  p.L0 = double(r[Ix::L0 - Ix::C]);
  const T *k0 = r + (Ix::k0 - Ix::C);
  p.kap = V3<T>{fma_rn(p.k.phi.x, il, -k0[0]), fma_rn(p.k.phi.y, il, -k0[1]), fma_rn(p.k.phi.z, il, -k0[2])};
#pragma unroll
  for (int q = 0; q < 6; ++q) p.Cd[q] = r[q];
  if (Y::kPlastic && m.plastic) yield_elem(m, r[Ix::ec - Ix::C], r[Ix::ec - Ix::C + 1], p.ye);
}

// Elements of 3 or 4 nodes: node positions, the reference rotation and the
// local rotation vectors (gathered from P/Q, the node state to use), and per
// Gauss point the strains minus the reference values (in T), with the point's
// weight and shape data.
struct ElemPreN {
  V3<double> x[kMaxElemNodes];
  Q4<double> Lr;
  V3<double> psi[kMaxElemNodes];
};
template <class T>
__device__ __forceinline__ void elem_pre_n(const DevModel<T> &m, int e, const double4 *P, const double4 *Q,
                                           ElemPreN &p) {
  const int E = m.E, n = m.nen;
  Q4<double> L[kMaxElemNodes];
  for (int a = 0; a < n; ++a) {
    const int nd = m.conn_n[a * E + e];
    p.x[a] = ldx(P + nd);
    L[a] = qmul(ldq(Q + nd), toq(m.qN[a * E + e]));
  }
  line_ref(L, n, p.Lr, p.psi);
}
template <class T>
__device__ __forceinline__ GpKinN gp_eps_n(const DevModel<T> &m, int e, int g, const ElemPreN &p, T eps[6],
                                           double &w, double N[kMaxElemNodes], double dN[kMaxElemNodes]) {
  const int E = m.E, n = m.nen;
  const double *sh = m.shp + (static_cast<size_t>(e) * m.G + g) * (n + 1);
  w = sh[0];
  for (int a = 0; a < n; ++a) {
    N[a] = m.Nq[a][g];
    dN[a] = sh[1 + a];
  }
  const GpKinN k = gp_kin_n(p.x, p.Lr, p.psi, n, N, dN);
  const double *s0 = m.s0_n + static_cast<size_t>(g) * 6 * E + e;
  eps[0] = T(k.gme3.x - s0[0]);
  eps[1] = T(k.gme3.y - s0[E]);
  eps[2] = T(k.gme3.z - s0[2 * E]);
  eps[3] = T(k.K.x - s0[3 * E]);
  eps[4] = T(k.K.y - s0[4 * E]);
  eps[5] = T(k.K.z - s0[5 * E]);
  return k;
}

// Internal force of an element of 3 or 4 nodes (SpecialCosseratRodModel::
// getStrains_/assemble_, SpecialCosseratRodModel.cpp:694-744, 899-949, with
// Line3D, Line3D.cpp:117-273): kinematics in FP64 (gp_kin_n), material and
// end forces in T,
//   f_a += w [ N_a' n ; N_a' m - N_a phi' x n ],  n = Lambda sigma_n, m = Lambda sigma_m.
// Out of line, so that the kernels' two-node paths keep their register
// allocation.  P/Q: the node positions and rotations to use.
template <class T, class Y, bool X, int HM>
__device__ __noinline__ void element_force_n(const DevModel<T> &m, int e, bool commit, bool energy,
                                             ElemEnergy &en, int64_t tslot, const double4 *P, const double4 *Q,
                                             const HistOut<T> *ho, int64_t bslot) {
  const int E = m.E, n = m.nen, G = m.G;
  ElemPreN p;
  elem_pre_n(m, e, P, Q, p);
  T Cd[6];
  for (int q = 0; q < 6; ++q) Cd[q] = m.C[q * E + e];
  YieldElem<T, Y> ye;
  if (Y::kPlastic && m.plastic) yield_elem(m, m.ec[e], m.ec[E + e], ye);
  T f[kMaxElemNodes][6];
  for (int a = 0; a < n; ++a)
    for (int q = 0; q < 6; ++q) f[a][q] = T(0);
  for (int g = 0; g < G; ++g) {
    T eps[6];
    double w, N[kMaxElemNodes], dN[kMaxElemNodes];
    const GpKinN k = gp_eps_n(m, e, g, p, eps, w, N, dN);
    T sig[6];
    HistIn<T, Y> hi;
    hist_in(m, e, g, hi);
    material<T, Y, X, HM>(m, e, g, eps, Cd, ye, hi, sig, commit, energy, w, en, tslot, ho, bslot);
    const Q4<T> qg = cvtq<T>(k.L);
    const V3<T> nn = qrot(qg, V3<T>{sig[0], sig[1], sig[2]});
    const V3<T> mm = qrot(qg, V3<T>{sig[3], sig[4], sig[5]});
    const V3<T> pxn = cross(cvt<T>(k.phiP), nn);
    for (int a = 0; a < n; ++a) {
      const T wg = T(w * dN[a]), wn = T(w * N[a]);
      f[a][0] += wg * nn.x;
      f[a][1] += wg * nn.y;
      f[a][2] += wg * nn.z;
      f[a][3] += wg * mm.x - wn * pxn.x;
      f[a][4] += wg * mm.y - wn * pxn.y;
      f[a][5] += wg * mm.z - wn * pxn.z;
    }
  }
  for (int a = 0; a < n; ++a) store_end(m.ef + static_cast<size_t>(m.eslot_n[a * E + e]) * 6, f[a]);
}

// Internal force of one element: the end states, kinematics and the sum of
// its Gauss points' contributions into the two node-ordered end slots.
// HM != HM_COMMIT (predictor-corrector): the node state is read from pos/rot
// and the history is handled as material() describes.
// GC: the Gauss-point count when known at compile time (0: m.G); with a
// constant count the point loop unrolls and the points' independent
// strain/stress chains interleave.
template <class T, class Y, bool X, int HM, int GC, bool EN, bool FAST, class S>
__device__ __forceinline__ bool element_body(const DevModel<T> &m, const S &src, T *efb, int e, bool commit,
                                             bool energy, ElemEnergy &en, int64_t tslot, const HistOut<T> *ho,
                                             int64_t bslot) {
  const int G = GC > 0 ? GC : m.G;
  // FAST: the history early, so that its loads are under way while the kinematics
  // are formed; else where it is used (the registers are short)
  HistIn<T, Y> h0, h1;
  if (FAST && GC > 0) hist_in(m, e, 0, h0);
  if (FAST && GC == 2) hist_in(m, e, 1, h1);
  ElemPre<T, Y> p;
  elem_pre(m, e, G, src, p);
  V3<T> S0, S1, SM;
  if (GC == 1) {
    if (!FAST) hist_in(m, e, 0, h0);
    V3<T> n0, m0;
    if (!gp_local<T, Y, X, HM, EN, false, S::kReadOnly, FAST>(m, e, 0, 1, p.rec, p.k, nullptr, p.kap, p.L0, p.Cd, p.ye, h0, commit, energy, en, tslot, ho, bslot, n0, m0))
      return false;
    S0 = T(2) * n0;
    S1 = V3<T>{T(0), T(0), T(0)};
    SM = T(2) * m0;
  } else {
    // R(e) - 1 of the largest Gauss abscissa's e = exp(-xi phi/2)
    T turn[3][3];
    qmat_less_one(qexp_near((T(-0.5) * T(c_gxi[G - 1][G - 1])) * p.k.phi), turn);
    if (GC == 2) {
      // the sums as the half-element path forms them, so both give the same bits
      V3<T> n0, m0, n1, m1;
      T t0[3][3];
      gp_turn(turn, T(-1), t0);
      if (!FAST) hist_in(m, e, 0, h0);
      if (!gp_local<T, Y, X, HM, EN, true, S::kReadOnly, FAST>(m, e, 0, 2, p.rec, p.k, t0, p.kap, p.L0, p.Cd, p.ye, h0, commit, energy, en, tslot, ho, bslot, n0, m0))
        return false;
      if (!FAST) hist_in(m, e, 1, h1);
      if (!gp_local<T, Y, X, HM, EN, true, S::kReadOnly, FAST>(m, e, 1, 2, p.rec, p.k, turn, p.kap, p.L0, p.Cd, p.ye, h1, commit, energy, en, tslot, ho, bslot, n1, m1))
        return false;
      S0 = n0 + n1;
      S1 = T(c_gxi[1][1]) * (n1 - n0);
      SM = m0 + m1;
    } else {
      S0 = S1 = SM = V3<T>{T(0), T(0), T(0)};
      for (int g = 0; g < G; ++g) {
        const T xi = T(c_gxi[G - 1][g]), W = T(c_gw[G - 1][g]);
        V3<T> ng, mg;
        T tg[3][3];
        hist_in(m, e, g, h0);
        gp_turn(turn, xi, tg);
        if (!gp_local<T, Y, X, HM, EN, true, S::kReadOnly, FAST>(m, e, g, G, p.rec, p.k, tg, p.kap, p.L0, p.Cd, p.ye, h0, commit, energy, en, tslot, ho, bslot, ng, mg))
          return false;
        S0 = S0 + W * ng;
        S1 = S1 + (W * xi) * ng;
        SM = SM + W * mg;
      }
    }
  }
  const EndForces<T> ef = end_forces(p.k, p.L0, S0, S1, SM);
  T f[6];
  end_i(ef, f);
  store_end(efb + static_cast<size_t>(p.slot.x) * 6, f);
  end_j(ef, f);
  store_end(efb + static_cast<size_t>(p.slot.y) * 6, f);
  return true;
}

// The same with the return map, out of line: few elements flow in a step, and
// inline the map's registers spill those of the elements that do not: FP64 20^3
// BCC lattice 42.9 against 37.4 us per step, 8^3 (mixed, one block per SM) 8.0
// against 7.3.  With FP32 elements at two blocks per SM the call's own saves cost
// as much as the spills (20^3 20.0 against 21.4), and the map stays inline.
template <class T, class Y, bool X, int GC, bool EN, class S>
__device__ __noinline__ ElemEnergy element_flow(const DevModel<T> &m, S src, T *efb, int e, bool commit, bool energy,
                                                int64_t tslot, int64_t bslot) {
  ElemEnergy en;
  element_body<T, Y, X, HM_COMMIT, GC, EN, false>(m, src, efb, e, commit, energy, en, tslot, nullptr, bslot);
  return en;
}

// One element from its end states to its end forces.  ELA: plastic elements try
// the elastic form first.
template <class T, class Y, bool X, int HM, int GC, bool EN, bool ELA, class S>
__device__ __forceinline__ void element_force_from(const DevModel<T> &m, const S &src, T *efb, int e, bool commit,
                                                   bool energy, ElemEnergy &en, bool lat_energy_step, int64_t tslot,
                                                   const HistOut<T> *ho, int64_t bslot) {
  ElemEnergy one;
  if constexpr (ELA && Y::kPlastic && HM == HM_COMMIT) {
    bool done = false;
    if constexpr (GC > 0)
      done = m.plastic && element_body<T, Y, X, HM, GC, EN, true>(m, src, efb, e, true, energy, one, tslot, ho, bslot);
    if (!done) one = element_flow<T, Y, X, GC, EN>(m, src, efb, e, commit, energy, tslot, bslot);
  } else {
    element_body<T, Y, X, HM, GC, EN, false>(m, src, efb, e, commit, energy, one, tslot, ho, bslot);
  }
  en.pot += one.pot;
  en.diss += one.diss;
  if (energy && lat_energy_step && m.lat_energy) {
    atomicAdd(m.lat_energy + m.elat[e] * 5 + 1, one.pot);
    atomicAdd(m.lat_energy + m.elat[e] * 5 + 2, one.diss);
  }
}

template <class T, class Y, bool X, int HM = HM_COMMIT, int GC = 0, bool EN = false>
__device__ __forceinline__ void element_force(const DevModel<T> &m, int e, bool commit,
                                              bool energy, ElemEnergy &en, bool lat_energy_step = false,
                                              int64_t tslot = -1, const double4 *pos = nullptr,
                                              const double4 *rot = nullptr, const HistOut<T> *ho = nullptr,
                                              int64_t bslot = -1) {
  // elements of 3 or 4 nodes (no batches: no per-lattice energies); compiled
  // into the extended kernels and the predictor-corrector's history modes
  // only: the plain step kernels never see them (the launch picks the
  // extended variant), and a call site would cost them registers
  if (GC == 0 && (X || HM != HM_COMMIT) && m.nen > 2) {
    element_force_n<T, Y, X, HM>(m, e, commit, energy, en, tslot, HM == HM_COMMIT ? m.pos : pos,
                                 HM == HM_COMMIT ? m.rot : rot, ho, bslot);
    return;
  }
  element_force_from<T, Y, X, HM, GC, EN, sizeof(T) == 8>(
      m, GlobalEnds{HM == HM_COMMIT ? m.pos : pos, HM == HM_COMMIT ? m.rot : rot}, m.ef, e, commit, energy, en,
      lat_energy_step, tslot, ho, bslot);
}

// Half of a two-point element on one lane of an adjacent lane pair: both
// lanes gather the end states and form the kinematics, each lane evaluates
// Gauss point g = lane (the same instructions, so the pair does not
// diverge), the pair sums its end forces by shuffles and each lane writes one
// end slot.  Explicit step only (history committed in place).
template <class T, class Y, bool EN, bool ELA, class S>
__device__ __forceinline__ void element_force_half(const DevModel<T> &m, const S &src, T *efb, int e, int lane,
                                                   bool energy, ElemEnergy &en, bool lat_energy_step) {
  ElemEnergy one;
  HistIn<T, Y> h;
  if (ELA) hist_in(m, e, lane, h);
  ElemPre<T, Y> p;
  elem_pre(m, e, 2, src, p);
  T turn[3][3], tg[3][3];
  qmat_less_one(qexp_near((T(-0.5) * T(c_gxi[1][1])) * p.k.phi), turn);
  gp_turn(turn, lane ? T(1) : T(-1), tg);
  if (!ELA) hist_in(m, e, lane, h);
  V3<T> ng, mg;
  constexpr bool fast = ELA && Y::kPlastic;
  const bool ok = gp_local<T, Y, false, HM_COMMIT, EN, true, S::kReadOnly, fast>(
      m, e, lane, 2, p.rec, p.k, tg, p.kap, p.L0, p.Cd, p.ye, h, true, energy, one, -1, nullptr, -1, ng, mg);
  const unsigned pm = 3u << ((threadIdx.x & 31) & ~1u);
  if (fast && __any_sync(pm, !ok)) {  // a point flows: the whole element on the first lane
    if (lane) return;
    one = element_flow<T, Y, false, 2, EN>(m, src, efb, e, true, energy, -1, -1);
    en.pot += one.pot;
    en.diss += one.diss;
    if (energy && lat_energy_step && m.lat_energy) {
      atomicAdd(m.lat_energy + m.elat[e] * 5 + 1, one.pot);
      atomicAdd(m.lat_energy + m.elat[e] * 5 + 2, one.diss);
    }
    return;
  }
  const V3<T> no{__shfl_xor_sync(pm, ng.x, 1), __shfl_xor_sync(pm, ng.y, 1), __shfl_xor_sync(pm, ng.z, 1)};
  const V3<T> mo{__shfl_xor_sync(pm, mg.x, 1), __shfl_xor_sync(pm, mg.y, 1), __shfl_xor_sync(pm, mg.z, 1)};
  const V3<T> dn = lane ? ng - no : no - ng;
  const EndForces<T> ef = end_forces(p.k, p.L0, ng + no, T(c_gxi[1][1]) * dn, mg + mo);
  T fi[6], mine[6];
  end_i(ef, fi);
  end_j(ef, mine);
#pragma unroll
  for (int q = 0; q < 6; ++q) mine[q] = lane ? mine[q] : fi[q];  // selected, not indexed: registers
  store_end(efb + static_cast<size_t>(lane ? p.slot.y : p.slot.x) * 6, mine);
  en.pot += one.pot;
  en.diss += one.diss;
  if (energy && lat_energy_step && m.lat_energy) {
    atomicAdd(m.lat_energy + m.elat[e] * 5 + 1, one.pot);
    atomicAdd(m.lat_energy + m.elat[e] * 5 + 2, one.diss);
  }
}

// Contact of one candidate pair at the positions of the step's start; its
// closed flag and node forces go to the pair's slots, which the node phase
// sums per node in a fixed order (internal force, translations only:
// RodContactModel adds its contributions to fint, RodContactModel.cpp:709).
template <class T>
__device__ __noinline__ void contact_pair(const DevModel<T> &m, int p, int64_t step, bool energy, double &econ) {
  const int4 q = m.c_quad[p];  // the end nodes directly: one dependent load less than pair -> elements -> nodes
  PairGeom g;
  const double4 a0 = m.pos[q.x], a1 = m.pos[q.y], b0 = m.pos[q.z], b1 = m.pos[q.w];
  g.A[0][0] = a0.x; g.A[0][1] = a0.y; g.A[0][2] = a0.z;
  g.A[1][0] = a1.x; g.A[1][1] = a1.y; g.A[1][2] = a1.z;
  g.B[0][0] = b0.x; g.B[0][1] = b0.y; g.B[0][2] = b0.z;
  g.B[1][0] = b1.x; g.B[1][1] = b1.y; g.B[1][2] = b1.z;
  double f[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) f[k] = 0.0;
  double gap = 0.0, en = 0.0;
  // every closed evaluation of pair_contact (segment to segment, node to
  // segment) has two points of the segments within 2r: a pair whose segments
  // are further apart (with a margin far above the distance's rounding) is
  // open, and its branch logic is skipped
  const bool apart = segment_distance(g) > 2.0 * m.c_radius * (1.0 + 1e-6);
  const bool closed = !apart && pair_contact(g, m.c_radius, m.c_ks, m.c_kn, f, gap, en);
  if (energy) {
    econ += en;
    m.pair_gap[p] = closed ? gap : 1e300;
  }
  m.pclosed[p] = closed ? 1 : 0;
  if (!closed) return;
  if (m.cstamp) m.cstamp[q.x] = m.cstamp[q.y] = m.cstamp[q.z] = m.cstamp[q.w] = step;
  double *o = m.pforce + static_cast<size_t>(p) * 12;
#pragma unroll
  for (int k = 0; k < 12; ++k) o[k] = f[k];
}

// Joint contact of one candidate pair at the positions of the step's start
// (JointContactModel::computeContact_, JointContactModel.cpp:318-340): with
// n = (x_B - x_A)/d, f_int(A) -= k (2r - d) n and f_int(B) += k (2r - d) n
// when d <= 2r; its energy is -k (2r - d)^2 / 2.  No force at d = 0.
template <class T>
__device__ __noinline__ void joint_pair(const DevModel<T> &m, int p, int64_t step, bool energy, double &econ) {
  const int2 pr = m.jpairs[p];
  const double4 a = m.pos[pr.x], b = m.pos[pr.y];
  const double dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
  const double d = sqrt(dx * dx + dy * dy + dz * dz);
  const double r2 = 2.0 * m.j_radius;
  const bool closed = d <= r2;
  if (energy) m.jpair_gap[p] = closed ? d - r2 : 1e300;
  const double g = r2 - d;
  if (closed && energy) econ -= 0.5 * m.j_k * g * g;
  const bool force = closed && d > 0.0;
  m.jclosed[p] = force ? 1 : 0;
  if (!force) return;
  if (m.cstamp) m.cstamp[pr.x] = m.cstamp[pr.y] = step;
  const double s = m.j_k * g / d;
  double *o = m.jforce + static_cast<size_t>(p) * 6;
  o[0] = -s * dx;
  o[1] = -s * dy;
  o[2] = -s * dz;
  o[3] = s * dx;
  o[4] = s * dy;
  o[5] = s * dz;
}

// ---------------------------------------------------------------------------
// node phase
// ---------------------------------------------------------------------------
struct NodeOut {
  double ekin = 0.0;
  double wext = 0.0;
  double econtact = 0.0;
  int64_t last_step = -1;
};

__device__ __forceinline__ double scale_of(const double *scales, int n_scales, int64_t row, int s) {
  return s < 0 ? 1.0 : scales[row * n_scales + s];
}

// masked solve of M a = r for the free components (constrained ones preset in a);
// out of line: only nodes with partially constrained rotations call it
static __device__ __noinline__ void solve3_masked(const double M[3][3], const double r[3], double a[3],
                                              unsigned mask) {
  int fr[3], nf = 0;
  for (int i = 0; i < 3; ++i)
    if (!(mask & (1u << i))) fr[nf++] = i;
  if (nf == 0) return;
  double A[3][3], b[3];
  for (int i = 0; i < nf; ++i) {
    b[i] = r[fr[i]];
    for (int j = 0; j < 3; ++j)
      if (mask & (1u << j)) b[i] -= M[fr[i]][j] * a[j];
    for (int j = 0; j < nf; ++j) A[i][j] = M[fr[i]][fr[j]];
  }
  if (nf == 1) {
    a[fr[0]] = b[0] / A[0][0];
  } else if (nf == 2) {
    const double det = A[0][0] * A[1][1] - A[0][1] * A[1][0];
    a[fr[0]] = (b[0] * A[1][1] - A[0][1] * b[1]) / det;
    a[fr[1]] = (A[0][0] * b[1] - A[1][0] * b[0]) / det;
  } else {
    const double c00 = A[1][1] * A[2][2] - A[1][2] * A[2][1];
    const double c01 = A[1][2] * A[2][0] - A[1][0] * A[2][2];
    const double c02 = A[1][0] * A[2][1] - A[1][1] * A[2][0];
    const double det = A[0][0] * c00 + A[0][1] * c01 + A[0][2] * c02;
    const double id = 1.0 / det;
    const double inv[3][3] = {
        {c00 * id, (A[0][2] * A[2][1] - A[0][1] * A[2][2]) * id, (A[0][1] * A[1][2] - A[0][2] * A[1][1]) * id},
        {c01 * id, (A[0][0] * A[2][2] - A[0][2] * A[2][0]) * id, (A[0][2] * A[1][0] - A[0][0] * A[1][2]) * id},
        {c02 * id, (A[0][1] * A[2][0] - A[0][0] * A[2][1]) * id, (A[0][0] * A[1][1] - A[0][1] * A[1][0]) * id}};
    for (int i = 0; i < 3; ++i) a[fr[i]] = inv[i][0] * b[0] + inv[i][1] * b[1] + inv[i][2] * b[2];
  }
}

// A node's state, kept by the caller, and its record's constants.
struct NodeState {
  V3<double> x;
  Q4<double> R;
  double v[6];
};
template <class T>
struct NodeConst {
  int4 ptr;  // end-force slots and boundary terms
  T rc[NodeRecIx<T>::Dinv + 3 - NodeRecIx<T>::P];
};

// What a node's rotational update needs besides its moments: in space, the
// inverse inertia A = R P D^-1 P^T R^T (xx, yy, zz, xy, xz, yz) and the gyroscopic
// part of the acceleration, c = -A (w x M w) (SpecialCosseratRodModel::assembleGyro_,
// :951-967), for a node whose rotations are all free.  It depends on the state
// alone, so the one-barrier kernel forms it while its barrier is under way.
struct NodePre {
  double A[6], c[3];
};
template <class T>
__device__ __forceinline__ NodePre node_pre(const DevModel<T> &m, const Q4<double> &R, const V3<double> &w,
                                            const T *rc) {
  using Ix = NodeRecIx<T>;
  const Q4<double> P{double(rc[0]), double(rc[1]), double(rc[2]), double(rc[3])};
  const T *Dv = rc + (Ix::D - Ix::P), *Di = rc + (Ix::Dinv - Ix::P);
  double B[3][3];  // R P: its columns are the principal axes in space
  qmat_less_one(qmul(R, P), B);
#pragma unroll
  for (int i = 0; i < 3; ++i) B[i][i] += 1.0;
  NodePre o;
  double S[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) S[i][k] = B[i][k] * double(Di[k]);
  auto dot3 = [&](int i, int j) { return fma_rn(S[i][2], B[j][2], fma_rn(S[i][1], B[j][1], mul_rn(S[i][0], B[j][0]))); };
  o.A[0] = dot3(0, 0);
  o.A[1] = dot3(1, 1);
  o.A[2] = dot3(2, 2);
  o.A[3] = dot3(0, 1);
  o.A[4] = dot3(0, 2);
  o.A[5] = dot3(1, 2);
  o.c[0] = o.c[1] = o.c[2] = 0.0;
  if (m.gyro) {
    double l[3];  // w in the principal frame
#pragma unroll
    for (int k = 0; k < 3; ++k) l[k] = fma_rn(B[2][k], w.z, fma_rn(B[1][k], w.y, mul_rn(B[0][k], w.x)));
    const V3<double> h = cross(V3<double>{l[0], l[1], l[2]},
                                  V3<double>{mul_rn(l[0], double(Dv[0])), mul_rn(l[1], double(Dv[1])),
                                             mul_rn(l[2], double(Dv[2]))});
#pragma unroll
    for (int i = 0; i < 3; ++i) o.c[i] = -fma_rn(S[i][2], h.z, fma_rn(S[i][1], h.y, mul_rn(S[i][0], h.x)));
  }
  return o;
}

// The accelerations of a node in the cases that nodes rarely have: added point
// masses, the lumped mass, partly constrained rotations, or the internal force to
// be recorded.  Out of line: the others carry none of it.
template <class T, bool X>
__device__ __noinline__ void node_accel_general(const DevModel<T> &m, int n, bool last, const Q4<double> &R,
                                                const double v[6], const T *rc, unsigned mask, const double fx[6],
                                                double im, double r[6], double a[6], double dg[3]) {
  using Ix = NodeRecIx<T>;
  const int N = m.N;
  const bool madd = m.madd != nullptr;
  const unsigned rm = (mask >> 3) & 7u;
  const Q4<double> P{double(rc[0]), double(rc[1]), double(rc[2]), double(rc[3])};
  const T *Dv = rc + (Ix::D - Ix::P), *Di = rc + (Ix::Dinv - Ix::P);
  // rotational inertia M = R P D P^T R^T with R the current rotation
  const double D[3] = {double(Dv[0]), double(Dv[1]), double(Dv[2])};
  const double Dinv[3] = {double(Di[0]), double(Di[1]), double(Di[2])};
  const Q4<double> RP = qmul(R, P);
  const Q4<double> RPc = qconj(RP);
  const V3<double> w0{v[3], v[4], v[5]};
  if (m.gyro) {  // SpecialCosseratRodModel::assembleGyro_ (:951-967): omega x (M omega)
    V3<double> wl = qrot(RPc, w0);
    V3<double> Mw = qrot(RP, V3<double>{D[0] * wl.x, D[1] * wl.y, D[2] * wl.z});
    if (m.madd) {  // M is the explicit module's matrix, Mass models included
      Mw.x += m.madd[3 * N + n] * w0.x;
      Mw.y += m.madd[4 * N + n] * w0.y;
      Mw.z += m.madd[5 * N + n] * w0.z;
    }
    V3<double> gy = cross(w0, Mw);
    r[3] -= gy.x;
    r[4] -= gy.y;
    r[5] -= gy.z;
  }
  if (X && m.fint_last && last)  // internal force of this step (GroupOutput "resp")
    store_fint_last(m, n, fx[0] - r[0], fx[1] - r[1], fx[2] - r[2], fx[3] - r[3], fx[4] - r[4], fx[5] - r[5]);
  // added point masses (MassModel, MassModel.cpp:77-99): the explicit
  // module's mass matrix is the sum of all GET_MATRIX2 contributions, m +
  // madd per translational DOF and R P D P^T R^T + diag(madd) for the
  // rotations (then solved in full)
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (!(mask & (1u << k))) a[k] = madd ? r[k] / (m.mass[n] + m.madd[k * N + n]) : r[k] * im;
  // lumped mass (ExplicitModule LUMPED, ExplicitModule.cpp:339-357): the
  // diagonal of R P D P^T R^T (+ added masses), one DOF at a time
  if (X && m.lumped) {
    double Rm[3][3];
    qmat(RP, Rm);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      dg[i] = Rm[i][0] * Rm[i][0] * D[0] + Rm[i][1] * Rm[i][1] * D[1] + Rm[i][2] * Rm[i][2] * D[2];
      if (madd) dg[i] += m.madd[(3 + i) * N + n];
      if (!(rm & (1u << i))) a[3 + i] = r[3 + i] / dg[i];
    }
  } else if (rm == 0u && !madd) {
    V3<double> rl = qrot(RPc, V3<double>{r[3], r[4], r[5]});
    V3<double> al = qrot(RP, V3<double>{rl.x * Dinv[0], rl.y * Dinv[1], rl.z * Dinv[2]});
    a[3] = al.x;
    a[4] = al.y;
    a[5] = al.z;
  } else if (rm != 7u) {
    double Rm[3][3], M3[3][3];
    qmat(RP, Rm);
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j)
        M3[i][j] = Rm[i][0] * D[0] * Rm[j][0] + Rm[i][1] * D[1] * Rm[j][1] + Rm[i][2] * D[2] * Rm[j][2];
    if (madd)
      for (int i = 0; i < 3; ++i) M3[i][i] += m.madd[(3 + i) * N + n];
    double rr[3] = {r[3], r[4], r[5]};
    double ar[3] = {a[3], a[4], a[5]};
    solve3_masked(M3, rr, ar, rm);
    a[3] = ar[0];
    a[4] = ar[1];
    a[5] = ar[2];
  }
}

// Internal force of a launch's last step (GroupOutput "resp"): the end and contact
// forces f and the gyroscopic moment w x (M w).
template <class T>
__device__ __noinline__ void record_fint(const DevModel<T> &m, int n, Q4<double> R, V3<double> w, double f0,
                                         double f1, double f2, double f3, double f4, double f5) {
  using Ix = NodeRecIx<T>;
  T rc[Ix::Dinv + 3 - Ix::P];
  rec_load<Ix::P, Ix::Dinv + 3 - Ix::P>(m.nrec + static_cast<size_t>(n >> 5) * (Ix::vecs * 32) + (n & 31), rc);
  V3<double> gy{0.0, 0.0, 0.0};
  if (m.gyro) {
    const Q4<double> RP = qmul(R, Q4<double>{double(rc[0]), double(rc[1]), double(rc[2]), double(rc[3])});
    const T *D = rc + (Ix::D - Ix::P);
    const V3<double> wl = qrot(qconj(RP), w);
    gy = cross(w, qrot(RP, V3<double>{double(D[0]) * wl.x, double(D[1]) * wl.y, double(D[2]) * wl.z}));
  }
  store_fint_last(m, n, f0, f1, f2, f3 + gy.x, f4 + gy.y, f5 + gy.z);
}

// The update of node n's state from its summed end (and contact) forces f:
// loads, block mass solve with constraints, velocities, positions and the
// exponential-map rotation (LeapFrogModule::solve, ExplicitModule::updateVec).
// rec, sampled: whether this caller records the node's energies, and its samples.
template <class T, bool X, bool EN>
__device__ __forceinline__ void node_core(const DevModel<T> &m, int n, int64_t step, bool energy,
                                          const SampleSpec &smp, int64_t sidx, NodeOut &out, const int4 &ptr,
                                          const T *rc, double im, const NodePre &np, bool rec, bool sampled, double f[6], NodeState &st) {
  const int N = m.N;
  const Q4<double> R = st.R;
  V3<double> x = st.x;
  double v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = st.v[k];
  const double mn = EN ? m.mass[n] : 0.0;  // E_kin on every step (EN): loaded early
  if (X && m.grp_hist && m.grp_flag[n]) atomicAdd(m.grp_hist + (step - m.grp_step0), f[m.grp_dof]);
  // boundary conditions at this step (scale table row)
  double fx[6] = {0, 0, 0, 0, 0, 0};
  double a[6] = {0, 0, 0, 0, 0, 0};
  // a node whose terms all hold DOFs (or that has none) carries their mask in
  // its record; walking its terms costs a round trip to memory each, and the
  // face of held nodes would keep all others waiting at the barrier
  unsigned mask = ptr.z < 0 ? static_cast<unsigned>(-1 - ptr.z) : 0u;
  const int64_t row = step - m.scale_step0;
  bool loaded = false;
  for (int b = ptr.z < 0 ? ptr.w : ptr.z; b < ptr.w; ++b) {
    const BcTerm t = m.bc[b];
    const double val = t.factor * scale_of(m.scales, m.n_scales, row, t.scale);
    // compare-and-select over the six DOFs keeps fx/a in registers
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      if (t.dof != k) continue;
      if (t.kind == BCD_NEUMANN) {
        fx[k] += val;
      } else {
        a[k] = val;
      }
    }
    if (t.kind == BCD_NEUMANN) loaded = true;
    else mask |= 1u << t.dof;
  }
  double r[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) r[k] = fx[k] - f[k];
  const bool madd = m.madd != nullptr;
  const unsigned rm = (mask >> 3) & 7u;
  double dg[3] = {0.0, 0.0, 0.0};  // lumped mass: the diagonal
  if (madd || (X && m.lumped) || (rm != 0u && rm != 7u)) {
    // copies for the call: its arguments' addresses would keep the node's own in memory
    T rg[NodeRecIx<T>::Dinv + 3 - NodeRecIx<T>::P];
    double vg[6], fg[6], rr[6], ag[6], dd[3] = {0.0, 0.0, 0.0};
    const Q4<double> Rg = R;
#pragma unroll
    for (int k = 0; k < int(sizeof rg / sizeof rg[0]); ++k) rg[k] = rc[k];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      vg[k] = v[k];
      fg[k] = fx[k];
      rr[k] = r[k];
      ag[k] = a[k];
    }
    node_accel_general<T, X>(m, n, step == out.last_step, Rg, vg, rg, mask, fg, im, rr, ag, dd);
#pragma unroll
    for (int k = 0; k < 6; ++k) a[k] = ag[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) dg[k] = dd[k];
  } else {
    if (X && m.fint_last && step == out.last_step)
      record_fint(m, n, R, V3<double>{v[3], v[4], v[5]}, f[0], f[1], f[2], f[3], f[4], f[5]);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (!(mask & (1u << k))) a[k] = r[k] * im;
    if (rm == 0u) {
      a[3] = fma_rn(np.A[4], r[5], fma_rn(np.A[3], r[4], fma_rn(np.A[0], r[3], np.c[0])));
      a[4] = fma_rn(np.A[5], r[5], fma_rn(np.A[1], r[4], fma_rn(np.A[3], r[3], np.c[1])));
      a[5] = fma_rn(np.A[2], r[5], fma_rn(np.A[5], r[4], fma_rn(np.A[4], r[3], np.c[2])));
    }
  }
  const double dt = m.dtn ? m.dtn[n] : m.dt;
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] += dt * a[k];
  const V3<double> du{dt * v[0], dt * v[1], dt * v[2]};
  x = x + du;
  const V3<double> dr{dt * v[3], dt * v[4], dt * v[5]};
  Q4<double> Rn;
  if (m.so3) {  // ExplicitModule::updateVec (:362-392): R <- exp(dt omega) R
    Rn = qnormalize(qmul(qexp_small(dr), R));
  } else {
    V3<double> th = qlog(R);
    Rn = qexp(th + dr);
  }
  if (loaded && rec)
    out.wext += fx[0] * du.x + fx[1] * du.y + fx[2] * du.z + fx[3] * dr.x + fx[4] * dr.y + fx[5] * dr.z;
  if (energy && rec) {  // E_kin = 1/2 v^T M v, M from the rotation at the start of the step
    const V3<double> wn{v[3], v[4], v[5]};
    double ek;
    if (X && m.lumped) {
      ek = 0.5 * ((EN ? mn : m.mass[n]) * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) + dg[0] * v[3] * v[3] +
                  dg[1] * v[4] * v[4] + dg[2] * v[5] * v[5]);
      if (madd)
#pragma unroll
        for (int k = 0; k < 3; ++k) ek += 0.5 * m.madd[k * N + n] * v[k] * v[k];
    } else {
      using Ix = NodeRecIx<T>;
      const T *D = rc + (Ix::D - Ix::P);
      const V3<double> wl = qrot(
          qconj(qmul(R, Q4<double>{double(rc[0]), double(rc[1]), double(rc[2]), double(rc[3])})), wn);
      ek = 0.5 * ((EN ? mn : m.mass[n]) * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) + double(D[0]) * wl.x * wl.x +
                  double(D[1]) * wl.y * wl.y + double(D[2]) * wl.z * wl.z);
      if (madd)  // the reference's E_kin uses the global mass matrix (LatticeModel.cpp:122-129, 223-250)
#pragma unroll
        for (int k = 0; k < 6; ++k) ek += 0.5 * m.madd[k * N + n] * v[k] * v[k];
    }
    out.ekin += ek;
    if (m.lat_energy && step == out.last_step) atomicAdd(m.lat_energy + m.nlat[n] * 5 + 0, ek);
  }
  bool finite = true;
#pragma unroll
  for (int k = 0; k < 6; ++k) finite = finite && isfinite(v[k]);
  if (!finite) atomicOr(m.err, 0x2u);
  st.x = x;
  st.R = Rn;
#pragma unroll
  for (int k = 0; k < 6; ++k) st.v[k] = v[k];
  if (sidx >= 0 && smp.n_watch > 0 && sampled) {
    const int slot = smp.watch_slot[n];
    if (slot >= 0) {
      double *o = smp.rows + (sidx * smp.n_watch + slot) * 13;
      o[0] = x.x; o[1] = x.y; o[2] = x.z;
      o[3] = Rn.w; o[4] = Rn.x; o[5] = Rn.y; o[6] = Rn.z;
#pragma unroll
      for (int k = 0; k < 6; ++k) o[7 + k] = v[k];
    }
  }
}


template <class T, bool X, bool EN = false>
__device__ __forceinline__ void node_update(const DevModel<T> &m, int n, int64_t step, bool energy,
                                            const SampleSpec &smp, int64_t sidx, NodeOut &out) {
  const int N = m.N;
  // independent loads first (node state and constants), then the slot run
  using Ix = NodeRecIx<T>;
  const typename Vec16<T>::type *nr = m.nrec + static_cast<size_t>(n >> 5) * (Ix::vecs * 32) + (n & 31);
  NodeConst<T> nc;
  nc.ptr = rec_ints(nr);  // end-force slots and boundary terms of the node
  double2 *const vp = reinterpret_cast<double2 *>(m.vel + vel_ix(n, 0));
  const double2 v01 = vp[0], v23 = vp[32], v45 = vp[64];
  NodeState st{ldx(m.pos + n), ldq(m.rot + n), {v01.x, v01.y, v23.x, v23.y, v45.x, v45.y}};
  const V3<double> &x = st.x;
  rec_load<Ix::P, Ix::Dinv + 3 - Ix::P>(nr, nc.rc);
  const int i0 = nc.ptr.x, i1 = nc.ptr.y;
  // the step of the node's last closed contact pair (rod or joint contact)
  const int64_t cst = (X && m.cstamp) ? m.cstamp[n] : step;
  if (X && m.xbuild) {  // the candidate lists cover motion up to half the margin
    const double dx = x.x - m.xbuild[3 * n], dy = x.y - m.xbuild[3 * n + 1], dz = x.z - m.xbuild[3 * n + 2];
    if (dx * dx + dy * dy + dz * dz > m.half_margin * m.half_margin) atomicOr(m.err, 0x20u);
  }
  double f[6] = {0, 0, 0, 0, 0, 0};
  // a node of a rigid tie group (the HingeModel's constraints, condensed):
  // the group's end forces and contact summed over its members in the
  // group's fixed order, so that every member computes the same update; the
  // first member (the master) records the group's energies
  int t0 = 0, t1 = 0;
  if (X && m.tie_ptr) {
    t0 = m.tie_ptr[n];
    t1 = m.tie_ptr[n + 1];
  }
  const bool rec = !(X && t1 > t0) || m.tie_nodes[t0] == n;
  if (X && t1 > t0) {
    for (int t = t0; t < t1; ++t) {
      const int q = m.tie_nodes[t];
      for (int i = m.slot_ptr[q]; i < m.slot_ptr[q + 1]; ++i) load_end(m.ef + static_cast<size_t>(i) * 6, f);
      if (m.c_ptr || m.j_ptr || m.n_plates) {
        const NodeExtra ex = node_contact(m, q, step, x.x, x.y, x.z, energy && rec, rec && step == out.last_step,
                                          !m.cstamp || m.cstamp[q] == step);
        f[0] += ex.f[0];
        f[1] += ex.f[1];
        f[2] += ex.f[2];
        if (rec) out.econtact += ex.energy;
      }
    }
  } else {
    sum_ends<sizeof(T) == 4 ? 4 : 2>(m.ef, i0, i1, f);
    if (X && (m.c_ptr || m.j_ptr || m.n_plates)) {
      const NodeExtra ex = node_contact(m, n, step, x.x, x.y, x.z, energy, step == out.last_step, cst == step);
      f[0] += ex.f[0];
      f[1] += ex.f[1];
      f[2] += ex.f[2];
      out.econtact += ex.energy;
    }
  }
  const NodePre np = node_pre(m, st.R, V3<double>{st.v[3], st.v[4], st.v[5]}, nc.rc);
  node_core<T, X, EN>(m, n, step, energy, smp, sidx, out, nc.ptr, nc.rc, rec_double(nc.rc + (Ix::imass - Ix::P)), np,
                      rec, true, f, st);
  const double *v = st.v;
  vp[0] = make_double2(v[0], v[1]);
  vp[32] = make_double2(v[2], v[3]);
  vp[64] = make_double2(v[4], v[5]);
  st32(m.pos + n, st.x.x, st.x.y, st.x.z, 0.0);
  st32(m.rot + n, st.R.w, st.R.x, st.R.y, st.R.z);
  if (X && m.tp_pos) {  // adjoint recomputation: node state after this step
    const size_t sl = static_cast<size_t>(step - m.tp_step0);
    m.tp_pos[sl * N + n] = make_double4(st.x.x, st.x.y, st.x.z, 0.0);
    m.tp_rot[sl * N + n] = make_double4(st.R.w, st.R.x, st.R.y, st.R.z);
    double2 *const tv = reinterpret_cast<double2 *>(m.tp_vel + sl * 6 * tiles32(N) + vel_ix(n, 0));
    tv[0] = make_double2(v[0], v[1]);
    tv[32] = make_double2(v[2], v[3]);
    tv[64] = make_double2(v[4], v[5]);
  }
}

// ---------------------------------------------------------------------------
// grid barrier with a bounded wait
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// release and acquire at gpu scope (lighter than __threadfence(), which is
// sequentially consistent)
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Launch-constant parameters of the grid barrier, read once per launch.
struct BarrierState {
  unsigned add0;                // block 0's arrival increment
  unsigned long long limit_ns;  // bound of one wait
  bool solo;                    // a launch of one block: its own barrier is the grid's
};
__device__ __forceinline__ BarrierState barrier_begin(const GridBarrier *b) {
  const unsigned expect = gridDim.x + b->phantom;
  const unsigned lim = b->limit_us;
  return BarrierState{0x80000000u - (expect - 1u), lim ? 1000ull * lim : 2000000000ull, expect == 1u};
}

// One atomic per block: the arrival (after a fence that publishes the block's
// writes) returns the word before it; the block then polls until bit 31 differs
// from that value, and one fence afterwards makes the other blocks' writes
// visible.  The polls are relaxed loads: an acquire load drops the SM's L1 each
// time, under the warps of the SM's other block that are still working.
// grid_arrive: every thread of the block, its writes done; the returned word
// (thread 0's) goes to grid_wait.  Between the two a thread may do what no other
// block waits for.
__device__ __forceinline__ unsigned grid_arrive(GridBarrier *b, const BarrierState &bs) {
  __syncthreads();
  unsigned old = 0;
  if (!bs.solo && threadIdx.x == 0) {
    const unsigned inc = blockIdx.x == 0 ? bs.add0 : 1u;
    fence_gpu();  // the block's writes (ordered by __syncthreads) before the arrival
    old = atomicAdd(&b->count, inc);
  }
  return old;
}
// Returns false when the barrier was abandoned (its wait ran out here or in
// another block).
static __device__ bool grid_wait(GridBarrier *b, const BarrierState &bs, unsigned old, uint32_t *err) {
  __shared__ int s_ok;
  if (bs.solo) return true;
  if (threadIdx.x == 0) {
    int ok = 1;
    unsigned polls = 0;
    unsigned long long t0 = 0;
    while (((ld_relaxed(&b->count) ^ old) & 0x80000000u) == 0u) {
      if ((++polls & 63u) == 0u) {  // the abort flag and the clock now and then
        if (ld_relaxed(&b->abort)) {
          ok = 0;
          break;
        }
        const unsigned long long t = global_ns();
        if (t0 == 0) {
          t0 = t;
        } else if (t - t0 > bs.limit_ns) {
          atomicOr(err, 0x4u);
          atomicExch(&b->abort, 1u);
          ok = 0;
          break;
        }
      }
    }
    fence_gpu();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}
__device__ __forceinline__ bool grid_barrier(GridBarrier *b, const BarrierState &bs, uint32_t *err) {
  return grid_wait(b, bs, grid_arrive(b, bs), err);
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ int64_t sample_index(const SampleSpec &smp, const StepCtx &c, int64_t step) {
  if (smp.every <= 0 || step % smp.every != 0) return -1;
  const int64_t idx = c.sample_base + step / smp.every - c.step0 / smp.every - 1;
  return idx < smp.capacity ? idx : -1;
}

// Energy sums of a block's elements and nodes into the sample and the launch's
// last-step slots (all threads of the block call them).
template <class T>
__device__ __forceinline__ void add_element_energies(const SampleSpec &smp, const StepCtx &c, int64_t sidx, bool last,
                                                     const ElemEnergy &en) {
  const double p = block_sum<T>(en.pot);
  const double d = block_sum<T>(en.diss);
  if (threadIdx.x == 0) {
    if (sidx >= 0) {
      atomicAdd(smp.energy + sidx * 5 + 1, p);
      atomicAdd(smp.energy + sidx * 5 + 2, d);
    }
    if (last) {
      atomicAdd(c.last_energy + 1, p);
      atomicAdd(c.last_energy + 2, d);
    }
  }
}
template <class T>
__device__ __forceinline__ void add_node_sums(const SampleSpec &smp, const StepCtx &c, int64_t step, int64_t sidx,
                                              bool last, bool energy, const NodeOut &out) {
  const double k = energy ? block_sum<T>(out.ekin) : 0.0;
  // external work: only models with loads (c.wstep is null without them), in
  // few of whose blocks a node is loaded
  const double w = c.wstep && __syncthreads_or(out.wext != 0.0) ? block_sum<T>(out.wext) : 0.0;
  if (threadIdx.x == 0) {
    if (w != 0.0) atomicAdd(c.wstep + (step - c.step0 - 1), w);
    if (sidx >= 0) atomicAdd(smp.energy + sidx * 5 + 0, k);
    if (last) atomicAdd(c.last_energy + 0, k);
    if (sidx >= 0 && blockIdx.x == 0) smp.steps[sidx] = step;
  }
}

template <class T, class Y, bool X, bool EN = false>
__device__ __forceinline__ void element_phase(const DevModel<T> &m, const SampleSpec &smp, const StepCtx &c,
                                              int64_t step, int gtid, int gstride) {
  const int64_t sidx = sample_index(smp, c, step);
  const bool last = (step == c.step0 + c.nsteps);
  const bool energy = EN || (sidx >= 0) || last;
  ElemEnergy en;
  const int64_t tslot = (X && m.tp_hist) ? step - m.tp_step0 : -1;
  const int64_t bslot = (X && m.br) ? step - m.br_step0 - 1 : -1;
  // one- and two-point elements of two nodes take the compile-time point count;
  // elements of 3 or 4 nodes run in the extended kernels, through the
  // generic path below
  if (m.G == 2 && !(X && m.nen > 2)) {
    const int E = m.E;
    bool split = false;
    if constexpr (!X && sizeof(T) == 4) {  // the FP64 kernel spills more with the extra path
      if (E > gstride && E - gstride <= gstride / 2) {
        // one element per thread, then the rest as half elements on lane
        // pairs: the longest thread does one element and a half instead of two
        split = true;
        element_force<T, Y, X, HM_COMMIT, 2, EN>(m, gtid, true, energy, en, last, tslot);
        const int e2 = gstride + (gtid >> 1);
        if (e2 < E)
          element_force_half<T, Y, EN, false>(m, GlobalEnds{m.pos, m.rot}, m.ef, e2, gtid & 1, energy, en, last);
      }
    }
    if (!split)
      for (int e = gtid; e < E; e += gstride)
        element_force<T, Y, X, HM_COMMIT, 2, EN>(m, e, true, energy, en, last, tslot, nullptr, nullptr, nullptr,
                                                 bslot);
  } else if (m.G == 1 && !(X && m.nen > 2)) {
    for (int e = gtid; e < m.E; e += gstride)
      element_force<T, Y, X, HM_COMMIT, 1, EN>(m, e, true, energy, en, last, tslot, nullptr, nullptr, nullptr, bslot);
  } else {
    for (int e = gtid; e < m.E; e += gstride)
      element_force<T, Y, X, HM_COMMIT, 0, EN>(m, e, true, energy, en, last, tslot, nullptr, nullptr, nullptr, bslot);
  }
  double econ = 0.0;
  if (X) {
    // on from the threads that have an element less
    for (int p = (gtid + gstride - m.E % gstride) % gstride; p < m.n_pairs; p += gstride)
      contact_pair(m, p, step, energy, econ);
    for (int p = gtid; p < m.n_jpairs; p += gstride) joint_pair(m, p, step, energy, econ);
  }
  if (energy) {
    add_element_energies<T>(smp, c, sidx, last, en);
    const double q = (X && (m.n_pairs || m.n_jpairs)) ? block_sum<T>(econ) : 0.0;
    if (threadIdx.x == 0 && q != 0.0) {
      if (sidx >= 0) atomicAdd(smp.energy + sidx * 5 + 4, q);
      if (last) atomicAdd(c.last_energy + 4, q);
    }
  }
}

template <class T, bool X, bool EN = false>
__device__ __forceinline__ void node_phase(const DevModel<T> &m, const SampleSpec &smp, const StepCtx &c,
                                           int64_t step, int gtid, int gstride) {
  const int64_t sidx = sample_index(smp, c, step);
  const bool last = (step == c.step0 + c.nsteps);
  const bool energy = EN || (sidx >= 0) || last;
  NodeOut out;
  out.last_step = c.step0 + c.nsteps;
  for (int n = gtid; n < m.N; n += gstride) node_update<T, X, EN>(m, n, step, energy, smp, sidx, out);
  add_node_sums<T>(smp, c, step, sidx, last, energy, out);
  const double q = (X && energy && m.n_plates) ? block_sum<T>(out.econtact) : 0.0;
  if (threadIdx.x == 0 && q != 0.0) {
    if (sidx >= 0) atomicAdd(smp.energy + sidx * 5 + 4, q);
    if (last) atomicAdd(c.last_energy + 4, q);
  }
}

// Threads per block of a full persistent grid.  The plain FP32-element
// kernel runs 320 threads at two blocks per SM (96 registers): 94,720
// resident threads, one node per thread for a 20^3 BCC lattice's 81,261
// nodes, and few enough elements left over after one per thread to run them
// as half elements (element_phase).  The FP64 kernel and the extended
// variants (contact, plates, adjoint tape) spill more at fewer registers and
// keep 256.
template <class T, bool X>
struct PersistShape {
  static constexpr int kThreads = (sizeof(T) == 4 && !X) ? 320 : 256;
};

// X: the extended-features variant (contact, rigid plates, adjoint tape,
// per-step group force, group output of the last step); plain runs take the
// X = false kernels, which carry none of that code.  EN: every step reports
// energies (a launch of one step, whose only step is its last): the energy
// code then has no branches and its loads are issued with the others; the
// state arithmetic is the same code as in the EN = false kernel.
template <class T, class Y, bool X, bool EN = false>
__global__ void __launch_bounds__(PersistShape<T, X>::kThreads, Y::kMinBlocks)
    k_persistent(const __grid_constant__ DevModel<T> m, const __grid_constant__ SampleSpec smp, const StepCtx c,
                 GridBarrier *bar) {
  const BarrierState bs = barrier_begin(bar);
  if (blockIdx.x == 0 && threadIdx.x < 5) c.next_energy[threadIdx.x] = 0.0;
  // Items (elements, nodes) in chunks of 32 per warp, the chunks dealt to
  // the blocks round robin: a warp's items stay contiguous (Morton order, for
  // the gathers), while every block takes chunks from all over the lattice,
  // so the costly regions (return-map iterations in the impact zone) are
  // shared by all blocks instead of falling to a few, which the others would
  // wait for at the grid barrier.
  const int gtid = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
  const int gstride = gridDim.x * blockDim.x;
  for (int s = 0; s < c.nsteps; ++s) {
    const int64_t step = c.step0 + s + 1;
    element_phase<T, Y, X, EN>(m, smp, c, step, gtid, gstride);
    if (!grid_barrier(bar, bs, m.err)) return;
    node_phase<T, X, EN>(m, smp, c, step, gtid, gstride);
    // the launch's end orders its last node phase before whatever follows
    // on the stream: no barrier after the last step
    if (s + 1 < c.nsteps && !grid_barrier(bar, bs, m.err)) return;
  }
}

template <class T, class Y, bool X>
__global__ void __launch_bounds__(256, Y::kMinBlocks)
    k_element(const __grid_constant__ DevModel<T> m, const __grid_constant__ SampleSpec smp, const StepCtx c,
              int64_t step) {
  element_phase<T, Y, X>(m, smp, c, step, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <class T, bool X>
__global__ void __launch_bounds__(256, 2)
    k_node(const __grid_constant__ DevModel<T> m, const __grid_constant__ SampleSpec smp, const StepCtx c,
           int64_t step) {
  node_phase<T, X>(m, smp, c, step, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <class T, class Y>
__global__ void k_internal_force(const __grid_constant__ DevModel<T> m) {
  ElemEnergy en;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m.E; e += gridDim.x * blockDim.x) {
    if (m.nen > 2)
      element_force_n<T, Y, false, HM_COMMIT>(m, e, false, false, en, -1, m.pos, m.rot, nullptr, -1);
    else
      element_force<T, Y, false>(m, e, false, false, en);
  }
}

// Each node's internal force: the sum of its end-force slots, written to row
// n of fint (engine numbering), or to row perm[n] when perm is given (the
// caller's numbering).
template <class T>
__global__ void k_gather_force(const __grid_constant__ DevModel<T> m, double *fint, const int32_t *perm) {
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < m.N; n += gridDim.x * blockDim.x) {
    double f[6] = {0, 0, 0, 0, 0, 0};
    for (int i = m.slot_ptr[n]; i < m.slot_ptr[n + 1]; ++i) load_end(m.ef + static_cast<size_t>(i) * 6, f);
    const size_t row = perm ? static_cast<size_t>(perm[n]) : static_cast<size_t>(n);
    for (int k = 0; k < 6; ++k) fint[row * 6 + k] = f[k];
  }
}

}  // namespace dl
