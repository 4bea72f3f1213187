// The step kernel of models whose nodes fit the blocks' shared memory: one grid
// barrier per step.
//
// Each block owns a run of elements and keeps, in shared memory, its own copy
// of every node those elements touch.  A step is
//   element phase: end states from the copies, end forces to the node-ordered
//     slots in global memory (two sets, by the step's parity);
//   grid barrier;
//   node phase: the block sums the slots of all its nodes and updates its
//     copies.  A node at the border of several blocks is updated by each of
//     them, from the same slots in the same order, to the same bits.
// The copies need no second barrier: the next element phase reads only what
// this block wrote.  A block runs at most one element phase ahead of another's
// node phase, which reads the other set of slots.  The block that owns a node
// (the first that touches it) records its energies, samples and final state.
//
// What bounds the step is latency, not bandwidth: a grid barrier is 1.7 us, a
// dependent round trip to L2 0.4 us.  Against the two-barrier kernel (step.cuh),
// which reads every node state from L2 in both phases, this one drops a
// barrier, the gathers and the state loads of a step for 10 to 50 % more node
// updates.  us per step, two barriers against one: 4^3 BCC 9.7 / 6.1, 8^3 10.5 / 6.3
// (FP64 12.4 / 6.4), 5^3 octet FP64 9.0 / 5.7, 17^3 SC 9.1 / 6.2, 20^3 BCC (two blocks
// per SM) 22.7 / 19.7 and FP64 37.4 / 33.8.
#pragma once

#include "step.cuh"

namespace dl {

// Shared memory of one block: per node copy its state (q, x, v as 14 doubles: rows
// of 112 bytes, whose 16-byte words spread over all banks), what its update needs
// besides forces (NodePre, 9 doubles), its record and its number; and, where they
// fit, the records of the block's elements.
template <class T>
struct LocalShape {
  static constexpr int row = 14;
  DL_HDI static size_t bytes(int cap, int chunk_recs, int G) {
    return static_cast<size_t>(cap) * (row * sizeof(double) + sizeof(double) * 9 + NodeRecIx<T>::vecs * 16 + 4) + 16 +
           static_cast<size_t>(tiles32(chunk_recs)) * ElemRecIx<T>::vecs(G) * 16;
  }
};

template <class T>
struct LocalEnds {
  static constexpr bool kReadOnly = false;
  const double *rows;
  const uint32_t *ends;
  const typename Vec16<T>::type *recs;  // of element e0 on (null: in global memory)
  int e0;
  template <class U>
  __device__ __forceinline__ const typename Vec16<U>::type *rec(const DevModel<U> &m, int e, int nv) const {
    const int i = recs ? e - e0 : e;
    return (recs ? recs : m.erec) + static_cast<size_t>(i >> 5) * (nv * 32) + (i & 31);
  }
  __device__ __forceinline__ void node(int i, V3<double> &x, Q4<double> &R) const {
    const double2 *r = reinterpret_cast<const double2 *>(rows + i * LocalShape<T>::row);
    const double2 a = r[0], b = r[1], c = r[2];
    R = Q4<double>{a.x, a.y, b.x, b.y};
    x = V3<double>{c.x, c.y, rows[i * LocalShape<T>::row + 6]};
  }
  __device__ __forceinline__ void get(int e, int4, V3<double> &xi, V3<double> &xj, Q4<double> &Ri,
                                      Q4<double> &Rj) const {
    const uint32_t c = __ldg(ends + e);
    node(static_cast<int>(c & 0xffffu), xi, Ri);
    node(static_cast<int>(c >> 16), xj, Rj);
  }
};

// MB: blocks per SM that the kernel's registers leave room for.  Models of at most
// a block per SM take the MB = 1 kernel: 168 (FP64 255) registers a thread and half
// the spills of MB = 2, which has 96 (128): 456 against 820 bytes (552 against 1,180).
template <class T, class Y, int MB>
__global__ void __launch_bounds__(LocalThreads<T>::value, Y::kMinBlocks < MB ? Y::kMinBlocks : MB)
    k_local(const __grid_constant__ DevModel<T> m, const __grid_constant__ SampleSpec smp, const StepCtx c,
            GridBarrier *bar, const LocalPlan plan) {
  extern __shared__ __align__(16) double s_rows[];
  constexpr int row = LocalShape<T>::row;
  constexpr bool ela = MB == 1 || sizeof(T) == 8;
  using Ix = NodeRecIx<T>;
  using V = typename Vec16<T>::type;
  V *const s_rec = reinterpret_cast<V *>(s_rows + static_cast<size_t>(plan.cap) * row);
  V *const s_erec = s_rec + static_cast<size_t>(plan.cap) * Ix::vecs;
  const int nv = ElemRecIx<T>::vecs(m.G);
  double *const s_pre = reinterpret_cast<double *>(s_erec + (plan.recs ? static_cast<size_t>(tiles32(plan.chunk)) * nv : 0));
  int32_t *const s_id = reinterpret_cast<int32_t *>(s_pre + static_cast<size_t>(plan.cap) * 9);
  const BarrierState bs = barrier_begin(bar);
  if (blockIdx.x == 0 && threadIdx.x < 5) c.next_energy[threadIdx.x] = 0.0;
  const int e0 = blockIdx.x * plan.chunk;
  const int ne = min(m.E - e0, plan.chunk);
  const int p0 = plan.node_ptr[blockIdx.x], nn = plan.node_ptr[blockIdx.x + 1] - p0;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < nn; i += nt) {
    s_id[i] = plan.nodes[p0 + i];
    const int n = s_id[i] & 0x7fffffff;
    double *r = s_rows + i * row;
    const V3<double> x = ldx(m.pos + n);
    const Q4<double> q = ldq(m.rot + n);
    r[0] = q.w; r[1] = q.x; r[2] = q.y; r[3] = q.z;
    r[4] = x.x; r[5] = x.y; r[6] = x.z;
    for (int k = 0; k < 6; ++k) r[8 + k] = m.vel[vel_ix(n, k)];
    const V *g = m.nrec + static_cast<size_t>(n >> 5) * (Ix::vecs * 32) + (n & 31);
    for (int v = 0; v < Ix::vecs; ++v) s_rec[v * plan.cap + i] = g[v * 32];
  }
  if (plan.recs)
    for (int i = tid; i < ne; i += nt) {
      const V *g = m.erec + static_cast<size_t>((e0 + i) >> 5) * (nv * 32) + ((e0 + i) & 31);
      V *o = s_erec + static_cast<size_t>(i >> 5) * (nv * 32) + (i & 31);
      for (int v = 0; v < nv; ++v) o[v * 32] = g[v * 32];
    }
  __syncthreads();
  const LocalEnds<T> src{s_rows, plan.ends, plan.recs ? s_erec : nullptr, e0};
  auto rec_scalar = [&](int i, int k) {
    return reinterpret_cast<const T *>(s_rec + (k / Vec16<T>::n) * plan.cap + i)[k % Vec16<T>::n];
  };
  const size_t set = static_cast<size_t>(m.E) * 12;
  for (int s = 0; s < c.nsteps; ++s) {
    const int64_t step = c.step0 + s + 1;
    T *const ef = m.ef + (s & 1) * set;
    const int64_t sidx = sample_index(smp, c, step);
    const bool last = s + 1 == c.nsteps;
    const bool energy = sidx >= 0 || last;
    // ---- element phase
    ElemEnergy en;
    if (m.G == 2) {
      bool split = false;
      if constexpr (sizeof(T) == 4) {
        if (ne > nt && ne - nt <= nt / 2) {
          // one element per thread, the rest as half elements on lane pairs
          split = true;
          element_force_from<T, Y, false, HM_COMMIT, 2, false, ela>(m, src, ef, e0 + tid, true, energy, en, last, -1,
                                                               nullptr, -1);
          const int e2 = nt + (tid >> 1);
          if (e2 < ne) element_force_half<T, Y, false, ela>(m, src, ef, e0 + e2, tid & 1, energy, en, last);
        }
      }
      if (!split)
        for (int e = tid; e < ne; e += nt)
          element_force_from<T, Y, false, HM_COMMIT, 2, false, ela>(m, src, ef, e0 + e, true, energy, en, last, -1,
                                                               nullptr, -1);
    } else if (m.G == 1) {
      for (int e = tid; e < ne; e += nt)
        element_force_from<T, Y, false, HM_COMMIT, 1, false, ela>(m, src, ef, e0 + e, true, energy, en, last, -1, nullptr,
                                                             -1);
    } else {
      for (int e = tid; e < ne; e += nt)
        element_force_from<T, Y, false, HM_COMMIT, 0, false, ela>(m, src, ef, e0 + e, true, energy, en, last, -1, nullptr,
                                                             -1);
    }
    if (energy) add_element_energies<T>(smp, c, sidx, last, en);
    const unsigned word = grid_arrive(bar, bs);
    // ---- while the barrier is under way: what the node updates need besides
    // the forces it guards
    for (int i = tid; i < nn; i += nt) {
      const double2 *r2 = reinterpret_cast<const double2 *>(s_rows + i * row);
      const double2 q0 = r2[0], q1 = r2[1], w0 = r2[5], w1 = r2[6];
      T rc[Ix::Dinv + 3 - Ix::P];
#pragma unroll
      for (int k = Ix::P; k < Ix::Dinv + 3; ++k) rc[k - Ix::P] = rec_scalar(i, k);
      const NodePre np = node_pre(m, Q4<double>{q0.x, q0.y, q1.x, q1.y}, V3<double>{w0.y, w1.x, w1.y}, rc);
#pragma unroll
      for (int k = 0; k < 6; ++k) s_pre[k * plan.cap + i] = np.A[k];
#pragma unroll
      for (int k = 0; k < 3; ++k) s_pre[(6 + k) * plan.cap + i] = np.c[k];
    }
    if (!grid_wait(bar, bs, word, m.err)) {
      // the owned copies go back here too: the state is then, as after the
      // two-barrier kernels, at most a phase or two behind the history, and not the
      // launch's first.  (One write-back behind the loop costs the FP64 kernel 2 % of
      // a step, in registers.)
      for (int i = tid; i < nn; i += nt) {
        if (s_id[i] >= 0) continue;
        const int n = s_id[i] & 0x7fffffff;
        const double *const r = s_rows + i * row;
        st32(m.pos + n, r[4], r[5], r[6], 0.0);
        st32(m.rot + n, r[0], r[1], r[2], r[3]);
        for (int k = 0; k < 6; ++k) m.vel[vel_ix(n, k)] = r[8 + k];
      }
      return;
    }
    // ---- node phase
    NodeOut out;
    out.last_step = c.step0 + c.nsteps;
    for (int i = tid; i < nn; i += nt) {
      const int id = s_id[i];
      const int n = id & 0x7fffffff;
      const bool own = id < 0;
      const int4 ptr = *reinterpret_cast<const int4 *>(s_rec + i);
      double f[6] = {0, 0, 0, 0, 0, 0};
      // the copies are sorted by their number of slots, most first: the first of the
      // warp's 32 chooses for all of them
      const int4 most = *reinterpret_cast<const int4 *>(s_rec + (i & ~31));
      if (most.y - most.x <= 2) sum_ends<2>(ef, ptr.x, ptr.y, f);
      else sum_ends<sizeof(T) == 4 ? 8 : 4>(ef, ptr.x, ptr.y, f);
      double *const r = s_rows + i * row;
      double2 *const r2 = reinterpret_cast<double2 *>(r);
      const double2 q0 = r2[0], q1 = r2[1], x0 = r2[2], v0 = r2[4], v1 = r2[5], v2 = r2[6];
      NodeState st{V3<double>{x0.x, x0.y, r[6]}, Q4<double>{q0.x, q0.y, q1.x, q1.y},
                   {v0.x, v0.y, v1.x, v1.y, v2.x, v2.y}};
      T rc[Ix::Dinv + 3 - Ix::P];
#pragma unroll
      for (int k = Ix::P; k < Ix::Dinv + 3; ++k) rc[k - Ix::P] = rec_scalar(i, k);
      NodePre np;
#pragma unroll
      for (int k = 0; k < 6; ++k) np.A[k] = s_pre[k * plan.cap + i];
#pragma unroll
      for (int k = 0; k < 3; ++k) np.c[k] = s_pre[(6 + k) * plan.cap + i];
      node_core<T, false, false>(m, n, step, energy, smp, sidx, out, ptr, rc, rec_double(rc + (Ix::imass - Ix::P)), np, own,
                                 own, f, st);
      r2[0] = make_double2(st.R.w, st.R.x);
      r2[1] = make_double2(st.R.y, st.R.z);
      r2[2] = make_double2(st.x.x, st.x.y);
      r[6] = st.x.z;
      r2[4] = make_double2(st.v[0], st.v[1]);
      r2[5] = make_double2(st.v[2], st.v[3]);
      r2[6] = make_double2(st.v[4], st.v[5]);
      if (last && own) {
        st32(m.pos + n, st.x.x, st.x.y, st.x.z, 0.0);
        st32(m.rot + n, st.R.w, st.R.x, st.R.y, st.R.z);
        for (int k = 0; k < 6; ++k) m.vel[vel_ix(n, k)] = st.v[k];
      }
    }
    add_node_sums<T>(smp, c, step, sidx, last, energy, out);
    __syncthreads();  // the copies, before the next element phase reads them
  }
}

}  // namespace dl
