// Expected-value (individual-based mean-field) replay and its adjoint.
//
// Same per-step window CSRs as the Monte Carlo replay (int32 contact-second
// weights w_ij, weight scale 1/steps-in-window), FP32 node probabilities
// x = (S, E, I, R), four planes of N floats.  One step t, with
// e_i = scale_t * sum_j w_ij I_j and P_i = 1 - exp(-beta s_i e_i):
//   new_i = S_i P_i                     (to E, or to I without an exposed state)
//   S' = S (1 - P) + p_rs R [+ p_ir I when I -> S]
//   E' = E (1 - p_ei) + new             (exposed state only)
//   I' = I (1 - p_ir) + p_ei E          (+ new without an exposed state)
//   R' = R (1 - p_rs) [+ p_ir I when I -> R]
// and the step's expected incidence is sum_i new_i.  This is the
// expectation of the geometric Monte Carlo step with every indicator
// replaced by its probability (p_S <- p_S exp(-beta s_i sum_j w_ij p_I,j)).
//
// The adjoint runs backwards over the same CSRs: with y = dL/dx_{t+1} and
// g_t = dL/dincidence_t, u_i = y_X,i - y_S,i + g_t (X the infection target),
//   dL/dS_i = y_S + P u,  dL/dE_i = y_E + p_ei (y_I - y_E),
//   dL/dR_i = y_R + p_rs (y_S - y_R),
//   dL/dI_j = y_I + p_ir (y_Y - y_I) + sum_i w_ij z_i,
//   z_i = scale S_i u_i exp(-beta s_i e_i) beta s_i
// (the transpose SpMV is the same CSR: the window graph is symmetric), and
// the parameter gradients
//   dL/dbeta += sum_i S u q s e,  dL/ds_i += S u q beta e,
//   dL/dp_ei += sum E (y_I - y_E), dL/dp_ir += sum I (y_Y - y_I),
//   dL/dp_rs += sum R (y_S - y_R).
// One kernel per reverse step finishes dL/dx_t of a row (gather of z_t over
// its neighbours) and immediately takes the local part of step t-1 for the
// same row.  Scalar gradients accumulate in FP64, per warp, in fixed order.
// The kernels read the rates from device memory, so that the host captures
// a whole forward (and a whole adjoint) once as a CUDA graph and replays it
// for any beta and rates.
#include "rp_device.cuh"
#include "rp_internal.h"

namespace rp {
namespace {

// A step is a short chain of dependent loads (row pointers, pairs, the
// neighbours' values, a few arithmetic operations): 1.6 KB a row pointer page
// and 24-32 B a node, all in L2, so launches and latency bound it and not
// bandwidth.  Hence: what does not depend on the previous step (row pointers
// and the first pairs, rates, susceptibility, the adjoint's stored states) is
// loaded before the wait for it, which programmatic dependent launch lets
// overlap the previous kernel; pairs and neighbours are loaded four at a time;
// sums leave a warp by shuffles, without a block barrier.  Per step kernel,
// launches included, over 336 steps: N = 100,000 6.5 us before, 3.6 us forward
// and 5.1 us reverse now.
constexpr int kMfThreads = 128;
constexpr int kMfWarps = kMfThreads / 32;

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
  return v;  // valid in lane 0
}

// The first four pairs of row i, loaded ahead of the values they select.
struct RowHead {
  int32_t beg = 0, end = 0;
  int2 q[4];
};
__device__ __forceinline__ RowHead row_head(const int32_t *__restrict__ rp,
                                            const int2 *__restrict__ ent, int32_t i) {
  RowHead h;
  h.beg = __ldg(rp + i);
  h.end = __ldg(rp + i + 1);
#pragma unroll
  for (int j = 0; j < 4; ++j)
    h.q[j] = h.beg + j < h.end ? __ldg(ent + h.beg + j) : make_int2(0, 0);
  return h;
}
// sum_k w_k v[col_k] in CSR order.  v was written by the previous kernel.
__device__ __forceinline__ float row_exposure(const RowHead &h, const int2 *__restrict__ ent,
                                              const float *v) {
  float e = 0.0f, val[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) val[j] = h.beg + j < h.end ? __ldcg(v + h.q[j].x) : 0.0f;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (h.beg + j < h.end) e = fmaf((float)h.q[j].y, val[j], e);
  for (int32_t k = h.beg + 4; k < h.end; k += 4) {
    int2 q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = k + j < h.end ? __ldg(ent + k + j) : make_int2(0, 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) val[j] = k + j < h.end ? __ldcg(v + q[j].x) : 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (k + j < h.end) e = fmaf((float)q[j].y, val[j], e);
  }
  return e;
}

// One node's step: its probabilities in, out in place; returns the new
// infections.  Products and sums are rounded as written, so that all kernels
// that take a step or its adjoint agree bit for bit.
struct MfNode {
  float S, E, I, R;
};
__device__ __forceinline__ float mf_node_step(const MfRates &r, float si, float es, MfNode &v,
                                              float &q) {
  const float a = __fmul_rn(__fmul_rn(r.beta, si), es);
  const float P = -expm1f(-a);
  q = expf(-a);
  const float newinf = __fmul_rn(v.S, P);
  const float f_ei = r.has_exposed ? __fmul_rn(v.E, r.p_ei) : 0.0f;
  const float f_i = __fmul_rn(v.I, r.p_ir), f_rs = __fmul_rn(v.R, r.p_rs);
  float S2 = fmaf(v.S, q, f_rs), E2 = __fsub_rn(v.E, f_ei);
  float I2 = __fadd_rn(__fsub_rn(v.I, f_i), f_ei), R2 = __fsub_rn(v.R, f_rs);
  if (r.has_exposed) E2 = __fadd_rn(E2, newinf); else I2 = __fadd_rn(I2, newinf);
  if (r.ir_to_s) S2 = __fadd_rn(S2, f_i); else R2 = __fadd_rn(R2, f_i);
  v.S = S2, v.E = E2, v.I = I2, v.R = R2;
  return newinf;
}
// One node's local adjoint: y = dL/dx_{t+1} in, the local part of dL/dx_t out
// in place; returns z without the step's factors (S u q).
__device__ __forceinline__ float mf_node_adjoint(const MfRates &r, const MfNode &x, float q,
                                                 float g, MfNode &y) {
  const float P = 1.0f - q;
  const float yX = r.has_exposed ? y.E : y.I;
  const float yY = r.ir_to_s ? y.S : y.R;
  const float u = __fadd_rn(__fsub_rn(yX, y.S), g);
  const float suq = __fmul_rn(__fmul_rn(x.S, u), q);
  const float aS = fmaf(P, u, y.S);
  const float aE = r.has_exposed ? fmaf(r.p_ei, __fsub_rn(y.I, y.E), y.E) : y.E;
  const float aI = fmaf(r.p_ir, __fsub_rn(yY, y.I), y.I);
  const float aR = fmaf(r.p_rs, __fsub_rn(y.S, y.R), y.R);
  y.S = aS, y.E = aE, y.I = aI, y.R = aR;
  return suq;
}

// A node's terms of the four rate gradients, added to the sums (FP64).
__device__ __forceinline__ void rate_terms(const MfRates &r, const MfNode &x, const MfNode &y,
                                           float suq, float si, float es, double &gb, double &ge,
                                           double &gi, double &gr) {
  gb += (double)suq * (double)si * (double)es;
  if (r.has_exposed) ge += (double)x.E * ((double)y.I - (double)y.E);
  gi += (double)x.I * ((double)(r.ir_to_s ? y.S : y.R) - (double)y.I);
  gr += (double)x.R * ((double)y.S - (double)y.R);
}

__global__ void __launch_bounds__(kMfThreads)
    k_mf_step(const int32_t *__restrict__ rp, const int2 *__restrict__ ent, int32_t n, float scale,
              const MfRates *__restrict__ rates, const float *__restrict__ sus, const float *x,
              float *xo, float *q_out, float *e_out, float *inc_part) {
  cudaTriggerProgrammaticLaunchCompletion();
  const MfRates r = *rates;
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  RowHead h;
  float si = 1.0f;
  if (i < n) {
    h = row_head(rp, ent, i);
    if (sus) si = __ldg(sus + i);
  }
  cudaGridDependencySynchronize();
  float newinf = 0.0f;
  if (i < n) {
    MfNode v{__ldcg(x + i), __ldcg(x + n + i), __ldcg(x + 2 * (size_t)n + i),
             __ldcg(x + 3 * (size_t)n + i)};
    const float es = row_exposure(h, ent, x + 2 * (size_t)n) * scale;
    float q;
    newinf = mf_node_step(r, si, es, v, q);
    xo[i] = v.S;
    xo[n + i] = v.E;
    xo[2 * (size_t)n + i] = v.I;
    xo[3 * (size_t)n + i] = v.R;
    if (q_out) q_out[i] = q;
    if (e_out) e_out[i] = es;
  }
  const float tot = warp_sum(newinf);
  if ((threadIdx.x & 31) == 0) inc_part[i >> 5] = tot;
}

// Incidence of each step: the sum of the step's warp partials, in FP64, one
// warp per step (always in the same order).
__global__ void __launch_bounds__(kMfThreads)
    k_mf_incidence(const float *__restrict__ part, int32_t nwarp, int32_t T,
                   float *__restrict__ inc) {
  const int32_t t = blockIdx.x * kMfWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  double s = 0.0;
  for (int32_t b = lane; b < nwarp; b += 32) s += (double)part[(size_t)t * nwarp + b];
  s = warp_sum(s);
  if (lane == 0) inc[t] = (float)s;
}

// One reverse step.  Coupling part (when rp_c != nullptr): the full adjoint
// of x_tc is a_loc + (0, 0, sum_j w_ij z_j, 0).  Local part (when x != nullptr):
// from that adjoint y (of x_{tl+1}) and the step tl data, the local adjoint
// of x_tl goes to a_out and z_tl to z_out; parameter gradients accumulate per
// warp.  Without a local part the full adjoint goes to a_out.  `early`: x, qv
// and ev were written before the previous kernel started (stored by the
// forward, not recomputed just now).
__global__ void __launch_bounds__(kMfThreads)
    k_mf_adjoint(int32_t n, const int32_t *__restrict__ rp_c, const int2 *__restrict__ ent_c,
                 const float *z_in, const float *a_in, const float *x, const float *qv,
                 const float *ev, const float *ginc, int32_t tl, float scale,
                 const MfRates *__restrict__ rates, const float *__restrict__ sus, float *a_out,
                 float *z_out, float *gsus, double *gpart, int32_t early) {
  cudaTriggerProgrammaticLaunchCompletion();
  const MfRates r = *rates;
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  RowHead h;
  MfNode v{};
  float q = 0, es = 0, si = 1.0f, g = 0;
  auto load_step = [&]() {
    v.S = __ldcg(x + i), v.E = __ldcg(x + n + i), v.I = __ldcg(x + 2 * (size_t)n + i),
    v.R = __ldcg(x + 3 * (size_t)n + i);
    q = __ldcg(qv + i), es = __ldcg(ev + i);
  };
  if (i < n) {
    if (rp_c) h = row_head(rp_c, ent_c, i);
    if (x && sus) si = __ldg(sus + i);
    if (x && early) load_step();
  }
  cudaGridDependencySynchronize();
  double gb = 0.0, ge = 0.0, gi = 0.0, gr = 0.0;
  if (i < n) {
    MfNode y{__ldcg(a_in + i), __ldcg(a_in + n + i), __ldcg(a_in + 2 * (size_t)n + i),
             __ldcg(a_in + 3 * (size_t)n + i)};
    if (x && !early) load_step();
    if (x && ginc) g = __ldcg(ginc + tl);  // dL/dincidence of step tl
    const float gs0 = x && gsus ? __ldcg(gsus + i) : 0.0f;
    if (rp_c) y.I = __fadd_rn(y.I, row_exposure(h, ent_c, z_in));
    if (x) {
      const MfNode full = y;
      const float suq = mf_node_adjoint(r, v, q, g, y);
      // d(es_i)/dI_j = scale w_ij, so z_i = scale * S u q beta s_i
      z_out[i] = suq * r.beta * si * scale;
      if (gsus) gsus[i] = fmaf(__fmul_rn(suq, r.beta), es, gs0);
      rate_terms(r, v, full, suq, si, es, gb, ge, gi, gr);
    }
    a_out[i] = y.S;
    a_out[n + i] = y.E;
    a_out[2 * (size_t)n + i] = y.I;
    a_out[3 * (size_t)n + i] = y.R;
  }
  if (!x) return;
  gb = warp_sum(gb);
  ge = warp_sum(ge);
  gi = warp_sum(gi);
  gr = warp_sum(gr);
  if ((threadIdx.x & 31) == 0) {
    double2 *p = reinterpret_cast<double2 *>(gpart + 4 * (size_t)(i >> 5));
    double2 p0 = __ldcg(p), p1 = __ldcg(p + 1);
    p0.x += gb;
    p0.y += ge;
    p1.x += gi;
    p1.y += gr;
    p[0] = p0;
    p[1] = p1;
  }
}

// ---- the whole replay in one cluster ------------------------------------
// A small network's step is bound by the chain launch -> loads from L2 ->
// stores, with nearly all of the chip idle.  Up to kMfClusterNodes nodes are
// held by one cluster of eight blocks instead, a node to a thread with its
// state in registers; the plane that neighbours read (I forward, z in reverse)
// is copied to all eight blocks' shared memory, double buffered, so that a
// step is one cluster barrier, a gather from the block's own copy and eight
// coalesced remote stores.  The barrier's release waits for what the block has
// in flight, 0.4 us of a step, so loads are issued up to three steps ahead and
// nothing is stored that can be had afterwards (k_mf_after).
// Per step over 336 steps, forward and reverse, copies included: N = 2,000
// with 180 contacts a node 1.74 and 2.62 us with a launch per step, 0.94 and
// 1.00 us here; with 2,000 contacts a node 5.19 and 5.72 against 3.00 and 2.93;
// N = 500 1.58 and 2.34 against 0.84 and 0.86; N = 4,000 1.81 and 2.76 against
// 1.30 and 1.36.  Gathering from the owner's shared memory, without the
// copies, is slower: 1.42 and 1.57 us at N = 2,000, 2.36 and 2.21 at 4,000
// (a 4-byte remote load a pair).  Above 4,096 nodes a block would need more
// than 512 threads, whose registers spill, and the gain has shrunk.
constexpr int kMfCluster = 8;
constexpr int kMfClusterThreads = kMfClusterNodes / kMfCluster;
static_assert(kMfClusterThreads <= 1024, "one node per thread");

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// The plane that neighbours read, a copy in each block: a node's thread stores
// its value to all eight (128 B a warp and block), a gather stays in the block.
struct ClusterPlane {
  uint32_t local;              // of element 0 of buffer 0
  uint32_t mine[kMfCluster];   // of this thread's element in each block
  __device__ __forceinline__ ClusterPlane(const float *plane, uint32_t node) {
    local = (uint32_t)__cvta_generic_to_shared(plane);
#pragma unroll
    for (int k = 0; k < kMfCluster; ++k)
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(mine[k]) : "r"(local + 4u * node), "r"(k));
  }
  __device__ __forceinline__ void store(uint32_t buffer, float v) const {
#pragma unroll
    for (int k = 0; k < kMfCluster; ++k)
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mine[k] + buffer), "f"(v) : "memory");
  }
};
__device__ __forceinline__ float ld_plane(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// The steps' rows of one node, loaded ahead while step t is computed: pairs of
// the next step in the order the steps are run, row bounds of the one after
// it, that step's pointers one earlier still, so that no load waits for
// another one of the same step.
constexpr int kAhead = 8;  // pairs of a row that are loaded ahead
struct RowAhead {
  const MfStep *steps;
  int32_t node, n_steps, dir;  // node < 0: no row
  uint32_t plane;  // ClusterPlane::local
  MfStep s1, s2, s3;  // of the next steps; s1.entries + beg1 are its pairs
  int32_t beg1 = 0, end1 = 0, beg2 = 0, end2 = 0;
  int2 q1[kAhead];
  // the current step's
  const int2 *ent = nullptr;
  int32_t beg = 0, end = 0;
  uint32_t at[kAhead];
  float w[kAhead], scale = 0.0f;

  __device__ __forceinline__ MfStep step(int32_t t) const {
    return t >= 0 && t < n_steps ? steps[t] : MfStep{nullptr, nullptr, 0.0f};
  }
  __device__ __forceinline__ void load_bounds() {
    beg2 = end2 = 0;
    if (node >= 0 && s2.row_ptr) {
      beg2 = __ldg(s2.row_ptr + node);
      end2 = __ldg(s2.row_ptr + node + 1);
    }
  }
  __device__ __forceinline__ void load_pairs() {
    const int2 *p = s1.entries + beg1;
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      q1[j] = beg1 + j < end1 ? __ldg(p + j) : make_int2(0, 0);
  }
  __device__ __forceinline__ void start(int32_t t) {
    s2 = step(t);
    load_bounds();
    s1 = s2, beg1 = beg2, end1 = end2;
    load_pairs();
    s2 = step(t + dir);
    load_bounds();
    s3 = step(t + 2 * dir);
  }
  // Makes step t current; starts the loads of the three after it.
  __device__ __forceinline__ void advance(int32_t t) {
    ent = s1.entries;
    beg = beg1, end = end1, scale = s1.scale;
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      at[j] = plane + 4u * (uint32_t)q1[j].x;
      w[j] = (float)q1[j].y;
    }
    s1 = s2, beg1 = beg2, end1 = end2;
    load_pairs();
    s2 = s3;
    load_bounds();
    s3 = step(t + 3 * dir);
  }
  // sum_k w_k v[col_k] in row order, as row_exposure.
  __device__ __forceinline__ float exposure(uint32_t buffer) const {
    float e = 0.0f;
#pragma unroll
    for (int h = 0; h < kAhead; h += 4) {
      if (beg + h >= end) break;
      float val[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) val[j] = beg + h + j < end ? ld_plane(at[h + j] + buffer) : 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) e = fmaf(w[h + j], val[j], e);  // none: 0 * 0
    }
    for (int32_t k = beg + kAhead; k < end; k += 4) {
      int2 q[4];
      float val[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) q[j] = k + j < end ? __ldg(ent + k + j) : make_int2(0, 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) val[j] = k + j < end ? ld_plane(plane + 4u * (uint32_t)q[j].x + buffer) : 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) e = fmaf((float)q[j].y, val[j], e);
    }
    return e;
  }
};

__global__ void __launch_bounds__(kMfClusterThreads) __cluster_dims__(kMfCluster, 1, 1)
    k_mf_forward(const MfStep *__restrict__ steps, int32_t n_steps, int32_t n,
                 const MfRates *__restrict__ rates, const float *__restrict__ sus, float *states,
                 float *ev) {
  __shared__ float s_plane[2][kMfClusterNodes];
  const MfRates r = *rates;
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < n;
  const size_t N = n;
  const ClusterPlane plane(&s_plane[0][0], i);
  MfNode v{};
  float si = 1.0f;
  if (on) {
    v = MfNode{states[i], states[N + i], states[2 * N + i], states[3 * N + i]};
    si = __ldg(sus + i);
  }
  cluster_arrive();
  cluster_wait();  // every block has started
  plane.store(0, v.I);
  cluster_arrive();
  RowAhead rows{steps, on ? i : -1, n_steps, 1, plane.local};
  rows.start(0);
  float q, es = 0.0f;
  float *xo = states + i, *eo = ev + i;
  auto store = [&]() {  // what the last step computed
    xo += 4 * N;
    if (on) {
      xo[0] = v.S;
      xo[N] = v.E;
      xo[2 * N] = v.I;
      xo[3 * N] = v.R;
      eo[0] = es;
    }
    eo += N;
  };
  for (int32_t t = 0; t < n_steps; ++t) {
    if (t > 0) store();
    rows.advance(t);
    cluster_wait();
    es = rows.exposure((t & 1) * (uint32_t)sizeof(s_plane[0])) * rows.scale;
    mf_node_step(r, si, es, v, q);
    plane.store(((t & 1) ^ 1) * (uint32_t)sizeof(s_plane[0]), v.I);
    cluster_arrive();
  }
  store();
  cluster_wait();  // no block leaves while its plane is read
}

__global__ void __launch_bounds__(kMfClusterThreads) __cluster_dims__(kMfCluster, 1, 1)
    k_mf_reverse(const MfStep *__restrict__ steps, int32_t n_steps, int32_t n,
                 const MfRates *__restrict__ rates, const float *__restrict__ sus,
                 const float *__restrict__ a_in, const float *__restrict__ states,
                 const float *__restrict__ qv, const float *__restrict__ ev,
                 const float *__restrict__ ginc, float *__restrict__ gx0,
                 float *__restrict__ gsus, double *__restrict__ gpart, int32_t nwarp) {
  __shared__ float s_plane[2][kMfClusterNodes];
  const MfRates r = *rates;
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < n;
  const size_t N = n;
  const ClusterPlane plane(&s_plane[0][0], i);
  MfNode y{};
  float si = 1.0f, gs = 0.0f;
  if (on) {
    y = MfNode{a_in[i], a_in[N + i], a_in[2 * N + i], a_in[3 * N + i]};
    si = __ldg(sus + i);
  }
  // the last step's adjoint has no coupling: its neighbours' z are zero
  cluster_arrive();
  cluster_wait();  // every block has started
  plane.store(0, 0.0f);
  cluster_arrive();
  RowAhead rows{steps, on ? i : -1, n_steps, -1, plane.local};
  rows.start(n_steps);  // an empty row, then step n_steps - 1
  MfNode x1{};
  float q1 = 0.0f, e1 = 0.0f, g1 = 0.0f;
  auto load_step = [&](int32_t t) {
    if (t < 0) return;
    g1 = __ldg(ginc + t);
    if (!on) return;
    const float *x = states + (size_t)t * 4 * N + i;
    x1 = MfNode{__ldg(x), __ldg(x + N), __ldg(x + 2 * N), __ldg(x + 3 * N)};
    q1 = __ldg(qv + (size_t)t * N + i);
    e1 = __ldg(ev + (size_t)t * N + i);
  };
  load_step(n_steps - 1);
  double gb = 0.0, ge = 0.0, gi = 0.0, gr = 0.0;
  uint32_t buf = 0;
  for (int32_t t = n_steps - 1; t >= 0; --t, buf ^= 1) {
    const MfNode x = x1;
    const float q = q1, es = e1, g = g1;
    load_step(t - 1);
    rows.advance(t + 1);
    const float scale = rows.s1.scale;  // of step t
    cluster_wait();
    y.I = __fadd_rn(y.I, rows.exposure(buf * (uint32_t)sizeof(s_plane[0])));
    const MfNode full = y;
    const float suq = mf_node_adjoint(r, x, q, g, y);
    plane.store((buf ^ 1) * (uint32_t)sizeof(s_plane[0]), suq * r.beta * si * scale);
    cluster_arrive();
    gs = fmaf(__fmul_rn(suq, r.beta), es, gs);
    rate_terms(r, x, full, suq, si, es, gb, ge, gi, gr);
  }
  rows.advance(0);
  cluster_wait();
  y.I = __fadd_rn(y.I, rows.exposure(buf * (uint32_t)sizeof(s_plane[0])));
  cluster_arrive();
  if (on) {
    gx0[i] = y.S;
    gx0[N + i] = y.E;
    gx0[2 * N + i] = y.I;
    gx0[3 * N + i] = y.R;
    gsus[i] = gs;
  }
  gb = warp_sum(gb);
  ge = warp_sum(ge);
  gi = warp_sum(gi);
  gr = warp_sum(gr);
  if ((threadIdx.x & 31) == 0 && (i >> 5) < nwarp) {
    double2 *p = reinterpret_cast<double2 *>(gpart + 4 * (size_t)(i >> 5));
    p[0] = make_double2(gb, ge);
    p[1] = make_double2(gi, gr);
  }
  cluster_wait();
}

// What k_mf_forward leaves to all SMs: exp(-beta s e) of every step for the
// adjoint and the warps' incidence sums, from the kept states and exposures.
__global__ void __launch_bounds__(kMfThreads)
    k_mf_after(int32_t n, int32_t blocks, const MfRates *__restrict__ rates,
               const float *__restrict__ sus, const float *__restrict__ states,
               const float *__restrict__ ev, float *__restrict__ qv, float *__restrict__ inc_part) {
  const MfRates r = *rates;
  const int32_t t = blockIdx.x / blocks, i = (blockIdx.x % blocks) * kMfThreads + threadIdx.x;
  float newinf = 0.0f;
  if (i < n) {
    MfNode v{states[(size_t)t * 4 * n + i], 0.0f, 0.0f, 0.0f};
    newinf = mf_node_step(r, __ldg(sus + i), ev[(size_t)t * n + i], v, qv[(size_t)t * n + i]);
  }
  const float tot = warp_sum(newinf);
  if ((threadIdx.x & 31) == 0) inc_part[(size_t)t * blocks * kMfWarps + (i >> 5)] = tot;
}

// The four rate gradients: one warp each, lanes over the warp partials.
__global__ void k_mf_finish(const double *__restrict__ gpart, int32_t nwarp,
                            double *__restrict__ out) {
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = 0.0;
  for (int32_t b = lane; b < nwarp; b += 32) s += gpart[4 * (size_t)b + k];
  s = warp_sum(s);
  if (lane == 0) out[k] = s;
}

// Launches after another of this file's kernels may start early (dependent
// launch); `after_kernel` is false after a copy or a memset.
template <typename... Params, typename... Args>
void mf_launch(void (*kernel)(Params...), int grid, bool after_kernel, cudaStream_t st,
               Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kMfThreads);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = after_kernel ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

int mf_grid(int32_t n) { return (n + kMfThreads - 1) / kMfThreads; }

}  // namespace

int32_t mf_warps(int32_t n) { return mf_grid(n) * kMfWarps; }

void mf_step(const int32_t *rp, const int2 *ent, int32_t n, float scale, const MfRates *r,
             const float *sus, const float *x, float *xo, float *q_out, float *e_out,
             float *inc_part, bool after_kernel, cudaStream_t st) {
  mf_launch(k_mf_step, mf_grid(n), after_kernel, st, rp, ent, n, scale, r, sus, x, xo, q_out,
            e_out, inc_part);
}

void mf_incidence(const float *part, int32_t nwarp, int32_t T, float *inc, cudaStream_t st) {
  if (T <= 0) return;
  k_mf_incidence<<<(T + kMfWarps - 1) / kMfWarps, kMfThreads, 0, st>>>(part, nwarp, T, inc);
}

void mf_adjoint(int32_t n, const int32_t *rp_c, const int2 *ent_c, const float *z_in,
                const float *a_in, const float *x, const float *q, const float *e,
                const float *ginc, int32_t tl, float scale, const MfRates *r, const float *sus,
                float *a_out, float *z_out, float *gsus, double *gpart, bool early,
                bool after_kernel, cudaStream_t st) {
  mf_launch(k_mf_adjoint, mf_grid(n), after_kernel, st, n, rp_c, ent_c, z_in, a_in, x, q, e, ginc,
            tl, scale, r, sus, a_out, z_out, gsus, gpart, (int32_t)early);
}

// One cluster: eight blocks of the fewest warps that hold the nodes.
static int cluster_threads(int32_t n) { return (n + 32 * kMfCluster - 1) / (32 * kMfCluster) * 32; }
void mf_forward_cluster(const MfStep *steps, int32_t n_steps, int32_t n, const MfRates *r,
                        const float *sus, float *states, float *q, float *e, float *inc_part,
                        cudaStream_t st) {
  const int threads = cluster_threads(n);
  k_mf_forward<<<kMfCluster, threads, 0, st>>>(steps, n_steps, n, r, sus,
                                               states, e);
  const int blocks = mf_grid(n);
  k_mf_after<<<(unsigned)n_steps * blocks, kMfThreads, 0, st>>>(n, blocks, r, sus, states, e, q,
                                                                inc_part);
}

void mf_reverse_cluster(const MfStep *steps, int32_t n_steps, int32_t n, const MfRates *r,
                        const float *sus, const float *a_in, const float *states, const float *q,
                        const float *e, const float *ginc, float *gx0, float *gsus, double *gpart,
                        cudaStream_t st) {
  const int threads = cluster_threads(n);
  k_mf_reverse<<<kMfCluster, threads, 0, st>>>(steps, n_steps, n, r, sus,
                                               a_in, states, q, e, ginc, gx0, gsus, gpart,
                                               mf_warps(n));
}

void mf_finish(const double *gpart, int32_t nwarp, double *out, cudaStream_t st) {
  k_mf_finish<<<1, 128, 0, st>>>(gpart, nwarp, out);
}

}  // namespace rp
