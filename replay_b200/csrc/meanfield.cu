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
// and 5.1 us reverse now; N = 2,000 4.3 us before, 1.7 and 2.8 us now.
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
    const float S = __ldcg(x + i), E = __ldcg(x + n + i), I = __ldcg(x + 2 * (size_t)n + i),
                R = __ldcg(x + 3 * (size_t)n + i);
    const float es = row_exposure(h, ent, x + 2 * (size_t)n) * scale;
    const float a = r.beta * si * es;
    const float P = -expm1f(-a), q = expf(-a);
    newinf = S * P;
    const float f_ei = r.has_exposed ? E * r.p_ei : 0.0f;
    const float f_i = I * r.p_ir, f_rs = R * r.p_rs;
    float S2 = S * q + f_rs, E2 = E - f_ei, I2 = I - f_i + f_ei, R2 = R - f_rs;
    if (r.has_exposed) E2 += newinf; else I2 += newinf;
    if (r.ir_to_s) S2 += f_i; else R2 += f_i;
    xo[i] = S2;
    xo[n + i] = E2;
    xo[2 * (size_t)n + i] = I2;
    xo[3 * (size_t)n + i] = R2;
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
  float S = 0, E = 0, I = 0, R = 0, q = 0, es = 0, si = 1.0f, g = 0;
  auto load_step = [&]() {
    S = __ldcg(x + i), E = __ldcg(x + n + i), I = __ldcg(x + 2 * (size_t)n + i),
    R = __ldcg(x + 3 * (size_t)n + i);
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
    const float yS = __ldcg(a_in + i), yE = __ldcg(a_in + n + i),
                yR = __ldcg(a_in + 3 * (size_t)n + i);
    float yI = __ldcg(a_in + 2 * (size_t)n + i);
    if (x && !early) load_step();
    if (x && ginc) g = __ldcg(ginc + tl);  // dL/dincidence of step tl
    const float gs0 = x && gsus ? __ldcg(gsus + i) : 0.0f;
    if (rp_c) yI += row_exposure(h, ent_c, z_in);
    if (!x) {
      a_out[i] = yS;
      a_out[n + i] = yE;
      a_out[2 * (size_t)n + i] = yI;
      a_out[3 * (size_t)n + i] = yR;
    } else {
      const float P = 1.0f - q;
      const float yX = r.has_exposed ? yE : yI;
      const float yY = r.ir_to_s ? yS : yR;
      const float u = yX - yS + g;
      const float suq = S * u * q;
      a_out[i] = yS + P * u;
      a_out[n + i] = r.has_exposed ? yE + r.p_ei * (yI - yE) : yE;
      a_out[2 * (size_t)n + i] = yI + r.p_ir * (yY - yI);
      a_out[3 * (size_t)n + i] = yR + r.p_rs * (yS - yR);
      // d(es_i)/dI_j = scale w_ij, so z_i = scale * S u q beta s_i
      z_out[i] = suq * r.beta * si * scale;
      if (gsus) gsus[i] = gs0 + suq * r.beta * es;
      gb = (double)suq * (double)si * (double)es;
      if (r.has_exposed) ge = (double)E * ((double)yI - (double)yE);
      gi = (double)I * ((double)yY - (double)yI);
      gr = (double)R * ((double)yS - (double)yR);
    }
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

void mf_finish(const double *gpart, int32_t nwarp, double *out, cudaStream_t st) {
  k_mf_finish<<<1, 128, 0, st>>>(gpart, nwarp, out);
}

}  // namespace rp
