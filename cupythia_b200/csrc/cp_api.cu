// cp_api.cu -- handles, errors, the counter-RNG surface, the batched SigmaProcess surface and
// the partonic gg -> gg kernels.
#include <math.h>
#include <string.h>
#include <mutex>
#include "cp_internal.cuh"

int cp_had_launch_shape(cp_handle* h);

// ------------------------------------------------------------------------------------------
// errors and scratch
// ------------------------------------------------------------------------------------------
int cp_fail(cp_handle* h, int code, const std::string& msg)
{
  if (h) h->err = msg;
  return code;
}

int cp_fail_cuda(cp_handle* h, cudaError_t e, const char* what)
{
  if (h) h->err = std::string(what) + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? CP_ERR_NOMEM : CP_ERR_CUDA;
}

// Workspaces that grow: the capacity is zero from the moment the old block goes until the new one is there, so a
// growth that fails leaves a workspace that the next call allocates, not one that counts as large and is null.
int cp_ensure_slots(cp_handle* h, size_t doubles)
{
  if (doubles <= h->slots_cap) return CP_OK;
  if (h->d_slots) {
    CP_CUDA(h, cudaStreamSynchronize(h->stream));
    CP_CUDA(h, cudaFree(h->d_slots));
    h->d_slots = nullptr;
    h->slots_cap = 0;
  }
  CP_CUDA(h, cudaMalloc(&h->d_slots, doubles * sizeof(double)));
  h->slots_cap = doubles;
  return CP_OK;
}

int cp_ensure_iters(cp_handle* h, int n)
{
  if (n <= h->iters_cap) return CP_OK;
  if (h->h_iters) {
    CP_CUDA(h, cudaStreamSynchronize(h->stream));
    CP_CUDA(h, cudaFreeHost(h->h_iters));
    h->h_iters = nullptr;
    h->iters_cap = 0;
  }
  CP_CUDA(h, cudaHostAlloc(&h->h_iters, sizeof(CpIterDev) * (size_t)n, cudaHostAllocMapped | cudaHostAllocPortable));
  h->iters_cap = n;
  return CP_OK;
}

int cp_ensure_losses(cp_handle* h, int n)
{
  if (n <= h->losses_cap) return CP_OK;
  if (h->h_losses) {
    CP_CUDA(h, cudaStreamSynchronize(h->stream));
    CP_CUDA(h, cudaFreeHost(h->h_losses));
    h->h_losses = nullptr;
    h->losses_cap = 0;
  }
  CP_CUDA(h, cudaHostAlloc(&h->h_losses, sizeof(double) * (size_t)n, cudaHostAllocMapped | cudaHostAllocPortable));
  h->losses_cap = n;
  return CP_OK;
}

static int ensure_kin(cp_handle* h, int64_t n)
{
  if (n <= h->kin_cap) return CP_OK;
  float** bufs[8] = {&h->d_x1, &h->d_x2, &h->d_sH, &h->d_tH, &h->d_uH, &h->d_as, &h->d_q2r, &h->d_q2f};
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  h->kin_cap = h->kin_n = 0;   // the batch goes with its arrays
  for (auto b : bufs) {
    if (*b) CP_CUDA(h, cudaFree(*b));
    *b = nullptr;
  }
  for (auto b : bufs) CP_CUDA(h, cudaMalloc(b, sizeof(float) * (size_t)n));
  h->kin_cap = n;
  return CP_OK;
}

// ------------------------------------------------------------------------------------------
// handles
// ------------------------------------------------------------------------------------------
extern "C" int cp_abi_version(void) { return CP_ABI_VERSION; }

extern "C" int cp_config_default(cp_config* c)
{
  if (!c) return CP_ERR_INVALID;
  memset(c, 0, sizeof *c);
  c->sqrt_s = 13000.0;
  c->pt_hat_min = 20.0;
  c->alphas_mz = 0.13;
  c->k_ren = 1.0;
  c->k_fac = 1.0;
  c->convert2mb = 0.389380;
  c->n_quark_in = 5;
  c->n_quark_new = 3;
  c->proc_mask = CP_PROC_ALL;
  c->n_bins = 50;
  c->device = 0;
  c->seed = 42;
  return CP_OK;
}

static int apply_config(cp_handle* h, const cp_config* c)
{
  if (c->n_bins < 2 || c->n_bins > CP_MAX_BINS)
    return cp_fail(h, CP_ERR_INVALID, "n_bins must be in [2, 128]");
  if ((c->proc_mask & ~CP_PROC_ALL) || c->proc_mask == 0)
    return cp_fail(h, CP_ERR_INVALID, "proc_mask must be a nonzero OR of CP_PROC_*");
  CpHadConfig hc{c->sqrt_s, c->pt_hat_min, c->alphas_mz, c->k_ren, c->k_fac, c->convert2mb,
                 c->n_quark_in, c->n_quark_new, c->proc_mask};
  if (cp_build_had_params(hc, h->P))
    return cp_fail(h, CP_ERR_INVALID,
                   "unsupported configuration (need pT_hat_min >= 2 GeV, 2 pT_hat_min < sqrt_s, "
                   "0.05 < alphas_mz < 0.3, positive scale factors, n_quark_in == 5)");
  h->cfg = *c;
  h->nb = c->n_bins;
  return CP_OK;
}

// A page of pinned memory per device, held from its first handle to the end of the process and never read or
// written.  The driver maps a chunk for a process's first pinned allocation and unmaps it with the last one, 1 to 3
// and 0.4 ms, and serves the others from it in about a microsecond: with the page, handles that come and go one after
// another cost 0.05 ms each instead of 3.  Failure to get it costs that time alone.
static void hold_pinned_chunk(int device)
{
  static std::mutex mutex;
  static void* page[64];
  if (device >= 64) return;
  std::lock_guard<std::mutex> lock(mutex);
  if (!page[device] &&
      cudaHostAlloc(&page[device], 4096, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
    page[device] = nullptr;
    cudaGetLastError();
  }
}

extern "C" int cp_create(const cp_config* cfg, cp_handle** out)
{
  if (!out) return CP_ERR_INVALID;
  *out = nullptr;
  cp_config def;
  cp_config_default(&def);
  if (!cfg) cfg = &def;
  cp_handle* h = new cp_handle();
  int rc = apply_config(h, cfg);
  if (rc) { delete h; return rc; }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { delete h; return CP_ERR_CUDA; }
  if (cfg->device < 0 || cfg->device >= ndev) { delete h; return CP_ERR_INVALID; }
  h->device = cfg->device;
  CpDeviceGuard guard(h->device);
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess || cur != h->device) { delete h; return CP_ERR_CUDA; }
  cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, h->device);
  hold_pinned_chunk(h->device);
  bool ok = cudaHostAlloc(&h->mail, sizeof(CpMail), cudaHostAllocMapped | cudaHostAllocPortable) == cudaSuccess &&
            cudaMalloc(&h->d_edges, sizeof(double) * 3 * (CP_MAX_BINS + 1)) == cudaSuccess &&
            cudaMalloc(&h->d_red, sizeof(double) * (CP_SLOT_HEAD + 3 * CP_MAX_BINS)) == cudaSuccess &&
            cudaMalloc(&h->d_qhist, sizeof(unsigned long long) * CP_QBINS) == cudaSuccess &&
            cudaMalloc(&h->d_wmax, sizeof(double) * 2) == cudaSuccess &&
            cudaMalloc(&h->d_counter, sizeof(unsigned long long) * 2) == cudaSuccess &&
            cudaMemset(h->d_wmax, 0, sizeof(double) * 2) == cudaSuccess &&
            cudaMalloc(&h->d_cteq, sizeof(CpCteqPoly) * 8) == cudaSuccess &&
            cudaMemcpy(h->d_cteq, h->P.cteq, sizeof(CpCteqPoly) * 8, cudaMemcpyHostToDevice) == cudaSuccess;
  if (h->mail) memset(h->mail, 0, sizeof(CpMail));
  if (!ok || cp_had_launch_shape(h) != CP_OK || cp_ensure_iters(h, 16) != CP_OK) {
    cp_destroy(h);
    return CP_ERR_NOMEM;
  }
  rc = cp_grid_reset(h);
  if (rc) { cp_destroy(h); return rc; }
  *out = h;
  return CP_OK;
}

extern "C" int cp_destroy(cp_handle* h)
{
  if (!h) return CP_OK;
  CpDeviceGuard guard(h->device);
  // kernels in flight write to the pinned memory below (a null stream is the default one, and can be busy as well)
  cudaStreamSynchronize(h->stream);
  if (h->gen_copy) cudaStreamSynchronize(h->gen_copy);
  for (cudaEvent_t e : h->tpool) cudaEventDestroy(e);
  for (int k = 0; k < CP_GEN_BUFS; ++k) {
    if (h->gen_counted[k]) cudaEventDestroy(h->gen_counted[k]);
    if (h->gen_copied[k]) cudaEventDestroy(h->gen_copied[k]);
  }
  if (h->gen_copy) cudaStreamDestroy(h->gen_copy);
  void* pinned[] = {h->h_gen_cnt, h->h_gen_red, h->h_iters, h->h_losses, h->mail};
  for (void* b : pinned)
    if (b) cudaFreeHost(b);
  void* bufs[] = {h->d_edges, h->d_slots, h->d_red, h->d_x1, h->d_x2, h->d_sH,
                  h->d_tH, h->d_uH, h->d_as, h->d_q2r, h->d_q2f, h->d_qhist, h->d_wmax, h->d_counter, h->d_cteq, h->d_flow, h->d_flow_pk,
                  h->d_flow_bias, h->d_flow_buf, h->d_flow_tc, h->d_flow_ticket, h->d_staging,
                  h->d_gen_stage, h->d_ftrain, h->d_adj};
  for (void* b : bufs)
    if (b) cudaFree(b);
  delete h;
  return CP_OK;
}

extern "C" const char* cp_last_error(const cp_handle* h) { return h ? h->err.c_str() : "null handle"; }

// Offset of this handle's point indices (cuPythia/common/rng.cuh:5-19: shard i of M points per
// shard works on the global points [i M, i M + count)); every pass then draws the Philox block of
// global point offset + p, so shards are disjoint and their union is the single-device run.
extern "C" int cp_set_point_offset(cp_handle* h, uint64_t offset)
{
  CP_CHECK_HANDLE(h);
  h->point_offset = offset;
  return CP_OK;
}

extern "C" int cp_set_stream(cp_handle* h, void* s)
{
  CP_CHECK_HANDLE(h);
  h->stream = (cudaStream_t)s;
  return CP_OK;
}

extern "C" int cp_synchronize(cp_handle* h)
{
  CP_CHECK_HANDLE(h);
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_device_sm_count(cp_handle* h, int* n)
{
  CP_CHECK_HANDLE(h);
  if (!n) return CP_ERR_INVALID;
  *n = h->num_sms;
  return CP_OK;
}

// ------------------------------------------------------------------------------------------
// grid
// ------------------------------------------------------------------------------------------
extern "C" int cp_grid_reset(cp_handle* h)
{
  CP_CHECK_HANDLE(h);
  double e[3 * (CP_MAX_BINS + 1)];
  for (int d = 0; d < 3; ++d)
    for (int k = 0; k <= h->nb; ++k) e[d * (h->nb + 1) + k] = (double)k / (double)h->nb;
  return cp_grid_set(h, e);
}

extern "C" int cp_grid_set(cp_handle* h, const double* e)
{
  CP_CHECK_HANDLE(h);
  if (!e) return cp_fail(h, CP_ERR_INVALID, "cp_grid_set: null edges");
  const int nb = h->nb;
  for (int d = 0; d < 3; ++d) {
    const double* ed = e + d * (nb + 1);
    if (ed[0] != 0.0 || ed[nb] != 1.0) return cp_fail(h, CP_ERR_INVALID, "grid must span [0, 1]");
    for (int k = 0; k < nb; ++k)
      if (!(ed[k + 1] > ed[k])) return cp_fail(h, CP_ERR_INVALID, "grid edges must increase");
  }
  CP_CUDA(h, cudaMemcpyAsync(h->d_edges, e, sizeof(double) * 3 * (nb + 1), cudaMemcpyHostToDevice,
                             h->stream));
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_grid_get(cp_handle* h, double* e)
{
  CP_CHECK_HANDLE(h);
  if (!e) return cp_fail(h, CP_ERR_INVALID, "cp_grid_get: null edges");
  CP_CUDA(h, cudaMemcpyAsync(e, h->d_edges, sizeof(double) * 3 * (h->nb + 1), cudaMemcpyDeviceToHost,
                             h->stream));
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

// ------------------------------------------------------------------------------------------
// counter RNG surface
// ------------------------------------------------------------------------------------------
__global__ void k_philox_words(uint64_t seed, uint64_t p0, uint64_t n, uint32_t iter, uint32_t stream,
                               uint4* out)
{
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t w[4];
    cp_point_words(seed, p0 + i, iter, stream, w);
    out[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__device__ __forceinline__ double cp_u01(uint64_t u) { return (double)(u >> 11) * (1.0 / 9007199254740992.0); }

__global__ void k_splitmix(uint64_t seed, uint64_t nthr, uint64_t kper, double* out)
{
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nthr;
       t += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t ctr = seed + t * 0x100000001B3ULL;
    for (uint64_t i = 0; i < kper; ++i) out[t * kper + i] = cp_u01(cp_splitmix64(ctr++));
  }
}

__global__ void k_event_keys(uint64_t base, uint64_t e0, uint64_t n, uint64_t* out)
{
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = cp_splitmix64(base ^ ((e0 + i) * 0x9E3779B97F4A7C15ULL));
}

static int grid_for(cp_handle* h, uint64_t n)
{
  uint64_t b = (n + 255) / 256;
  uint64_t cap = (uint64_t)h->num_sms * 32;
  return (int)(b < cap ? (b > 0 ? b : 1) : cap);
}

extern "C" int cp_philox_words(cp_handle* h, uint64_t seed, uint64_t p0, uint64_t n, uint32_t iter,
                               uint32_t stream, uint32_t* out)
{
  CP_CHECK_HANDLE(h);
  if (n && !out) return cp_fail(h, CP_ERR_INVALID, "cp_philox_words: null output");
  if (((uintptr_t)out & 15) != 0) return cp_fail(h, CP_ERR_INVALID, "cp_philox_words: output must be 16-byte aligned");
  if (!n) return CP_OK;
  k_philox_words<<<grid_for(h, n), 256, 0, h->stream>>>(seed, p0, n, iter, stream, (uint4*)out);
  CP_LAUNCH_CHECK(h, "k_philox_words");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_splitmix_uniforms(cp_handle* h, uint64_t seed, uint64_t nthr, uint64_t kper, double* out)
{
  CP_CHECK_HANDLE(h);
  if (nthr && kper && !out) return cp_fail(h, CP_ERR_INVALID, "cp_splitmix_uniforms: null output");
  if (!nthr || !kper) return CP_OK;
  k_splitmix<<<grid_for(h, nthr), 256, 0, h->stream>>>(seed, nthr, kper, out);
  CP_LAUNCH_CHECK(h, "k_splitmix");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_event_keys(cp_handle* h, uint64_t base, uint64_t e0, uint64_t n, uint64_t* out)
{
  CP_CHECK_HANDLE(h);
  if (n && !out) return cp_fail(h, CP_ERR_INVALID, "cp_event_keys: null output");
  if (!n) return CP_OK;
  k_event_keys<<<grid_for(h, n), 256, 0, h->stream>>>(base, e0, n, out);
  CP_LAUNCH_CHECK(h, "k_event_keys");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

// ------------------------------------------------------------------------------------------
// SigmaProcess surface
// ------------------------------------------------------------------------------------------
__global__ void k_set2kin(const CpHadParams P, int64_t n, const float* __restrict__ sH,
                          const float* __restrict__ tH, float* uH, float* as, float* q2r, float* q2f)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float s = sH[i], t = tH[i], u = -(s + t);
    float pT2 = t * u / s;
    float qr = P.kR * pT2, qf = P.kF * pT2;
    uH[i] = u;
    q2r[i] = qr;
    q2f[i] = qf;
    as[i] = cp_alphas(P, qr);
  }
}

// The same from FP64 kinematics (what Pythia's set2Kin receives): uHat = -(sHat + tHat) and
// pT^2 = tHat uHat / sHat are formed in FP64 and only then rounded, so a small |uHat| (a large
// sHat near the pT cut, where the FP32 sum of sHat and tHat would cancel) keeps its precision.
__global__ void k_set2kin_f64(const CpHadParams P, int64_t n, const double* __restrict__ x1d,
                              const double* __restrict__ x2d, const double* __restrict__ sHd,
                              const double* __restrict__ tHd, float* x1, float* x2, float* sH, float* tH,
                              float* uH, float* as, float* q2r, float* q2f)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double s = sHd[i], t = tHd[i], u = -(s + t);
    const float pT2 = (float)(t * u / s);
    const float qr = P.kR * pT2, qf = P.kF * pT2;
    x1[i] = (float)x1d[i];
    x2[i] = (float)x2d[i];
    sH[i] = (float)s;
    tH[i] = (float)t;
    uH[i] = (float)u;
    q2r[i] = qr;
    q2f[i] = qf;
    as[i] = cp_alphas(P, qr);
  }
}

// which: 0 = sigmaKin of code (flavour independent), 1 = sigmaHat(id1, id2), 2 = sigmaPDF(mask)
__global__ void k_sigma(const CpHadParams P, const CpCteqPoly* cteq_g, int64_t n, int which, int code,
                        int id1, int id2, int mask, const float* __restrict__ x1,
                        const float* __restrict__ x2, const float* __restrict__ sH,
                        const float* __restrict__ tH, const float* __restrict__ uH,
                        const float* __restrict__ as, const float* __restrict__ q2f, float* out)
{
  __shared__ CpCteqPoly cteq[8];
  cp_stage_cteq(cteq, cteq_g);
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float s = sH[i], t = tH[i], u = uH[i];
    float tp = t / s, up = u / s;
    CpBrackets b;
    cp_brackets(P, tp, up, b);
    float a = as[i];
    float pref = CP_PI_F * (a * a) / (s * s);   // dsigma/dtHat = pref * bracket
    float v;
    if (which == 2) {
      float m[5];
      for (int k = 0; k < 5; ++k) m[k] = (mask >> k) & 1 ? 1.f : 0.f;
      float fa[8], fb[8];
      cp_cteq_pair<1>(cteq, q2f[i], logf(x1[i]), 0.f, logf(x2[i]), 0.f, fa, fb);
      b.qqD = cp_addr(cp_addr(b.qqU, b.qqTU), -b.qqT);   // each term rounded, as in sigmaHat
      v = P.conv * pref * cp_channel_sum(m, b, fa, fb);
    } else {
      float br = 0.f;
      if (code == 111) br = b.gg2gg;
      else if (code == 112) br = b.gg2qqbar;
      else if (code == 113) br = b.qg2qg;
      else if (code == 115) br = b.qqbar2gg;
      else if (code == 114) {
        if (id2 == id1) br = 0.5f * (b.qqT + b.qqU + b.qqTU);
        else if (id2 == -id1) br = b.qqT + b.qqST;
        else br = b.qqT;
      }
      v = pref * br;
    }
    out[i] = v;
  }
}

// pickInState + setIdColAcol of one process over the stored batch: per point the uniforms
// r = (pair, new flavour, colour topology, gg -> gg orientation); PDFs at Q2Fac of the batch.
__global__ void k_pick_state(const CpHadParams P, const CpCteqPoly* cteq_g, int64_t n, int k,
                             const float* __restrict__ x1, const float* __restrict__ x2,
                             const float* __restrict__ sH, const float* __restrict__ tH,
                             const float* __restrict__ uH, const float* __restrict__ q2f,
                             const float4* __restrict__ r,
                             short4* __restrict__ ids, uint16_t* __restrict__ colour)
{
  __shared__ CpCteqPoly cteq[8];
  cp_stage_cteq(cteq, cteq_g);
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float s = sH[i], t = tH[i], u = uH[i];
    const float tp = t / s, up = u / s;
    CpPoint pt;
    cp_brackets(P, tp, up, pt.b);
    cp_cteq_pair<1>(cteq, q2f[i], logf(x1[i]), 0.f, logf(x2[i]), 0.f, pt.fa, pt.fb);
    const float4 ri = r[i];
    int id[4];
    cp_pick_pair(P, k, pt, ri.x, ri.y, id);
    ids[i] = make_short4((short)id[0], (short)id[1], (short)id[2], (short)id[3]);
    colour[i] = (uint16_t)cp_colour_flow(111 + k, id, tp, up, ri.z, ri.w);
  }
}

__global__ void k_pdf(const CpCteqPoly* cteq_g, int64_t n, const float* __restrict__ x,
                      const float* __restrict__ q2, float* out)
{
  __shared__ CpCteqPoly cteq[8];
  cp_stage_cteq(cteq, cteq_g);
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float f[8], g[8];
    float lx = logf(x[i]);
    cp_cteq_pair<1>(cteq, q2[i], lx, 0.f, lx, 0.f, f, g);
    // id order -5..-1, 1..5, 21; f = {d, u, g, ubar, dbar, s, c, b}
    float* o = out + 11 * i;
    o[0] = f[7]; o[1] = f[6]; o[2] = f[5]; o[3] = f[3]; o[4] = f[4];
    o[5] = f[0]; o[6] = f[1]; o[7] = f[5]; o[8] = f[6]; o[9] = f[7]; o[10] = f[2];
  }
}

extern "C" int cp_set2kin_batch(cp_handle* h, const float* x1, const float* x2, const float* sH,
                                const float* tH, int64_t n)
{
  CP_CHECK_HANDLE(h);
  if (n < 0 || (n > 0 && (!x1 || !x2 || !sH || !tH)))
    return cp_fail(h, CP_ERR_INVALID, "cp_set2kin_batch: bad arguments");
  int rc = ensure_kin(h, n > 0 ? n : 1);
  if (rc) return rc;
  h->kin_n = n;
  if (!n) return CP_OK;
  size_t bytes = sizeof(float) * (size_t)n;
  CP_CUDA(h, cudaMemcpyAsync(h->d_x1, x1, bytes, cudaMemcpyDeviceToDevice, h->stream));
  CP_CUDA(h, cudaMemcpyAsync(h->d_x2, x2, bytes, cudaMemcpyDeviceToDevice, h->stream));
  CP_CUDA(h, cudaMemcpyAsync(h->d_sH, sH, bytes, cudaMemcpyDeviceToDevice, h->stream));
  CP_CUDA(h, cudaMemcpyAsync(h->d_tH, tH, bytes, cudaMemcpyDeviceToDevice, h->stream));
  k_set2kin<<<grid_for(h, n), 256, 0, h->stream>>>(h->P, n, h->d_sH, h->d_tH, h->d_uH, h->d_as, h->d_q2r, h->d_q2f);
  CP_LAUNCH_CHECK(h, "k_set2kin");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_set2kin_batch_f64(cp_handle* h, const double* x1, const double* x2, const double* sH,
                                    const double* tH, int64_t n)
{
  CP_CHECK_HANDLE(h);
  if (n < 0 || (n > 0 && (!x1 || !x2 || !sH || !tH)))
    return cp_fail(h, CP_ERR_INVALID, "cp_set2kin_batch_f64: bad arguments");
  int rc = ensure_kin(h, n > 0 ? n : 1);
  if (rc) return rc;
  h->kin_n = n;
  if (!n) return CP_OK;
  k_set2kin_f64<<<grid_for(h, n), 256, 0, h->stream>>>(h->P, n, x1, x2, sH, tH, h->d_x1, h->d_x2, h->d_sH, h->d_tH,
                                                       h->d_uH, h->d_as, h->d_q2r, h->d_q2f);
  CP_LAUNCH_CHECK(h, "k_set2kin_f64");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

static int sigma_launch(cp_handle* h, int which, int code, int id1, int id2, int mask, float* out)
{
  if (h->kin_n == 0) return CP_OK;
  if (!out) return cp_fail(h, CP_ERR_INVALID, "null output");
  k_sigma<<<grid_for(h, h->kin_n), 256, 0, h->stream>>>(h->P, h->d_cteq, h->kin_n, which, code, id1, id2, mask,
                                                         h->d_x1, h->d_x2, h->d_sH, h->d_tH, h->d_uH,
                                                         h->d_as, h->d_q2f, out);
  CP_LAUNCH_CHECK(h, "k_sigma");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_sigma_kin_batch(cp_handle* h, int code, float* out)
{
  CP_CHECK_HANDLE(h);
  if (code != 111 && code != 112 && code != 113 && code != 115)
    return cp_fail(h, CP_ERR_INVALID,
                   "cp_sigma_kin_batch: codes 111, 112, 113, 115 (114 depends on the flavour pair: "
                   "use cp_sigma_hat_batch)");
  return sigma_launch(h, 0, code, 0, 0, 0, out);
}

extern "C" int cp_sigma_hat_batch(cp_handle* h, int code, int id1, int id2, float* out)
{
  CP_CHECK_HANDLE(h);
  if (code < 111 || code > 115) return cp_fail(h, CP_ERR_INVALID, "cp_sigma_hat_batch: code 111..115");
  return sigma_launch(h, 1, code, id1, id2, 0, out);
}

extern "C" int cp_sigma_pdf_batch(cp_handle* h, int mask, float* out)
{
  CP_CHECK_HANDLE(h);
  if ((mask & ~CP_PROC_ALL) || !mask) return cp_fail(h, CP_ERR_INVALID, "cp_sigma_pdf_batch: bad mask");
  return sigma_launch(h, 2, 0, 0, 0, mask, out);
}

extern "C" int cp_pick_state_batch(cp_handle* h, int code, const float* r_dev, int16_t* ids_dev, uint16_t* colour_dev)
{
  CP_CHECK_HANDLE(h);
  if (code < 111 || code > 115) return cp_fail(h, CP_ERR_INVALID, "cp_pick_state_batch: code 111..115");
  if (!h->kin_n) return CP_OK;
  if (!r_dev || !ids_dev || !colour_dev || ((uintptr_t)r_dev & 15) || ((uintptr_t)ids_dev & 7))
    return cp_fail(h, CP_ERR_INVALID, "cp_pick_state_batch: r (16-byte aligned) and ids (8-byte aligned) required");
  k_pick_state<<<grid_for(h, h->kin_n), 256, 0, h->stream>>>(h->P, h->d_cteq, h->kin_n, code - 111, h->d_x1, h->d_x2,
                                                             h->d_sH, h->d_tH, h->d_uH, h->d_q2f,
                                                             reinterpret_cast<const float4*>(r_dev),
                                                             reinterpret_cast<short4*>(ids_dev), colour_dev);
  CP_LAUNCH_CHECK(h, "k_pick_state");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_scales_batch(cp_handle* h, float* as, float* q2r, float* q2f)
{
  CP_CHECK_HANDLE(h);
  size_t bytes = sizeof(float) * (size_t)h->kin_n;
  if (!h->kin_n) return CP_OK;
  if (as) CP_CUDA(h, cudaMemcpyAsync(as, h->d_as, bytes, cudaMemcpyDeviceToDevice, h->stream));
  if (q2r) CP_CUDA(h, cudaMemcpyAsync(q2r, h->d_q2r, bytes, cudaMemcpyDeviceToDevice, h->stream));
  if (q2f) CP_CUDA(h, cudaMemcpyAsync(q2f, h->d_q2f, bytes, cudaMemcpyDeviceToDevice, h->stream));
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_pdf_batch(cp_handle* h, const float* x, const float* q2, int64_t n, float* out)
{
  CP_CHECK_HANDLE(h);
  if (n < 0 || (n > 0 && (!x || !q2 || !out))) return cp_fail(h, CP_ERR_INVALID, "cp_pdf_batch: bad arguments");
  if (!n) return CP_OK;
  k_pdf<<<grid_for(h, n), 256, 0, h->stream>>>(h->d_cteq, n, x, q2, out);
  CP_LAUNCH_CHECK(h, "k_pdf");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

// ------------------------------------------------------------------------------------------
// partonic gg -> gg, FP64 (cuPythia/03_fused_resident_me/fused_gg2gg.cu:28-51)
// ------------------------------------------------------------------------------------------
struct PartonicArgs {
  double s, aS, cMax, scale;  // scale = (2 cMax)(s/2) conv
  uint64_t seed, p0, n;       // Philox mode: points; SplitMix mode: reference threads
  uint64_t kper;              // SplitMix mode: draws per reference thread
  double* slots;              // gridDim.x * 4
  double* w_out;
};

// Sigma2gg2gg::sigmaKin (pythia8317/src/SigmaQCD.cc:115-129; pipeline/physics.cuh:9-16) for a fixed
// s-hat.  With s + t + u = 0 the three brackets sigTS + sigUS + sigTU sum to the textbook form
// (9/2) (3 - t u / s^2 - s u / t^2 - s t / u^2) of the g g -> g g matrix element.  With
// t = -s (1 - c) / 2, u = -s (1 + c) / 2 and p = 1 - c^2 = 4 t u / s^2 it depends on p alone,
//   s u / t^2 + s t / u^2 = s (t^3 + u^3) / (t u)^2 = -s^2 (s^2 - 3 t u) / (t u)^2
//                         = 12 / p - 16 / p^2,
// so it is 3 - p/4 + (16 y - 12) y with y = 1 / p: with p <= 1 both 3 - p/4 and 16 y - 12 >= 4 y
// are sums without cancellation, and p is the FMA 1 - c c, rounded once, so the form is within a
// few 1e-16 of the exact value at its c (the bracket form: 1.1e-15 over |cos theta| < 0.9).
// Twelve FP64 operations a draw with the sums, against 27 and an IEEE division in terms of t and u
// (1.05e9 SplitMix64 draws: 3.03 ms there, 1.68 ms here); the prefactor
// (pi / s^2) alpha_s^2 / 2 (9/2) is the same for every draw and multiplies the sums.
__device__ __forceinline__ double cp_gg2gg_form(double c)
{
  const double p = fma(-c, c, 1.0);
  // 1 / p for p in (0, 1], normal: the hardware's approximation (its input and result are the upper
  // words, so within about 2^-19) and one third-order step y (1 + e + e^2), e = 1 - p y, which
  // leaves e^3 < 2^-56 and the rounding
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(p));
  const double e = fma(-p, y, 1.0);
  y = fma(y, fma(e, e, e), y);
  return fma(fma(16.0, y, -12.0), y, fma(-0.25, p, 3.0));
}

// cos theta = (2 u01 - 1) cMax of 64 random bits, u01 = (v >> 11) 2^-53.  2 u01 - 1 is exact: the
// upper 32 bits and the next 21 become the low mantissa words of 2^21 + H 2^-31 and 1 + L 2^-52, and
// both additions are exact (multiples of 2^-52 below 2), without a 64-bit integer conversion.
__device__ __forceinline__ double cp_partonic_cos(uint32_t hi, uint32_t lo, double cMax)
{
  const double dh = __hiloint2double(0x41400000, (int)hi), dl = __hiloint2double(0x3FF00000, (int)(lo >> 11));
  return ((dh - 2097154.0) + dl) * cMax;
}

// Sums of the matrix element over draws.
struct CpPartonicSums {
  double s1 = 0.0, s2 = 0.0, wm = 0.0;
  __device__ __forceinline__ void add(double v)
  {
    s1 += v;
    s2 = fma(v, v, s2);
    if (v > wm) wm = v;
  }
  // The same for several draws.  A draw seldom raises the largest one, so the upper words (order-preserving:
  // the values are positive) decide whether any can: one compare and a branch for eight draws instead of a
  // compare and two selects each (1.05e9 draws: 1.78 -> 1.72 ms).
  template <int N>
  __device__ __forceinline__ void add(const double (&v)[N])
  {
    int top = __double2hiint(v[0]);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      s1 += v[j];
      s2 = fma(v[j], v[j], s2);
      top = max(top, __double2hiint(v[j]));
    }
    if (top >= __double2hiint(wm)) {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (v[j] > wm) wm = v[j];
    }
  }
};

// MODE 0: Philox sums over points; 1 and 3: SplitMix64 sums over the reference's (thread, draw) pairs, for
// many and for few threads; 2: Philox per-point weights.  Sums are of the bare form above; each block scales its slot.
// Bound by instruction issue: about 20 integer operations (SplitMix64) and 12 FP64 a draw.
template <int MODE>
__global__ void __launch_bounds__(CP_THREADS, 5) k_partonic(const PartonicArgs a)
{
  __shared__ double sRed[CP_WARPS][3];
  const double scale = M_PI / (a.s * a.s) * (a.aS * a.aS) * 0.5 * 4.5 * a.scale;
  CpPartonicSums S;
  const uint64_t nthr = (uint64_t)gridDim.x * CP_THREADS;
  const uint64_t t = (uint64_t)blockIdx.x * CP_THREADS + threadIdx.x;
  if (MODE == 1 || MODE == 3) {
    // the reference's thread i makes draws k = 0 .. kper-1 from counter seed + i 0x100000001B3 + k
    // (cuPythia/03_fused_resident_me/fused_gg2gg.cu:43-50)
    const auto draw = [&](uint64_t c) {
      const uint64_t v = cp_splitmix64(c);
      return cp_gg2gg_form(cp_partonic_cos((uint32_t)(v >> 32), (uint32_t)v, a.cMax));
    };
    const auto draws = [&](uint64_t ctr, uint32_t m) {
      uint32_t j = 0;
      for (; j + 8 <= m; j += 8) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = draw(ctr + j + q);
        S.add(v);
      }
      for (; j < m; ++j) S.add(draw(ctr + j));
    };
    if (MODE == 1) {
      // A warp's lanes take 32 consecutive reference threads at the same k, and the warps equal contiguous
      // shares of the (group of 32, k) pairs, so the lanes are converged over runs of up to kper draws (shares
      // of single lanes cross their threads' ends at different draws: 2^20 threads x 1000 draws 1.72 -> 1.68 ms,
      // x 100 draws 268 -> 206 us).
      const int lane = threadIdx.x & 31;
      const uint64_t warps = nthr / 32, wi = t / 32;
      const uint64_t total = (a.n + 31) / 32 * a.kper, q = total / warps, rem = total % warps;
      const uint64_t w0 = q * wi + (wi < rem ? wi : rem);
      uint64_t left = q + (wi < rem ? 1 : 0), g = w0 / a.kper, k = w0 - g * a.kper;
      while (left) {
        uint64_t run = a.kper - k;
        run = run < left ? run : left;
        const uint32_t m = run < (1u << 30) ? (uint32_t)run : (1u << 30);
        const uint64_t i = 32 * g + lane;
        if (i < a.n) draws(a.seed + i * 0x100000001B3ULL + k, m);
        left -= m;
        k += m;
        if (k == a.kper) { k = 0; ++g; }
      }
    } else {
      // Few reference threads: the n kper pairs are split into
      // equal contiguous shares, so every thread here does the same number of draws (the first
      // total % nthr threads one more).  Within a reference thread the counters are consecutive; a
      // warp advances by the draws that all of its lanes have left in theirs, so its lanes stay
      // converged (lanes that loop over their own runs were 59% active at 1000 draws a thread).
      const uint64_t total = a.n * a.kper, q = total / nthr, rem = total % nthr;
      const uint64_t w0 = q * t + (t < rem ? t : rem);
      uint64_t left = q, i = w0 / a.kper, k = w0 - i * a.kper;
      uint64_t ctr = a.seed + i * 0x100000001B3ULL + k;
      while (left) {
        uint64_t run = a.kper - k;
        run = run < left ? run : left;
        const uint32_t m = __reduce_min_sync(0xffffffffu, run < (1u << 30) ? (uint32_t)run : (1u << 30));
        draws(ctr, m);
        left -= m;
        k += m;
        ctr += m;
        if (k == a.kper) { k = 0; ++i; ctr = a.seed + i * 0x100000001B3ULL; }
      }
      if (t < rem) S.add(draw(ctr));
    }
  } else {
    for (uint64_t i = t; i < a.n; i += nthr) {
      uint32_t wd[4];
      cp_point_words(a.seed, a.p0 + i, 0, 0, wd);
      const double v = cp_gg2gg_form(cp_partonic_cos(wd[1], wd[0], a.cMax));
      if (MODE == 2) { a.w_out[i] = v * scale; continue; }
      S.add(v);
    }
  }
  if (MODE == 2) return;
  const double s1 = cp_warp_sum_d(S.s1), s2 = cp_warp_sum_d(S.s2), wm = cp_warp_max_d(S.wm);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { sRed[warp][0] = s1; sRed[warp][1] = s2; sRed[warp][2] = wm; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double b1 = 0, b2 = 0, bm = 0;
    for (int k = 0; k < CP_WARPS; ++k) { b1 += sRed[k][0]; b2 += sRed[k][1]; bm = fmax(bm, sRed[k][2]); }
    double* slot = a.slots + 4 * (size_t)blockIdx.x;
    slot[0] = b1 * scale; slot[1] = b2 * (scale * scale); slot[2] = bm * scale; slot[3] = 0.0;
  }
}

static int partonic_run(cp_handle* h, int mode, PartonicArgs a, uint64_t npoints, cp_result* out)
{
  if (!(a.s > 0) || !(a.cMax > 0) || !(a.cMax < 1)) return cp_fail(h, CP_ERR_INVALID, "partonic: bad kinematics");
  // Equal shares for one wave of resident blocks, or for four waves once that leaves a thread 64 draws: the
  // warps of a wave finish far apart (at 75% of the issue slots some are served less), and the later blocks fill
  // what the early ones leave (1.05e9 draws: one wave 1.86 ms, 4 waves 1.78, 40 waves 1.88).
  int per_sm = 0;
  const cudaError_t oe = mode == 0 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_partonic<0>, CP_THREADS, 0)
                       : mode == 1 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_partonic<1>, CP_THREADS, 0)
                                   : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_partonic<3>, CP_THREADS, 0);
  if (oe != cudaSuccess || per_sm < 1) per_sm = 4;
  const int wave = h->num_sms * per_sm;
  const int blocks = npoints / ((uint64_t)wave * CP_THREADS) >= 4 * 64 ? 4 * wave : wave;
  int rc = cp_ensure_slots(h, (size_t)blocks * 4);
  if (rc) return rc;
  a.slots = h->d_slots;
  if (mode == 0) k_partonic<0><<<blocks, CP_THREADS, 0, h->stream>>>(a);
  else if (mode == 1) k_partonic<1><<<blocks, CP_THREADS, 0, h->stream>>>(a);
  else k_partonic<3><<<blocks, CP_THREADS, 0, h->stream>>>(a);
  CP_LAUNCH_CHECK(h, "k_partonic");
  k_reduce_slots<0><<<1, 4 * 32, 0, h->stream>>>(h->d_slots, blocks, 4, h->mail->sums);
  CP_LAUNCH_CHECK(h, "k_reduce_slots");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  const double* red = h->mail->sums;
  if (out) {
    double n = (double)npoints, mean = red[0] / n, var = (red[1] / n - mean * mean) / (n - 1.0);
    out->sigma = mean;
    out->sigma_err = sqrt(var > 0 ? var : 0);
    out->sum_w = red[0]; out->sum_w2 = red[1]; out->w_max = red[2];
    out->n_points = npoints; out->n_bad = 0;
    out->eta = red[2] > 0 ? mean / red[2] : 0;
  }
  return CP_OK;
}

extern "C" int cp_partonic_integrate(cp_handle* h, double sqrt_shat, double alphas, double cmax,
                                     double conv, uint64_t seed, uint64_t n, cp_result* out)
{
  CP_CHECK_HANDLE(h);
  if (n < 2) return cp_fail(h, CP_ERR_INVALID, "n_points < 2");
  double s = sqrt_shat * sqrt_shat;
  PartonicArgs a{s, alphas, cmax, (2.0 * cmax) * (s / 2.0) * conv, seed, 0, n, 0, nullptr, nullptr};
  return partonic_run(h, 0, a, n, out);
}

extern "C" int cp_partonic_splitmix(cp_handle* h, double sqrt_shat, double alphas, double cmax,
                                    double conv, uint64_t seed, uint64_t nthr, uint64_t kper,
                                    cp_result* out)
{
  CP_CHECK_HANDLE(h);
  if (kper && nthr > UINT64_MAX / kper) return cp_fail(h, CP_ERR_INVALID, "too many draws");
  if (nthr * kper < 2) return cp_fail(h, CP_ERR_INVALID, "too few draws");
  double s = sqrt_shat * sqrt_shat;
  PartonicArgs a{s, alphas, cmax, (2.0 * cmax) * (s / 2.0) * conv, seed, 0, nthr, kper, nullptr, nullptr};
  // groups of 32 reference threads, the last one possibly short, once that idles at most 3% of the lanes
  return partonic_run(h, nthr >= 1024 ? 1 : 3, a, nthr * kper, out);
}

extern "C" int cp_partonic_weights(cp_handle* h, double sqrt_shat, double alphas, double cmax,
                                   double conv, uint64_t seed, uint64_t p0, uint64_t n, double* w)
{
  CP_CHECK_HANDLE(h);
  if (n && !w) return cp_fail(h, CP_ERR_INVALID, "null output");
  if (!n) return CP_OK;
  double s = sqrt_shat * sqrt_shat;
  PartonicArgs a{s, alphas, cmax, (2.0 * cmax) * (s / 2.0) * conv, seed, p0, n, 0, nullptr, w};
  k_partonic<2><<<grid_for(h, n), CP_THREADS, 0, h->stream>>>(a);
  CP_LAUNCH_CHECK(h, "k_partonic");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}
