// cp_flow_train.cu -- training of the learned proposal on weights the integrator generates.
//
// Objective: the relative second moment of the weights, L = <w^2> / <w>^2 (= 1 + Var[w]/sigma^2),
// minimised over the flow parameters theta at fixed VEGAS grid (cp_flow_set_objective selects
// the relative p-th moment <w^p>/<w>^p instead, which weighs the tail of the weights more).  With w = f(x(x_v; theta)) J,
// x_v the VEGAS-mapped point (fixed by the random numbers), f the integrand and J the VEGAS
// Jacobian times |dx/dx_v|, the pathwise gradient is
//   dL/dtheta = 2/(B sigma^2) sum_points w^2 (d ln f/dx . dx/dtheta + d ln J/dtheta),
// so one step is: flow forward (saving each coupling's input) -> integrand value and d ln f/dx
// (forward-mode FP32 duals, the adjoint machinery) -> backward through sigmoid and couplings
// with each coupling's MLP recomputed on the tensor cores -> weight-gradient GEMMs on the tensor
// cores -> Adam (FP32 master weights) -> BF16 fragment repack.
#include "cp_dual.cuh"
#include "cp_flow.cuh"
#include "cp_internal.cuh"
#include "cp_tc.cuh"

int cp_flow_ensure(cp_handle* h);
int cp_flow_repack(cp_handle* h);

// Layout of the BF16 operands of the weight gradients, written by the backward pass: per coupling,
// stages of 64 points; in a stage of F features the feature groups of 8 one after the other, each
// its 8 core matrices (8 points x 8 features, 128 bytes: point q at (q % 8) * 16, feature f at
// (f % 8) * 2) and 32 bytes of padding.  A warp's mma.sync fragment register is one core matrix, so
// it stores as one contiguous 128-byte line (row-major rows of 128 bytes took eight half-used
// sectors a store: the backward pass of 65,536 points 79.5 -> 53 us); a stage is copied into shared memory as it is, one bulk copy per operand, where
// the core matrices are the MN-major no-swizzle operand (feature groups CP_WGT_FG apart, point
// groups 128); and the padding puts the four feature groups that a warp adds up for the bias into
// different banks.
#define CP_WGT_STAGE 64                            // points per stage (four K = 16 MMAs)
#define CP_WGT_FG (CP_WGT_STAGE * 16 + 32)         // bytes from a feature group to the next
#define CP_WGT_BYTES(F) ((F) / 8 * CP_WGT_FG)      // bytes of a stage of F features

struct FlowTrainBufs {
  float* zs;           // [B][4][3] input z of each coupling
  float4* vj;          // [B] (v0, v1, v2, ln J)
  float4* wg;          // [B] (w, d ln F / dv)
  uint64_t nst;        // stages per coupling; the arrays below are [4][nst] stages
  uint8_t* X;          // 16 wide: bf16 MLP inputs
  uint8_t* H1;         // 64: bf16 post-ReLU hidden 1
  uint8_t* H2;         // 64: bf16 post-ReLU hidden 2
  uint8_t* D1;         // 64: bf16 d pre-activation 1
  uint8_t* D2;         // 64: bf16 d pre-activation 2
  uint8_t* DO;         // 16: bf16 d outputs (s_raw, t)
  double* sums;        // [2] sum w, sum w^2 of the batch
  double* loss;        // per-step relative second moment
  float* gpart;        // [CP_WG_MAXBLK][CP_FLOW_NPARAM] per-block weight and bias gradients
};

// ------------------------------------------------------------------------------------------
// 1. forward, saving the input z of every coupling
// ------------------------------------------------------------------------------------------
// One block of 16 warps per SM: the weight fragments arrive in its shared memory once, by bulk copies
// that run while the warps draw and map their points (element copies by two blocks of 8 warps cost
// a third of the kernel: 65,536 points 26.4 -> 17.6 us).
#define CP_TRAIN_THREADS 512

// Starts the copies of the first `count` fragments of every coupling into shared memory (one thread,
// which has initialised the barrier; under the test hook, stall = 1, no kernel does), and the bounded wait for them (whole warps; on expiry the
// status word is raised and the copies get one more bounded wait before the warp may leave).
__device__ __forceinline__ void cp_train_weights_load(uint32_t bar, uint2* dst, const uint2* __restrict__ pk_g, int count)
{
  const uint32_t bytes = (uint32_t)count * (uint32_t)sizeof(uint2);
  cp_mbar_expect_tx(bar, CP_FLOW_NC * bytes);
  for (int c = 0; c < CP_FLOW_NC; ++c) cp_bulk_load(cp_smem_u32(dst + c * count), pk_g + c * CP_FLOW_P_PER, bytes, bar);
}
__device__ __forceinline__ bool cp_train_weights_wait(uint32_t bar, int* __restrict__ status)
{
  volatile int gave_up = 0;
  if (__all_sync(0xffffffffu, cp_mbar_wait_bounded(bar, 0u, &gave_up))) return true;
  *(volatile int*)status = 1;
  gave_up = 0;
  cp_mbar_wait_bounded(bar, 0u, &gave_up);
  __syncwarp();
  return false;
}

__global__ void __launch_bounds__(CP_TRAIN_THREADS) k_flow_fwd_train(const uint2* __restrict__ pk_g, const float* __restrict__ bias_g,
                                                               const double* __restrict__ edges, int nb,
                                                               uint64_t seed, uint32_t iter, uint32_t stream, uint64_t point0,
                                                               uint64_t n, float* __restrict__ zs, float4* __restrict__ vj,
                                                               int* __restrict__ status, int stall)
{
  extern __shared__ __align__(16) uint2 sPk[];
  float* sBias = reinterpret_cast<float*>(sPk + CP_FLOW_NC * CP_FLOW_P_FWD);
  __shared__ float2 sEdge[3][CP_MAX_BINS];
  __shared__ __align__(8) uint64_t sBar;
  const uint32_t bar = cp_smem_u32(&sBar);
  if (threadIdx.x == 0) {
    cp_mbar_init(bar, 1);
    cp_mbar_init_fence();
  }
  cp_wait_previous();
  cp_next_may_launch();
  if (threadIdx.x == 0 && stall != 1) cp_train_weights_load(bar, sPk, pk_g, CP_FLOW_P_FWD);
  for (int k = threadIdx.x; k < 3 * nb; k += CP_TRAIN_THREADS) {
    const int d = k / nb, b = k - d * nb;
    sEdge[d][b] = make_float2((float)edges[d * (nb + 1) + b], (float)(edges[d * (nb + 1) + b + 1] - edges[d * (nb + 1) + b]));
  }
  for (int j = threadIdx.x; j < CP_FLOW_NC * CP_FLOW_NB; j += CP_TRAIN_THREADS) sBias[j] = bias_g[j];
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * CP_TRAIN_THREADS;
  const uint64_t rounds = (n + stride - 1) / stride;
  for (uint64_t r = 0; r < rounds; ++r) {
    // consecutive warps' points to consecutive blocks: a batch that is not whole blocks loads every SM alike (the
    // same in k_flow_bwd; 65,536 points are 128 of 148 blocks; 100 steps 12.68 -> 12.50 ms)
    const uint64_t p = r * stride + ((uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
    const bool active = p < n;
    float z[3], jv = 1.f, logdet = 0.f;
    uint32_t w[4] = {0x80000000u, 0x80000000u, 0x80000000u, 0u};
    if (active) cp_point_words(seed, point0 + p, iter, stream, w);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      int bin;
      logdet += cp_flow_logit(cp_flow_vegas_in(sEdge[d], nb, w[d], jv, bin), z[d]);
    }
    logdet += logf(jv);
    if (r == 0 && !cp_train_weights_wait(bar, status)) return;   // no barrier follows
#pragma unroll 1
    for (int c = 0; c < CP_FLOW_NC; ++c) {
      if (active)
        for (int d = 0; d < 3; ++d) zs[(p * CP_FLOW_NC + c) * 3 + d] = z[d];
      const CpCoupling k = cp_coupling(c);
      const float* b = sBias + c * CP_FLOW_NB;
      float o[4];
      cp_flow_mlp_warp(sPk + c * CP_FLOW_P_FWD, b, z[k.cin[0]], k.nin > 1 ? z[k.cin[1]] : 0.f, o);
      for (int j = 0; j < k.nt; ++j) {
        const float s = CP_FLOW_S * tanhf(o[j] / CP_FLOW_S);
        z[k.tr[j]] = fmaf(z[k.tr[j]], expf(s), o[k.nt + j]);
        logdet += s;
      }
    }
    float v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) logdet += cp_flow_sigmoid(z[d], v[d]);
    if (active) vj[p] = make_float4(v[0], v[1], v[2], logdet);
  }
}

// ------------------------------------------------------------------------------------------
// 2. integrand value and d ln f / dx at the flow's points (3-tangent duals), batch sums
// ------------------------------------------------------------------------------------------
// Each block writes its (sum w, sum w^2) to its slot; the block that finishes last (integer
// ticket, after a fence) adds all slots in a fixed order (strided per-thread sums, the xor tree
// of each warp, the warps in order) into moments[0..1], writes the batch loss <w^2>/<w>^2 over
// n_loss points when loss != null, and re-arms the ticket.
// Four blocks per SM (128 registers, some spilled): the 2048 warps of 65,536 points are then resident
// at once; at the 190 registers it would take, eight warps per SM ran in two waves (65,536
// points 27.5 -> 26.7 us).
__global__ void __launch_bounds__(128, 4) k_flow_igrad(const CpHadParams P, const CpCteqPoly* __restrict__ cteq_g,
                                                    uint64_t n, float lnTauMin, const float4* __restrict__ vj,
                                                    float4* __restrict__ wg, double* __restrict__ slots,
                                                    unsigned* __restrict__ ticket, double* __restrict__ moments,
                                                    double n_loss, double* __restrict__ loss)
{
  __shared__ CpCteqPoly sCteq[8];
  __shared__ double sRed[4][2];
  __shared__ int sLast;
  cp_stage_cteq(sCteq, cteq_g);
  __syncthreads();
  cp_wait_previous();
  cp_next_may_launch();
  typedef CpDual<3> D3;
  CpHadParamsT<D3> Q;
  Q.lnTauMin = cp_dconst<3>(lnTauMin);
  Q.kR = cp_dconst<3>(P.kR);
  for (int k = 0; k < 4; ++k) Q.lnL2[k] = cp_dconst<3>(P.lnL2[k]);
  double s1 = 0.0, s2 = 0.0;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (uint64_t)gridDim.x * blockDim.x) {
    const float4 f = vj[p];
    D3 F = cp_had_weight_t<D3>(P, Q, sCteq, cp_dvar<3>(f.x, 0), cp_dvar<3>(f.y, 1), cp_dvar<3>(f.z, 2));
    float w = F.v * expf(f.w);
    float g[3] = {0.f, 0.f, 0.f};
    if (F.v > 0.f && isfinite(w)) {
      for (int d = 0; d < 3; ++d) g[d] = F.d[d] / F.v;
    } else {
      w = 0.f;
    }
    wg[p] = make_float4(w, g[0], g[1], g[2]);
    s1 += w;
    s2 += (double)w * w;
  }
  s1 = cp_warp_sum_d(s1);
  s2 = cp_warp_sum_d(s2);
  if ((threadIdx.x & 31) == 0) { sRed[threadIdx.x >> 5][0] = s1; sRed[threadIdx.x >> 5][1] = s2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) { a += sRed[q][0]; b += sRed[q][1]; }
    slots[2 * blockIdx.x] = a;
    slots[2 * blockIdx.x + 1] = b;
    __threadfence();
    sLast = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!sLast) return;
  __threadfence();
  double a = 0.0, b = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
    a += __ldcg(slots + 2 * k);
    b += __ldcg(slots + 2 * k + 1);
  }
  a = cp_warp_sum_d(a);
  b = cp_warp_sum_d(b);
  __syncthreads();   // sRed is reused
  if ((threadIdx.x & 31) == 0) { sRed[threadIdx.x >> 5][0] = a; sRed[threadIdx.x >> 5][1] = b; }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = 0.0;
    b = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) { a += sRed[q][0]; b += sRed[q][1]; }
    moments[0] = a;
    moments[1] = b;
    if (loss) {
      const double m = a / n_loss;
      loss[0] = (b / n_loss) / (m * m);
    }
    *ticket = 0u;
  }
}

// ------------------------------------------------------------------------------------------
// 3. backward through the couplings (MLPs recomputed), writing the GEMM operands
// ------------------------------------------------------------------------------------------
// writes a 16 x 64 bf16 tile held as A fragments: register (kt, 0 | 1) is the core matrix of feature
// group 2 kt and the tile's first | second 8 points, (kt, 2 | 3) that of group 2 kt + 1.  `dst`: the
// tile's first point group in its stage + 4 lane; ra, rb: this lane's two rows lie inside the batch
__device__ __forceinline__ void cp_store_rowfrag(uint8_t* dst, bool ra, bool rb, const uint32_t (&h)[4][4])
{
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) {
    uint8_t* d = dst + 2 * kt * CP_WGT_FG;
    if (ra) {
      *reinterpret_cast<uint32_t*>(d) = h[kt][0];
      *reinterpret_cast<uint32_t*>(d + CP_WGT_FG) = h[kt][2];
    }
    if (rb) {
      *reinterpret_cast<uint32_t*>(d + 128) = h[kt][1];
      *reinterpret_cast<uint32_t*>(d + CP_WGT_FG + 128) = h[kt][3];
    }
  }
}

// ReLU masks of a tile's activations (A fragments, non-negative): bit 4 nt + e for element e of
// n-tile nt's accumulator, set where the activation is above zero
__device__ __forceinline__ uint32_t cp_relu_mask(const uint32_t (&h)[4][4])
{
  uint32_t m = 0u;
#pragma unroll
  for (int kt = 0; kt < 4; ++kt)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int bit = 4 * (2 * kt + (q >> 1)) + 2 * (q & 1);
      if (h[kt][q] & 0x00007fffu) m |= 1u << bit;
      if (h[kt][q] & 0x7fff0000u) m |= 2u << bit;
    }
  return m;
}

// one 64-wide backward product of KT k-tiles for both tiles: d = bf16(mask (A W)) as A fragments
template <int KT>
__device__ __forceinline__ void cp_flow_back64(const uint32_t (&a)[2][KT][4], const uint2* __restrict__ pk,
                                               const uint32_t (&keep)[2], uint32_t (&d)[2][4][4])
{
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k2 = 0; k2 < 4; ++k2) {
    float acc[2][2][4] = {};   // [n-tile][tile]
#pragma unroll
    for (int kt = 0; kt < KT; ++kt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint2 w = pk[(kt * 8 + 2 * k2 + j) * 32 + lane];
#pragma unroll
        for (int t = 0; t < 2; ++t) cp_mma_bf16(acc[j][t], a[t][kt], w);
      }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float m[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) m[e] = (keep[t] >> (4 * (2 * k2 + j) + e)) & 1u ? acc[j][t][e] : 0.f;
        d[t][k2][2 * j] = cp_bf2(m[0], m[1]);
        d[t][k2][2 * j + 1] = cp_bf2(m[2], m[3]);
      }
  }
}

// One block of 16 warps per SM, the 88 KB of weight fragments by bulk copies, as in the forward
// (65,536 points 53 -> 46.6 us).  The two tiles of a warp go together and only bit masks of the
// activations are kept; that by itself measured no faster than a tile at a time.
__global__ void __launch_bounds__(CP_TRAIN_THREADS) k_flow_bwd(const uint2* __restrict__ pk_g, const float* __restrict__ bias_g, uint64_t n,
                                                  double n_batch, const float* __restrict__ zs, const float4* __restrict__ vj,
                                                  const float4* __restrict__ wg, const double* __restrict__ sums,
                                                  FlowTrainBufs out, float loss_p, int* __restrict__ status, int stall)
{
  extern __shared__ __align__(16) uint2 sPk[];   // all CP_FLOW_P_PER fragments of the 4 couplings, then biases
  float* sBias = reinterpret_cast<float*>(sPk + CP_FLOW_NC * CP_FLOW_P_PER);
  __shared__ __align__(8) uint64_t sBar;
  const uint32_t bar = cp_smem_u32(&sBar);
  if (threadIdx.x == 0) {
    cp_mbar_init(bar, 1);
    cp_mbar_init_fence();
  }
  cp_wait_previous();
  cp_next_may_launch();
  if (threadIdx.x == 0 && stall != 1) cp_train_weights_load(bar, sPk, pk_g, CP_FLOW_P_PER);
  for (int j = threadIdx.x; j < CP_FLOW_NC * CP_FLOW_NB; j += blockDim.x) sBias[j] = bias_g[j];
  __syncthreads();
  const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  // the batch's moments and size (all ranks' points when the batch is sharded)
  const double sig = sums[0] / n_batch;
  const float cnorm = (float)(2.0 / (n_batch * sig * sig));
  // objective <w^p>/<w>^p: dL/d ln w of a point = p (w / sigma)^p / B (p = 2: 2 w^2 / (B sigma^2))
  const float cnorm_p = (float)(loss_p / n_batch), inv_sig = (float)(1.0 / sig);
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const uint64_t rounds = (n + 32 * warps - 1) / (32 * warps);
  for (uint64_t r = 0; r < rounds; ++r) {
    const uint64_t base = (r * warps + (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32;
    const uint64_t p = base + lane;
    const bool active = p < n;
    float dz[3] = {0.f, 0.f, 0.f}, cJ = 0.f;
    if (active) {
      const float4 f = vj[p], g = wg[p];
      cJ = loss_p == 2.f ? cnorm * g.x * g.x : cnorm_p * powf(g.x * inv_sig, loss_p);
      const float v[3] = {f.x, f.y, f.z}, gv[3] = {g.y, g.z, g.w};
      // sigmoid: dv/dz = v (1 - v); d ln(v (1 - v))/dz = 1 - 2 v
      for (int d = 0; d < 3; ++d) dz[d] = cJ * gv[d] * v[d] * (1.f - v[d]) + cJ * (1.f - 2.f * v[d]);
    }
    if (r == 0 && !cp_train_weights_wait(bar, status)) return;   // no barrier follows
#pragma unroll 1
    for (int c = CP_FLOW_NC - 1; c >= 0; --c) {
      const CpCoupling k = cp_coupling(c);
      const uint2* pk = sPk + c * CP_FLOW_P_PER;
      const float* b = sBias + c * CP_FLOW_NB;
      float zin[3] = {0.f, 0.f, 0.f};
      if (active)
        for (int d = 0; d < 3; ++d) zin[d] = zs[(p * CP_FLOW_NC + c) * 3 + d];
      const float in0 = zin[k.cin[0]], in1 = k.nin > 1 ? zin[k.cin[1]] : 0.f;
      // this lane's word of each tile's first core matrix in its stage (16- and 64-wide arrays)
      size_t at16[2], at64[2];
      bool rowa[2], rowb[2];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const uint64_t row0 = base + 16 * t;
        rowa[t] = row0 + gid < n;
        rowb[t] = row0 + gid + 8 < n;
        const uint64_t stage = (uint64_t)c * out.nst + row0 / CP_WGT_STAGE;
        const uint32_t inst = (uint32_t)(row0 % CP_WGT_STAGE) * 16u + 4u * lane;
        at16[t] = stage * CP_WGT_BYTES(16) + inst;
        at64[t] = stage * CP_WGT_BYTES(64) + inst;
      }
      // ---- the MLP forward again; of the activations only the ReLU masks stay
      float o[4];
      uint32_t keep1[2], keep2[2];
      {
        uint32_t a[2][1][4], h1[2][4][4], h2[2][4][4];
        {
          uint32_t f[2][4];
          cp_flow_in_frags(in0, in1, f);
#pragma unroll
          for (int t = 0; t < 2; ++t) {
#pragma unroll
            for (int q = 0; q < 4; ++q) a[t][0][q] = f[t][q];
            if (rowa[t]) *reinterpret_cast<uint32_t*>(out.X + at16[t]) = f[t][0];
            if (rowb[t]) *reinterpret_cast<uint32_t*>(out.X + at16[t] + 128) = f[t][1];
          }
        }
        cp_flow_layer64<1>(a, pk + CP_FLOW_P_W1, b, h1);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          cp_store_rowfrag(out.H1 + at64[t], rowa[t], rowb[t], h1[t]);
          keep1[t] = cp_relu_mask(h1[t]);
        }
        cp_flow_layer64<4>(h1, pk + CP_FLOW_P_W2, b + 64, h2);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          cp_store_rowfrag(out.H2 + at64[t], rowa[t], rowb[t], h2[t]);
          keep2[t] = cp_relu_mask(h2[t]);
        }
        cp_flow_layer_out(h2, pk + CP_FLOW_P_W3, b + 128, o);
      }
      // ---- coupling backward of this lane's point
      float dO[4] = {0.f, 0.f, 0.f, 0.f}, dzT[2] = {0.f, 0.f};
      if (active) {
        for (int j = 0; j < k.nt; ++j) {
          const float th = tanhf(o[j] / CP_FLOW_S), s = CP_FLOW_S * th, e = expf(s);
          const int d = k.tr[j];
          const float dzo = dz[d];
          const float ds = fmaf(dzo * zin[d], e, cJ);
          dO[j] = ds * (1.f - th * th);
          dO[k.nt + j] = dzo;
          dzT[j] = dzo * e;
        }
      }
      // dO as A fragments: columns 0..3, rows gid and gid + 8 of each tile
      // (a shuffle sends the value the source lane holds, so fetch all four and select here)
      uint32_t ad[2][4];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        float g0[4], g8[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          g0[q] = __shfl_sync(0xffffffffu, dO[q], 16 * t + gid);
          g8[q] = __shfl_sync(0xffffffffu, dO[q], 16 * t + gid + 8);
        }
        const bool odd = tig & 1;
        ad[t][0] = tig < 2 ? cp_bf2(odd ? g0[2] : g0[0], odd ? g0[3] : g0[1]) : 0u;
        ad[t][1] = tig < 2 ? cp_bf2(odd ? g8[2] : g8[0], odd ? g8[3] : g8[1]) : 0u;
        ad[t][2] = ad[t][3] = 0u;
        if (rowa[t]) *reinterpret_cast<uint32_t*>(out.DO + at16[t]) = ad[t][0];
        if (rowb[t]) *reinterpret_cast<uint32_t*>(out.DO + at16[t] + 128) = ad[t][1];
      }
      // dH2 = dO W3^T, masked by the ReLU of layer 2
      uint32_t d2[2][4][4], d1[2][4][4];
      {
        uint32_t a[2][1][4];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int q = 0; q < 4; ++q) a[t][0][q] = ad[t][q];
        cp_flow_back64<1>(a, pk + CP_FLOW_P_W3T, keep2, d2);
      }
#pragma unroll
      for (int t = 0; t < 2; ++t) cp_store_rowfrag(out.D2 + at64[t], rowa[t], rowb[t], d2[t]);
      // dH1 = dH2 W2^T, masked by the ReLU of layer 1
      cp_flow_back64<4>(d2, pk + CP_FLOW_P_W2T, keep1, d1);
#pragma unroll
      for (int t = 0; t < 2; ++t) cp_store_rowfrag(out.D1 + at64[t], rowa[t], rowb[t], d1[t]);
      // dX = dH1 W1^T: columns 0..1 are the gradients of the two input features
      float cx[2][4] = {};
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        const uint2 w = pk[CP_FLOW_P_W1T + kt * 32 + lane];
#pragma unroll
        for (int t = 0; t < 2; ++t) cp_mma_bf16(cx[t], d1[t][kt], w);
      }
      const int rr = lane & 15, src = 4 * (rr & 7);
      const bool hi = rr >= 8, second = lane >= 16;
      float dx[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float e0 = __shfl_sync(0xffffffffu, cx[0][q], src), e2 = __shfl_sync(0xffffffffu, cx[0][2 + q], src);
        const float f0 = __shfl_sync(0xffffffffu, cx[1][q], src), f2 = __shfl_sync(0xffffffffu, cx[1][2 + q], src);
        dx[q] = second ? (hi ? f2 : f0) : (hi ? e2 : e0);
      }
      if (active) {
        for (int j = 0; j < k.nt; ++j) dz[k.tr[j]] = dzT[j];
        dz[k.cin[0]] += dx[0];
        if (k.nin > 1) dz[k.cin[1]] += dx[1];
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// 4. weight and bias gradients of one layer shape for all couplings (blockIdx.y = coupling):
//    block b's chunk of points gives G_b[M][N] = sum_p A[p][0:M]^T B[p][0:N] on the tensor cores
//    and the bias gradient Gb_b[N] = sum_p B[p][0:N] from the same staged tiles, stored into its
//    own slot of the partial buffer (A, B bf16 in the stage layout above; M in {16, 64},
//    N in {16, 64}); k_flow_gsum then adds the slots in block order, so a training run is
//    reproducible bit for bit (no floating-point atomics).
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_ldsm_x4_t(uint32_t r[4], const void* p)
{
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// byte offset of (point p, feature f) in a coupling's operand of F features
template <int F>
__device__ __forceinline__ size_t cp_wgt_at(uint64_t p, int f)
{
  return p / CP_WGT_STAGE * CP_WGT_BYTES(F) + (size_t)((f >> 3) * CP_WGT_FG + (int)(p % CP_WGT_STAGE) * 16 + (f & 7) * 2);
}

#define CP_WG_ROWS 64   // points staged per iteration
#define CP_WG_MAXBLK 64 // blocks per coupling and layer (the batch is cut into at most this many chunks)

template <int M, int N>
__global__ void __launch_bounds__(128) k_flow_wgrad(const uint8_t* __restrict__ A0, const uint8_t* __restrict__ B0,
                                                    uint64_t nst, uint64_t n, float* __restrict__ part, int goff, int ldg, int nvalid,
                                                    int chunk, int bias_rel)
{
  constexpr int MT = M / 16, NT = N / 8, TPW = (MT * NT + 3) / 4;
  __shared__ __align__(16) uint16_t sA[CP_WG_ROWS * M];
  __shared__ __align__(16) uint16_t sB[CP_WG_ROWS * N];
  __shared__ float sBias[128];
  const int c = blockIdx.y;
  const uint8_t* A = A0 + (uint64_t)c * nst * CP_WGT_BYTES(M);
  const uint8_t* B = B0 + (uint64_t)c * nst * CP_WGT_BYTES(N);
  float* G = part + (size_t)blockIdx.x * CP_FLOW_NPARAM + c * CP_FLOW_PER + goff;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int mi = lane >> 3, rw = lane & 7;
  float acc[TPW][4];
#pragma unroll
  for (int j = 0; j < TPW; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  const int bcol = threadIdx.x % N, brow0 = threadIdx.x / N;
  float bsum = 0.f;
  const uint64_t p_begin = (uint64_t)blockIdx.x * chunk;
  const uint64_t p_end = p_begin + chunk < n ? p_begin + chunk : n;
  for (uint64_t p0 = p_begin; p0 < p_end; p0 += CP_WG_ROWS) {
    for (int e = threadIdx.x; e < CP_WG_ROWS * M / 8; e += blockDim.x) {
      const int row = e / (M / 8), col = (e % (M / 8)) * 8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (p0 + row < p_end) v = *reinterpret_cast<const uint4*>(A + cp_wgt_at<M>(p0 + row, col));
      *reinterpret_cast<uint4*>(&sA[row * M + col]) = v;
    }
    for (int e = threadIdx.x; e < CP_WG_ROWS * N / 8; e += blockDim.x) {
      const int row = e / (N / 8), col = (e % (N / 8)) * 8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (p0 + row < p_end) v = *reinterpret_cast<const uint4*>(B + cp_wgt_at<N>(p0 + row, col));
      *reinterpret_cast<uint4*>(&sB[row * N + col]) = v;
    }
    __syncthreads();
    for (int r = brow0; r < CP_WG_ROWS; r += 128 / N) bsum += __uint_as_float(((uint32_t)sB[r * N + bcol]) << 16);
#pragma unroll
    for (int ks = 0; ks < CP_WG_ROWS / 16; ++ks) {
      const uint16_t* tA = sA + ks * 16 * M;
      const uint16_t* tB = sB + ks * 16 * N;
#pragma unroll
      for (int j = 0; j < TPW; ++j) {
        const int t = warp + 4 * j;
        if (t < MT * NT) {
          const int mt = t / NT, nt = t % NT;
          uint32_t a[4], bq[2];
          // A^T of m-tile mt: 8x8 blocks (points 0-7 | 8-15) x (m +0 | +8), delivered transposed
          cp_ldsm_x4_t(a, &tA[((mi >> 1) * 8 + rw) * M + mt * 16 + (mi & 1) * 8]);
          // B of n-tile nt: blocks (points 0-7 | 8-15) x (n tile), delivered transposed
          {
            const uint32_t ad = (uint32_t)__cvta_generic_to_shared(&tB[((mi & 1) * 8 + rw) * N + nt * 8]);
            asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                         : "=r"(bq[0]), "=r"(bq[1]) : "r"(ad));
          }
          cp_mma_bf16(acc[j], a, make_uint2(bq[0], bq[1]));
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < TPW; ++j) {
    const int t = warp + 4 * j;
    if (t >= MT * NT) continue;
    const int mt = t / NT, nt = t % NT;
    const int m0 = mt * 16 + gid, n0 = nt * 8 + 2 * tig;
    if (n0 < nvalid) { G[m0 * ldg + n0] = acc[j][0]; G[(m0 + 8) * ldg + n0] = acc[j][2]; }
    if (n0 + 1 < nvalid) { G[m0 * ldg + n0 + 1] = acc[j][1]; G[(m0 + 8) * ldg + n0 + 1] = acc[j][3]; }
  }
  // the 128 / N threads of a bias column add their row sums in thread order
  sBias[threadIdx.x] = bsum;
  __syncthreads();
  if (threadIdx.x < N && threadIdx.x < nvalid) {
    float b = 0.f;
    for (int r = 0; r < 128 / N; ++r) b += sBias[r * N + threadIdx.x];
    G[bias_rel + threadIdx.x] = b;
  }
}

// ------------------------------------------------------------------------------------------
// 4'. The same weight and bias gradients on the 5th-generation tensor cores, all couplings and
//     the three layer shapes in one launch (blockIdx.y = coupling, blockIdx.z = layer).  Every
//     product has the hidden side (64 wide) as M and the other side as N:
//       layer 0: dW1^T[n][k] = sum_p D1[p][n] X[p][k]    M = 64 (n), N = 16 (k), bias b1 = sum D1
//       layer 1: dW2[k][n]   = sum_p H1[p][k] D2[p][n]   M = 64 (k), N = 64 (n), bias b2 = sum D2
//       layer 2: dW3[k][n]   = sum_p H2[p][k] DO[p][n]   M = 64 (k), N = 16 (n), bias b3 = sum DO
//     so D[M][N] += A[M][K] B[N][K]^T with K = the block's points, 64 per stage, both operands
//     MN-major (features contiguous) in the stage layout: the descriptor's stride in the feature
//     direction (SBO) is CP_WGT_FG and in the point direction (LBO) 128 bytes.  Thread 0 fetches each
//     stage with one bulk copy per operand (two stages in flight), issues its four K = 16 MMAs and
//     commits them; warps 2 and 3 add up the bias columns from the same stage; a stage's buffer is
//     refilled once its `empty` barrier has the commit and those two warps' arrivals.  Every wait is
//     bounded.  The M = 64 accumulator occupies TMEM lanes 0-15 of each 32-lane quarter (row r in
//     lane r % 16 + 32 (r / 16)), so thread t < 16 of warp w reads row 16 w + t.  Each block writes its
//     own slot of the partial buffer; k_flow_gsum adds the slots in block order.
//
//     What bounds it is reading the operands, 151 MB per 65,536 points, mostly from L2 where the
//     backward pass left them.  34 KB of stages let six blocks reside on an SM, so all 768 of a batch
//     run at once (five before, with 28 blocks left for a second wave):
//     71 -> 33 us per 65,536 points.
// ------------------------------------------------------------------------------------------
// two bias columns (a pair of features) and one residue class of the stage's points per thread of
// warps 2 and 3: 64 features x 2 residues, 16 features x 8; `res`: points res, res + step, ...
struct CpWgtBias {
  int fg, w, res, step;
  float lo = 0.f, hi = 0.f;
  __device__ __forceinline__ CpWgtBias(int width, int t)   // t in [0, 64)
  {
    w = t & 3;
    if (width == 64) { res = (t >> 2) & 1; fg = t >> 3; step = 2; }
    else { res = (t >> 2) & 7; fg = t >> 5; step = 8; }
  }
  __device__ __forceinline__ void add(const uint8_t* s)   // a stage's shared-memory copy
  {
    const uint8_t* at = s + fg * CP_WGT_FG + 4 * w;
    for (int q = res; q < CP_WGT_STAGE; q += step) {
      const uint32_t v = *reinterpret_cast<const uint32_t*>(at + 16 * q);
      lo += __uint_as_float(v << 16);
      hi += __uint_as_float(v & 0xffff0000u);
    }
  }
};

template <int NB>
__device__ __forceinline__ void cp_wgt_layer(const uint8_t* __restrict__ A, const uint8_t* __restrict__ B, bool bias_of_a,
                                             uint64_t st_begin, uint64_t st_end, float* __restrict__ G, int layer,
                                             uint8_t* smem, uint32_t tmem, uint32_t mbar, float* sBias,
                                             int* __restrict__ status)
{
  constexpr uint32_t AB = CP_WGT_BYTES(64), BB = CP_WGT_BYTES(NB);
  const uint32_t sbase = cp_smem_u32(smem);
  // barriers: full[0..1] (bulk copies landed), empty[0..1] (MMAs and bias reads done), all MMAs, drain
  const uint32_t full = mbar, empty = mbar + 16, done = mbar + 32, drain = mbar + 40;
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(NB >> 3) << 17) |
                         ((uint32_t)(64 >> 4) << 24);
  const int nst = (int)(st_end - st_begin), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int abort_flag = 0;
  bool ok = true;
  CpWgtBias bias(bias_of_a ? 64 : NB, tid & 63);
  if (tid == 0) {
    auto fetch = [&](int st) {
      const int b = st & 1;
      cp_mbar_expect_tx(full + 8 * b, AB + BB);
      cp_bulk_load(sbase + b * AB, A + (st_begin + st) * AB, AB, full + 8 * b);
      cp_bulk_load(sbase + 2 * AB + b * BB, B + (st_begin + st) * BB, BB, full + 8 * b);
    };
    int fetched = 0;
    for (; fetched < nst && fetched < 2; ++fetched) fetch(fetched);
    int st = 0;
    for (; st < nst; ++st) {
      const int b = st & 1;
      if (!(ok = cp_mbar_wait_bounded(full + 8 * b, (st >> 1) & 1, &abort_flag))) break;
      cp_tc_fence_after();
#pragma unroll
      for (int k = 0; k < CP_WGT_STAGE / 16; ++k) {
        const uint64_t da = cp_tc_desc(sbase + b * AB + k * 256, 128, CP_WGT_FG);   // K = 16: two point groups
        const uint64_t db = cp_tc_desc(sbase + 2 * AB + b * BB + k * 256, 128, CP_WGT_FG);
        cp_tc_mma(tmem, da, db, idesc, (st > 0 || k > 0) ? 1u : 0u);
      }
      cp_tc_commit(empty + 8 * b);
      if (fetched < nst) {
        if (!(ok = cp_mbar_wait_bounded(empty + 8 * b, (st >> 1) & 1, &abort_flag))) break;
        fetch(fetched++);
      }
    }
    cp_tc_commit(done);
    if (!ok) {   // the copies in flight land before the shared memory is given up
      volatile int drain_abort = 0;
      for (int f = st; f < fetched; ++f) cp_mbar_wait_bounded(full + 8 * (f & 1), (f >> 1) & 1, &drain_abort);
    }
  } else if (warp >= 2) {
    for (int st = 0; st < nst; ++st) {
      const int b = st & 1;
      if (!(ok = cp_mbar_wait_bounded(full + 8 * b, (st >> 1) & 1, &abort_flag))) break;
      bias.add(smem + (bias_of_a ? b * AB : 2 * AB + b * BB));
      __syncwarp();
      if (lane == 0) cp_mbar_arrive(empty + 8 * b);
    }
  }
  __syncwarp();
  ok = cp_mbar_wait_bounded(done, 0u, &abort_flag) && ok;
  cp_tc_fence_after();
  ok = __syncthreads_and(ok) != 0;
  if (!ok) {
    // a wait expired: record it, and before TMEM is released let every MMA this thread issued
    // complete (a fresh barrier, bounded wait)
    if (tid == 0) {
      *(volatile int*)status = 1;
      cp_tc_commit(drain);
      volatile int drain_abort = 0;
      cp_mbar_wait_bounded(drain, 0u, &drain_abort);
    }
    __syncthreads();
    return;
  }
  // accumulator: warp w, lane t < 16 = row 16 w + t
  const int row = 16 * warp + lane;
  const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16);
#pragma unroll
  for (int half = 0; half < NB / 16; half += 2) {
    float v[32];
    if (NB == 64) {
      cp_tc_ld32(taddr + half * 16, v);
    } else {
      float v4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        cp_tc_ld4(taddr + 4 * j, v4);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[4 * j + i] = v4[i];
      }
    }
    if (lane < 16) {
      const int ncol = NB == 64 ? 32 : 16;
#pragma unroll
      for (int j = 0; j < ncol; ++j) {
        const int c = half * 16 + j;
        if (layer == 0) G[CP_FLOW_W1 + c * 64 + row] = v[j];                 // dW1[k = c][n = row]
        else if (layer == 1) G[CP_FLOW_W2 + row * 64 + c] = v[j];            // dW2[k = row][n = c]
        else if (c < 8) G[CP_FLOW_W3 + row * 8 + c] = v[j];                  // dW3[k = row][n = c < 8]
      }
    }
  }
  // bias: the residue classes of a column added in order (a column's points res, res + step, ...
  // form one running sum, so the sums are those of 128 / width threads a column)
  const int bw = bias_of_a ? 64 : NB;
  if (warp >= 2) {
    const int col = bias.fg * 8 + 2 * bias.w;
    sBias[bias.res * bw + col] = bias.lo;
    sBias[bias.res * bw + col + 1] = bias.hi;
  }
  __syncthreads();
  const int nb_valid = layer == 2 ? 8 : 64;
  if (tid < bw && tid < nb_valid) {
    float acc = 0.f;
    for (int r = 0; r < 128 / bw; ++r) acc += sBias[r * bw + tid];
    G[(layer == 0 ? CP_FLOW_B1 : (layer == 1 ? CP_FLOW_B2 : CP_FLOW_B3)) + tid] = acc;
  }
}

__global__ void __launch_bounds__(128) k_flow_wgrad_tc(FlowTrainBufs t, int chunk, int* __restrict__ status)
{
  __shared__ __align__(1024) uint8_t smem[4 * CP_WGT_BYTES(64)];   // two A and two B stages
  __shared__ float sBias[128];
  __shared__ __align__(8) uint64_t mbar[6];
  __shared__ uint32_t tmem_slot;
  const int c = blockIdx.y, layer = blockIdx.z, tid = threadIdx.x;
  if (tid == 0) {
    // full: the fetching thread's arrival (and the copies' bytes); empty: the MMAs' commit and warps 2, 3
    for (int i = 0; i < 6; ++i) cp_mbar_init(cp_smem_u32(&mbar[i]), i == 2 || i == 3 ? 3 : 1);
    cp_mbar_init_fence();
  }
  if ((tid >> 5) == 0) {
    cp_tc_alloc(cp_smem_u32(&tmem_slot), 64);
    cp_tc_relinquish();
  }
  cp_tc_fence_before();
  __syncthreads();
  cp_tc_fence_after();
  cp_wait_previous();
  cp_next_may_launch();
  const uint32_t tmem = tmem_slot;
  // chunk is a whole number of stages; rows beyond n of the last one are zero
  const uint64_t sb = (uint64_t)blockIdx.x * (chunk / CP_WGT_STAGE);
  const uint64_t se = sb + chunk / CP_WGT_STAGE < t.nst ? sb + chunk / CP_WGT_STAGE : t.nst;
  float* G = t.gpart + (size_t)blockIdx.x * CP_FLOW_NPARAM + c * CP_FLOW_PER;
  const size_t o16 = (size_t)c * t.nst * CP_WGT_BYTES(16), o64 = (size_t)c * t.nst * CP_WGT_BYTES(64);
  const uint32_t mb = cp_smem_u32(&mbar[0]);
  if (sb < se) {
    if (layer == 0) cp_wgt_layer<16>(t.D1 + o64, t.X + o16, true, sb, se, G, 0, smem, tmem, mb, sBias, status);
    else if (layer == 1) cp_wgt_layer<64>(t.H1 + o64, t.D2 + o64, false, sb, se, G, 1, smem, tmem, mb, sBias, status);
    else cp_wgt_layer<16>(t.H2 + o64, t.DO + o16, false, sb, se, G, 2, smem, tmem, mb, sBias, status);
  }
  cp_tc_fence_before();
  __syncthreads();
  if ((tid >> 5) == 0) {
    cp_tc_fence_after();
    cp_tc_dealloc(tmem, 64);
  }
}

// G[i] += sum over the nblk block slots of the partial gradients, in block order
__global__ void k_flow_gsum(const float* __restrict__ part, int nblk, float* __restrict__ G)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= CP_FLOW_NPARAM) return;
  float s = 0.f;
  for (int b = 0; b < nblk; ++b) s += part[(size_t)b * CP_FLOW_NPARAM + i];
  G[i] += s;
}

// ------------------------------------------------------------------------------------------
// 5. Adam on the FP32 master weights (padding entries stay zero)
// ------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ bool cp_flow_param_used(int i)
{
  const int c = i / CP_FLOW_PER, o = i % CP_FLOW_PER;
  const CpCoupling k = cp_coupling(c);
  const int nout = 2 * k.nt;
  if (o < CP_FLOW_B1) return o / 64 < k.nin;
  if (o < CP_FLOW_B2) return true;
  if (o < CP_FLOW_W3) return true;
  if (o < CP_FLOW_B3) return ((o - CP_FLOW_W3) % 8) < nout;
  return (o - CP_FLOW_B3) < nout;
}

__device__ __forceinline__ void cp_flow_adam_one(int i, float g, float* __restrict__ P, float* __restrict__ Mo,
                                                 float* __restrict__ Vo, float lr, float b1t, float b2t)
{
  if (!cp_flow_param_used(i)) { P[i] = 0.f; return; }
  const float m = 0.9f * Mo[i] + 0.1f * g, v = 0.999f * Vo[i] + 0.001f * g * g;
  Mo[i] = m;
  Vo[i] = v;
  P[i] -= lr * (m / (1.f - b1t)) / (sqrtf(v / (1.f - b2t)) + 1e-8f);
}

__global__ void k_flow_adam(float* __restrict__ P, float* __restrict__ G, float* __restrict__ Mo, float* __restrict__ Vo,
                            float lr, float b1t, float b2t)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= CP_FLOW_NPARAM) return;
  const float g = G[i];
  G[i] = 0.f;
  cp_flow_adam_one(i, g, P, Mo, Vo, lr, b1t, b2t);
}

// k_flow_gsum into a cleared G, k_flow_adam and k_flow_pack in one pass (a single handle's training
// loop, where no exchange of G sits between them): the same block-order sum, 0 + sum as the gradient,
// the same update, and the parameter's BF16 value into its places in the packed fragments (the
// forward and the transposed one), which a full pack has laid out before; G is not touched.  The
// slots are read sixteen at a time: one after the other, their latencies were the kernel (7.4 us, and
// 3.9 us for the pack; 7.6 us together).
__device__ __forceinline__ void cp_flow_pack_one(int i, float v, uint2* __restrict__ pk, float* __restrict__ bias)
{
  const int c = i / CP_FLOW_PER, o = i % CP_FLOW_PER;
  uint16_t* q = reinterpret_cast<uint16_t*>(pk + c * CP_FLOW_P_PER);
  const __nv_bfloat16 bv = __float2bfloat16_rn(v);
  const uint16_t h = *reinterpret_cast<const uint16_t*>(&bv);
  // B fragment (first fragment f0, n-tiles per k-tile nnt) of element (row k, column n): lane
  // 4 (n % 8) + (k % 8) / 2, word k % 16 / 8, half k % 2
  const auto put = [&](int f0, int nnt, int k, int n) {
    const int e = f0 + ((k >> 4) * nnt + (n >> 3)) * 32 + 4 * (n & 7) + ((k & 7) >> 1);
    q[4 * e + 2 * ((k >> 3) & 1) + (k & 1)] = h;
  };
  if (o < CP_FLOW_B1) {
    const int k = o >> 6, n = o & 63;
    put(CP_FLOW_P_W1, 8, k, n);
    if (k < 8) put(CP_FLOW_P_W1T, 1, n, k);
  } else if (o < CP_FLOW_W2) {
    bias[c * CP_FLOW_NB + o - CP_FLOW_B1] = v;
  } else if (o < CP_FLOW_B2) {
    const int k = (o - CP_FLOW_W2) >> 6, n = (o - CP_FLOW_W2) & 63;
    put(CP_FLOW_P_W2, 8, k, n);
    put(CP_FLOW_P_W2T, 8, n, k);
  } else if (o < CP_FLOW_W3) {
    bias[c * CP_FLOW_NB + 64 + o - CP_FLOW_B2] = v;
  } else if (o < CP_FLOW_B3) {
    const int k = (o - CP_FLOW_W3) >> 3, n = (o - CP_FLOW_W3) & 7;
    put(CP_FLOW_P_W3, 1, k, n);
    put(CP_FLOW_P_W3T, 8, n, k);
  } else {
    bias[c * CP_FLOW_NB + 128 + o - CP_FLOW_B3] = v;
  }
}

__global__ void k_flow_gsum_adam(float* __restrict__ P, const float* __restrict__ part, int nblk, float* __restrict__ Mo,
                                 float* __restrict__ Vo, float lr, float b1t, float b2t, uint2* __restrict__ pk,
                                 float* __restrict__ bias)
{
  cp_wait_previous();
  cp_next_may_launch();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= CP_FLOW_NPARAM) return;
  float s = 0.f;
  int b = 0;
  for (; b + 16 <= nblk; b += 16) {
    float x[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) x[q] = part[(size_t)(b + q) * CP_FLOW_NPARAM + i];
#pragma unroll
    for (int q = 0; q < 16; ++q) s += x[q];
  }
  for (; b < nblk; ++b) s += part[(size_t)b * CP_FLOW_NPARAM + i];
  cp_flow_adam_one(i, 0.f + s, P, Mo, Vo, lr, b1t, b2t);
  cp_flow_pack_one(i, P[i], pk, bias);
}

// the batch's moments (summed over ranks) for the backward pass, and its loss <w^2> / <w>^2
__global__ void k_flow_batch_loss(const double* moments, double n, double* sums, double* loss)
{
  const double a = moments[0], b = moments[1];
  sums[0] = a;
  sums[1] = b;
  const double m = a / n;
  loss[0] = (b / n) / (m * m);
}

// ------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------
// The training buffers of B points, one after the other at multiples of 256 bytes; with base = null
// only their total size.
static size_t carve(void* base, uint64_t B, FlowTrainBufs& t)
{
  size_t at = 0;
  const auto take = [&](size_t bytes) {
    uint8_t* q = static_cast<uint8_t*>(base) + at;
    at += (bytes + 255) & ~(size_t)255;
    return q;
  };
  t.nst = (B + CP_WGT_STAGE - 1) / CP_WGT_STAGE;
  const size_t w16 = CP_FLOW_NC * t.nst * CP_WGT_BYTES(16), w64 = CP_FLOW_NC * t.nst * CP_WGT_BYTES(64);
  t.vj = reinterpret_cast<float4*>(take(sizeof(float4) * B));
  t.wg = reinterpret_cast<float4*>(take(sizeof(float4) * B));
  t.zs = reinterpret_cast<float*>(take(sizeof(float) * 12 * B));
  t.X = take(w16);
  t.H1 = take(w64);
  t.H2 = take(w64);
  t.D1 = take(w64);
  t.D2 = take(w64);
  t.DO = take(w16);
  t.sums = reinterpret_cast<double*>(take(2 * sizeof(double)));
  t.loss = reinterpret_cast<double*>(take(sizeof(double)));
  t.gpart = reinterpret_cast<float*>(take(sizeof(float) * CP_WG_MAXBLK * CP_FLOW_NPARAM));
  return at;
}

static size_t train_bytes(uint64_t B)
{
  FlowTrainBufs t;
  return carve(nullptr, B, t);
}

static size_t bwd_smem() { return sizeof(uint2) * CP_FLOW_NC * CP_FLOW_P_PER + sizeof(float) * CP_FLOW_NC * CP_FLOW_NB; }
static size_t fwd_smem() { return sizeof(uint2) * CP_FLOW_NC * CP_FLOW_P_FWD + sizeof(float) * CP_FLOW_NC * CP_FLOW_NB; }

// Training buffers for `count` points of a step, kept in the handle between the phases of a
// step and between calls.  A new layout (another count) starts from zeros: columns the kernels never write (the
// padding of the 16-wide operands) must read as zero.
static int train_buffers(cp_handle* h, uint64_t count, FlowTrainBufs& t)
{
  h->ftrain_idle = 0;
  if (!h->d_ftrain || count > h->ftrain_cap) {
    if (h->d_ftrain) {
      CP_CUDA(h, cudaStreamSynchronize(h->stream));
      CP_CUDA(h, cudaFree(h->d_ftrain));
      h->d_ftrain = nullptr;
      h->ftrain_cap = 0;
    }
    CP_CUDA(h, cudaMalloc(&h->d_ftrain, train_bytes(count)));
    h->ftrain_cap = count;
    h->ftrain_zeroed = 0;
  }
  if (count != h->ftrain_zeroed) CP_CUDA(h, cudaMemsetAsync(h->d_ftrain, 0, train_bytes(count), h->stream));
  h->ftrain_count = h->ftrain_zeroed = count;
  carve(h->d_ftrain, count, t);
  // per-device attributes: set on every use (host-side, cheap)
  CP_CUDA(h, cudaFuncSetAttribute(k_flow_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bwd_smem()));
  CP_CUDA(h, cudaFuncSetAttribute(k_flow_fwd_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem()));
  return CP_OK;
}

// Gives the training buffers back, unless a step is pending in them.
static void train_release(cp_handle* h)
{
  if (!h->d_ftrain || h->ftrain_count) return;
  cudaStreamSynchronize(h->stream);
  cudaFree(h->d_ftrain);
  h->d_ftrain = nullptr;
  h->ftrain_cap = h->ftrain_zeroed = 0;
}

// A production pass begins: the CP_TRAIN_IDLE-th since the buffers were last used gives them back.  Freeing and
// allocating them again takes 0.8 ms (a pass of 50,021 points: 0.04), so a program that trains and produces in
// turn keeps them, and one that has trained and now produces loses that time once.
#define CP_TRAIN_IDLE 8
void cp_train_idle(cp_handle* h)
{
  if (h->d_ftrain && ++h->ftrain_idle >= CP_TRAIN_IDLE) train_release(h);
}

// Ends a call's use of the training buffers: no step is pending any more, and buffers above
// CP_TRAIN_KEEP bytes go back to the device.  Smaller ones stay in the handle for the next training call
// (batches of 65,536 points: 160 MB), since allocating and freeing them took up to 3 ms of a call, until production
// passes give them back.
#define CP_TRAIN_KEEP ((size_t)1 << 30)
static void train_buffers_done(cp_handle* h)
{
  h->ftrain_count = 0;
  if (train_bytes(h->ftrain_cap) > CP_TRAIN_KEEP) train_release(h);
}

// The kernels of a step are chained launches: each starts its blocks, barriers and constants while the one
// before it drains, and reads what earlier kernels wrote only after its own wait (which alone promises that their
// writes are visible, the weights of the step before among them).  100 steps of 65,536 points: 13.55 -> 12.75 ms.
//
// Phase 1 of a step: forward and integrand over the batch points [point0, point0 + count) at
// counter iteration `iter` (Philox stream 2); moments[0..1] = (sum w, sum w^2) over them.
static int flow_phase_moments(cp_handle* h, const FlowTrainBufs& t, uint64_t point0, uint64_t count, uint32_t iter,
                              double* moments, double* loss_dev = nullptr)
{
  CP_CUDA(h, cp_launch_chained_smem(k_flow_fwd_train, h->num_sms, CP_TRAIN_THREADS, fwd_smem(), h->stream, h->d_flow_pk,
                                    h->d_flow_bias, h->d_edges, h->nb, h->cfg.seed, iter, 2u, point0, count, t.zs, t.vj,
                                    h->mail->status + 1, h->flow_stall));
  const int gblk = h->num_sms * 4;
  int rc = cp_ensure_slots(h, (size_t)2 * gblk);
  if (rc) return rc;
  const float lnTauMin = (float)log(4.0 * h->cfg.pt_hat_min * h->cfg.pt_hat_min / (h->cfg.sqrt_s * h->cfg.sqrt_s));
  CP_CUDA(h, cp_launch_chained(k_flow_igrad, gblk, 128, h->stream, h->P, h->d_cteq, count, lnTauMin, t.vj, t.wg, h->d_slots,
                               h->d_flow_ticket, moments, (double)count, loss_dev));
  return CP_OK;
}

// Phase 2: this handle's points' part of the gradient of the batch loss, from the batch's
// moments over n_batch points, into the gradient buffer G (cleared first); loss_dev = the loss.
// A single handle's loop passes local = true (moments already in t.sums, the loss written by
// phase 1): the per-block partial gradients are left in t.gpart for flow_phase_update_local,
// and *nblk_out receives their number.
static int flow_phase_gradient(cp_handle* h, const FlowTrainBufs& t, uint64_t count, const double* moments,
                               uint64_t n_batch, double* loss_dev, bool local = false, int* nblk_out = nullptr)
{
  if (!local) {
    k_flow_batch_loss<<<1, 1, 0, h->stream>>>(moments, (double)n_batch, t.sums, loss_dev);
    CP_LAUNCH_CHECK(h, "k_flow_batch_loss");
  }
  CP_CUDA(h, cp_launch_chained_smem(k_flow_bwd, h->num_sms, CP_TRAIN_THREADS, bwd_smem(), h->stream, h->d_flow_pk, h->d_flow_bias,
                                    count, (double)n_batch, t.zs, t.vj, t.wg, t.sums, t, (float)h->flow_loss_p,
                                    h->mail->status + 1, h->flow_stall));
  float* G = h->d_flow + CP_FLOW_NPARAM;
  // at most CP_WG_MAXBLK blocks per coupling and layer; chunks are whole multiples of the staged
  // rows.  The three launches share the grid, so together they write every entry of the
  // partial slots 0 .. nblk-1 (all of W1, b1, W2, b2, W3, b3 of every coupling).
  const uint64_t chunk = ((count + CP_WG_MAXBLK - 1) / CP_WG_MAXBLK + CP_WG_ROWS - 1) / CP_WG_ROWS * CP_WG_ROWS;
  const int nblk = (int)((count + chunk - 1) / chunk);
  if (h->flow_kernel == 0) {
    // tensor cores (tcgen05): every coupling and layer shape in one launch
    CP_CUDA(h, cp_launch_chained_smem(k_flow_wgrad_tc, dim3((unsigned)nblk, CP_FLOW_NC, 3), 128, 0, h->stream, t, (int)chunk,
                                      h->mail->status + 1));
  } else {
    // warp-level mma.sync, one launch per layer shape (the cross-check path)
    const dim3 grid((unsigned)nblk, CP_FLOW_NC);
    k_flow_wgrad<16, 64><<<grid, 128, 0, h->stream>>>(t.X, t.D1, t.nst, count, t.gpart, CP_FLOW_W1, 64, 64, (int)chunk,
                                                      CP_FLOW_B1 - CP_FLOW_W1);
    k_flow_wgrad<64, 64><<<grid, 128, 0, h->stream>>>(t.H1, t.D2, t.nst, count, t.gpart, CP_FLOW_W2, 64, 64, (int)chunk,
                                                      CP_FLOW_B2 - CP_FLOW_W2);
    // W3 [64][8] from the 16-wide output-gradient rows (columns 8..15 are zero padding)
    k_flow_wgrad<64, 16><<<grid, 128, 0, h->stream>>>(t.H2, t.DO, t.nst, count, t.gpart, CP_FLOW_W3, 8, 8, (int)chunk,
                                                      CP_FLOW_B3 - CP_FLOW_W3);
    CP_LAUNCH_CHECK(h, "k_flow_wgrad");
  }
  if (local) {
    *nblk_out = nblk;
    return CP_OK;
  }
  CP_CUDA(h, cudaMemsetAsync(G, 0, sizeof(float) * CP_FLOW_NPARAM, h->stream));
  k_flow_gsum<<<(CP_FLOW_NPARAM + 255) / 256, 256, 0, h->stream>>>(t.gpart, nblk, G);
  CP_LAUNCH_CHECK(h, "k_flow_gsum");
  return CP_OK;
}

// Phase 3: Adam step h->flow_t + 1 on the gradient in G (which it clears), BF16 repack.
static int flow_phase_update(cp_handle* h, double lr)
{
  float* G = h->d_flow + CP_FLOW_NPARAM;
  const long step = h->flow_t + 1;
  k_flow_adam<<<(CP_FLOW_NPARAM + 255) / 256, 256, 0, h->stream>>>(
      h->d_flow, G, G + CP_FLOW_NPARAM, G + 2 * CP_FLOW_NPARAM, (float)lr, (float)pow(0.9, (double)step),
      (float)pow(0.999, (double)step));
  CP_LAUNCH_CHECK(h, "k_flow_adam");
  const int rc = cp_flow_repack(h);
  if (rc) return rc;
  h->flow_t = step;
  return CP_OK;
}

// Phase 3 of a single handle's step: the block-order gradient sum, the Adam step and the BF16 repack in
// one kernel (the same parameters and fragments as k_flow_gsum + flow_phase_update).
static int flow_phase_update_local(cp_handle* h, const FlowTrainBufs& t, int nblk, double lr)
{
  float* G = h->d_flow + CP_FLOW_NPARAM;
  const long step = h->flow_t + 1;
  CP_CUDA(h, cp_launch_chained(k_flow_gsum_adam, (CP_FLOW_NPARAM + 127) / 128, 128, h->stream, h->d_flow, t.gpart, nblk,
                               G + CP_FLOW_NPARAM, G + 2 * CP_FLOW_NPARAM, (float)lr, (float)pow(0.9, (double)step),
                               (float)pow(0.999, (double)step), h->d_flow_pk, h->d_flow_bias));
  h->flow_tc_stale = 1;
  h->flow_t = step;
  return CP_OK;
}

extern "C" int cp_flow_set_objective(cp_handle* h, double p)
{
  CP_CHECK_HANDLE(h);
  if (!(p >= 2.0 && p <= 8.0)) return cp_fail(h, CP_ERR_INVALID, "cp_flow_set_objective: p must be in [2, 8]");
  h->flow_loss_p = p;
  return CP_OK;
}

// Trains the flow for n_steps batches of `batch` points on the current VEGAS grid; loss_host
// (n_steps doubles, may be NULL) receives <w^2>/<w>^2 of each batch before its update.  Step s
// draws its batch at counter iteration flow_t (the number of updates so far), points 0..batch-1.
extern "C" int cp_flow_train(cp_handle* h, int n_steps, uint64_t batch, double lr, double* loss_host)
{
  CP_CHECK_HANDLE(h);
  if (!h->d_flow) return cp_fail(h, CP_ERR_INVALID, "flow not initialised (cp_flow_init)");
  if (n_steps < 1 || batch < 64 || batch > (1ull << 24) || (batch & 31))
    return cp_fail(h, CP_ERR_INVALID, "cp_flow_train: batch must be a multiple of 32 in [64, 2^24]");
  int rc = cp_ensure_losses(h, n_steps);
  if (rc) return rc;
  FlowTrainBufs t;
  rc = train_buffers(h, batch, t);
  if (rc) return rc;
  double* losses = h->h_losses;   // each step's last integrand block writes its own
  for (int s = 0; s < n_steps && rc == CP_OK; ++s) {
    int nblk = 0;
    rc = flow_phase_moments(h, t, 0, batch, (uint32_t)h->flow_t, t.sums, losses + s);
    if (!rc) rc = flow_phase_gradient(h, t, batch, t.sums, batch, losses + s, true, &nblk);
    if (!rc) rc = flow_phase_update_local(h, t, nblk, lr);
  }
  const cudaError_t e = cudaStreamSynchronize(h->stream);
  if (!rc && e != cudaSuccess) rc = cp_fail_cuda(h, e, "cp_flow_train");
  if (!rc && loss_host) memcpy(loss_host, losses, sizeof(double) * n_steps);
  if (!rc) rc = cp_flow_tc_status(h);
  train_buffers_done(h);
  return rc;
}

// Loss gradient of one batch without updating (for the gradient checks): grad_host receives
// cp_flow_num_params() floats (dL/dtheta of L = <w^2>/<w>^2), loss_host the batch loss.
extern "C" int cp_flow_loss_grad(cp_handle* h, uint64_t batch, uint32_t iter, float* grad_host, double* loss_host)
{
  CP_CHECK_HANDLE(h);
  if (!h->d_flow) return cp_fail(h, CP_ERR_INVALID, "flow not initialised (cp_flow_init)");
  if (batch < 64 || batch > (1ull << 24) || (batch & 31)) return cp_fail(h, CP_ERR_INVALID, "bad batch");
  FlowTrainBufs t;
  int rc = train_buffers(h, batch, t);
  if (rc) return rc;
  float* G = h->d_flow + CP_FLOW_NPARAM;
  rc = flow_phase_moments(h, t, 0, batch, iter, t.sums);
  if (!rc) rc = flow_phase_gradient(h, t, batch, t.sums, batch, t.loss);
  cudaError_t e = cudaSuccess;
  if (!rc) {
    e = cudaMemcpyAsync(grad_host, G, sizeof(float) * CP_FLOW_NPARAM, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess && loss_host) e = cudaMemcpyAsync(loss_host, t.loss, sizeof(double), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(G, 0, sizeof(float) * CP_FLOW_NPARAM, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) rc = cp_fail_cuda(h, e, "cp_flow_loss_grad readback");
  }
  if (!rc) rc = cp_flow_tc_status(h);
  train_buffers_done(h);
  return rc;
}

// ------------------------------------------------------------------------------------------
// Data-parallel training: one step in three calls, the caller summing over ranks in between.
// ------------------------------------------------------------------------------------------
extern "C" int cp_flow_step_moments(cp_handle* h, uint64_t point0, uint64_t count, double* moments_dev)
{
  CP_CHECK_HANDLE(h);
  if (!h->d_flow) return cp_fail(h, CP_ERR_INVALID, "flow not initialised (cp_flow_init)");
  if (count < 1 || count > (1ull << 24) || !moments_dev)
    return cp_fail(h, CP_ERR_INVALID, "cp_flow_step_moments: count must be in [1, 2^24]");
  FlowTrainBufs t;
  int rc = train_buffers(h, count, t);
  if (rc) return rc;
  return flow_phase_moments(h, t, point0, count, (uint32_t)h->flow_t, moments_dev);
}

extern "C" int cp_flow_step_gradient(cp_handle* h, const double* moments_dev, uint64_t batch_total, float* grad_dev,
                                     double* loss_host)
{
  CP_CHECK_HANDLE(h);
  if (!h->d_ftrain || !h->ftrain_count || !moments_dev || batch_total < h->ftrain_count)
    return cp_fail(h, CP_ERR_INVALID, "cp_flow_step_gradient: call cp_flow_step_moments first (batch_total >= count)");
  FlowTrainBufs t;
  carve(h->d_ftrain, h->ftrain_count, t);
  int rc = flow_phase_gradient(h, t, h->ftrain_count, moments_dev, batch_total, t.loss);
  if (rc) return rc;
  if (grad_dev)
    CP_CUDA(h, cudaMemcpyAsync(grad_dev, h->d_flow + CP_FLOW_NPARAM, sizeof(float) * CP_FLOW_NPARAM,
                               cudaMemcpyDeviceToDevice, h->stream));
  if (loss_host) CP_CUDA(h, cudaMemcpyAsync(loss_host, t.loss, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  return cp_flow_tc_status(h);   // synchronises the stream
}

extern "C" int cp_flow_step_update(cp_handle* h, const float* grad_dev, double lr)
{
  CP_CHECK_HANDLE(h);
  if (!h->d_flow) return cp_fail(h, CP_ERR_INVALID, "flow not initialised (cp_flow_init)");
  if (!(lr > 0.0)) return cp_fail(h, CP_ERR_INVALID, "cp_flow_step_update: lr must be positive");
  if (grad_dev)
    CP_CUDA(h, cudaMemcpyAsync(h->d_flow + CP_FLOW_NPARAM, grad_dev, sizeof(float) * CP_FLOW_NPARAM,
                               cudaMemcpyDeviceToDevice, h->stream));
  return flow_phase_update(h, lr);
}
