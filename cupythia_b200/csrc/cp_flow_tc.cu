// cp_flow_tc.cu -- the flow forward (sampling) pass on the 5th-generation tensor cores.
//
// Same map as k_flow_fwd (Philox words -> VEGAS map -> logit -> 4 affine couplings -> sigmoid),
// with every dense layer as tcgen05.mma over 128-point tiles: B (weights) in shared memory, the
// FP32 accumulator and A (activations) in TMEM.
//
// Launch: one persistent CTA per SM of 5 warpgroups, each with one tile in flight at a time; thread r
// of a warpgroup is row r (one point) of the tile and TMEM lane r.  A tile has 96 TMEM columns: the
// accumulator (64) and the A operand (32: 64 BF16 in pairs).  Per coupling it has three steps
//   layer 1 done: accumulator -> ReLU -> BF16 pairs -> A operand; layer 2 is issued
//   layer 2 done: the same; layer 3 is issued
//   layer 3 done: read the 4 output columns, update the point, write the next coupling's layer-1 input
//     (8 columns of A); its layer 1 is issued
// and after the last coupling the next tile's layer 1 is issued first (its points are drawn while the last
// layer 3 runs), so the finished points' output runs beside it.  After each step the warpgroup's
// warps meet at a named barrier and its first warp issues the layer, from warp-uniform operands (formed
// by one lane of a divergent warp they cost a move per operand: five MMAs took 253 cycles to issue, now
// 80).  The biases of layers 1 and 2 are part of the MMAs: layer 1 has them as input
// columns 14 and 15 (constant 1) times weight rows holding the BF16 high and low parts of the
// FP32 bias; layer 2 adds one K = 16 MMA of a constant block (columns 0 and 1 equal to 1) against
// the hi/lo bias rows (hi + lo reproduces the FP32 bias to about 2^-17 relative).  Layer 3's
// biases are added in FP32 by the coupling update: its 2 or 4 outputs per point cost as many
// adds, against one more MMA per tile step.
//
// What bounds it: the round trips of a tile's 12 steps (about 195 of 710 cycles each are the MMAs'), with
// 55% of the issue slots and 54% of the tensor pipe's cycles taken.  With A in shared memory an MMA of
// 128 x 64 x 16 takes 48 cycles, the time to read A and B (6 KB at 128 B per cycle), against 32 with A in
// TMEM, and the epilogues' stores share that bandwidth.  TMEM then holds 5 tiles of 96 columns, against 8
// of 64 with A in shared memory.  2^26 points on a B200: 5.22 ms with two tiles per warpgroup, A in shared
// memory and issuing warps of their own; 4.66 with those warps' operands uniform; 3.63 with 8 tiles in 8
// warpgroups and no issuing warps; 3.15 with A in TMEM (4 tiles in flight: 3.42; 6 with half of A in
// shared memory: 3.19, and 3.61 with 5 of those).
//
// A production form (k_flow_accept_tc, opt-in through cp_flow_fuse_production) instantiates the
// same body and takes each finished tile on, from registers, through the integrand and the
// accept step of the production pass (the code of k_unw_accept, shared through cp_unweight.cuh),
// so no flow output is stored.  Its records equal the two-kernel path's byte for byte; the time is about
// the same (2^26 points: 6.4 ms, against 3.1 + 3.1 for the two kernels; 9.6 before this layout).
//
// Synchronisation: rows written by tcgen05.st (waited for) are ordered before the MMAs by the
// warpgroup's barrier; the issuing warp commits to the tile's mbarrier, which the warpgroup waits on before
// reading TMEM.  Every wait on it is bounded (about 1 s of clock without progress); on expiry the waiting
// warp raises its warpgroup's abort flag and issues no more, the warpgroup's warps run through their tiles without
// waiting or touching TMEM, the issuing warp waits (bounded) for the MMAs it still has in flight, every warp
// that gave up sets *status, and the kernel releases its TMEM.
#include "cp_flow.cuh"
#include "cp_internal.cuh"
#include "cp_tc.cuh"
#include "cp_unweight.cuh"

// weight image of one coupling, bytes (K-major, no swizzle; see cp_tc.cuh)
#define CP_TC_B1 0        // [N 64][K 16]: W1 rows 0..n_in-1, bias hi/lo in K 14/15
#define CP_TC_B2 2048     // [N 64][K 64]: W2
#define CP_TC_B2B 10240   // [N 64][K 16]: b2 hi/lo in K 0/1
#define CP_TC_B3 12288    // [N 16][K 64]: W3 (outputs 0..7, rest zero)
#define CP_TC_PER 14336
#define CP_TC_IMG (CP_FLOW_NC * CP_TC_PER)
#define CP_TC_TMEM_COLS 512                     // all of an SM's TMEM
#define CP_TC_A 64                              // tile's TMEM column of the A operand, after the 64 of the accumulator
#define CP_TC_COLS 96                           // TMEM columns of a tile
#define CP_TC_ONES 480                          // TMEM column of the constant block [128][16]: columns 0 and 1 of a row are 1
#define CP_TC_ONE2 0x3F803F80u                  // two BF16 ones
#define CP_TC_WG 5                              // warpgroups per CTA, one tile each

// Shared-memory layout of a CTA, bytes from the 1024-aligned base.
struct CpTcLayout {
  static constexpr int THREADS = CP_TC_WG * 128;
  static constexpr int EDGE = CP_TC_IMG;
  static constexpr int MISC = EDGE + 3 * CP_MAX_BINS * 8;  // mbarriers, TMEM address, abort flags
  static constexpr int B3 = MISC + 256;                    // FP32 layer-3 biases, 8 per coupling
  static constexpr int RED = B3 + 128;                     // production form: per-warp sums
  static constexpr int SMEM = RED + CP_TC_WG * 4 * 7 * 8 + 1024;        // + 1024-byte base alignment slack
  static_assert(RED % 16 == 0, "sums must stay aligned");
  static_assert(SMEM < (1 << 18), "descriptor offsets are added to the 14-bit address field");
  static_assert(SMEM <= 227 * 1024, "shared memory budget");
  static_assert(CP_TC_WG * CP_TC_COLS <= CP_TC_ONES && CP_TC_ONES + 8 <= CP_TC_TMEM_COLS, "TMEM columns");
};

static_assert(CP_TC_PER % 16 == 0, "coupling images are whole descriptor units");

constexpr uint32_t CP_TC_IDESC64 = cp_tc_idesc_bf16(64);
constexpr uint32_t CP_TC_IDESC16 = cp_tc_idesc_bf16(16);

// byte offset of element (row r, column k) in a K-major no-swizzle tile of R rows
__host__ __device__ __forceinline__ int cp_tc_off(int r, int k, int R) { return (k >> 3) * (R * 16) + (r >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2; }

__device__ __forceinline__ uint16_t cp_bf16_bits(float v)
{
  __nv_bfloat16 b = __float2bfloat16_rn(v);
  return *reinterpret_cast<uint16_t*>(&b);
}
__device__ __forceinline__ void cp_bf16_split(float v, uint16_t& hi, uint16_t& lo)
{
  hi = cp_bf16_bits(v);
  lo = cp_bf16_bits(v - __uint_as_float((uint32_t)hi << 16));
}

// FP32 master parameters -> the shared-memory weight image of every coupling
__global__ void k_flow_pack_tc(const float* __restrict__ P, uint8_t* __restrict__ img)
{
  const int c = blockIdx.x;
  const CpCoupling kc = cp_coupling(c);
  const float* W1 = P + c * CP_FLOW_PER + CP_FLOW_W1;
  const float* b1 = P + c * CP_FLOW_PER + CP_FLOW_B1;
  const float* W2 = P + c * CP_FLOW_PER + CP_FLOW_W2;
  const float* b2 = P + c * CP_FLOW_PER + CP_FLOW_B2;
  const float* W3 = P + c * CP_FLOW_PER + CP_FLOW_W3;
  uint8_t* q = img + c * CP_TC_PER;
  for (int e = threadIdx.x; e < CP_TC_PER / 2; e += blockDim.x) {
    uint16_t v = 0, hi, lo;
    int off;
    if (e < 1024) {                       // B1 [64][16]
      const int nn = e >> 4, k = e & 15;
      off = CP_TC_B1 + cp_tc_off(nn, k, 64);
      cp_bf16_split(b1[nn], hi, lo);
      if (k < kc.nin) v = cp_bf16_bits(W1[k * 64 + nn]);
      else if (k == 14) v = hi;
      else if (k == 15) v = lo;
    } else if (e < 5120) {                // B2 [64][64]
      const int i = e - 1024, nn = i >> 6, k = i & 63;
      off = CP_TC_B2 + cp_tc_off(nn, k, 64);
      v = cp_bf16_bits(W2[k * 64 + nn]);
    } else if (e < 6144) {                // B2B [64][16]
      const int i = e - 5120, nn = i >> 4, k = i & 15;
      off = CP_TC_B2B + cp_tc_off(nn, k, 64);
      cp_bf16_split(b2[nn], hi, lo);
      v = k == 0 ? hi : (k == 1 ? lo : (uint16_t)0);
    } else {                              // B3 [16][64]
      const int i = e - 6144, nn = i >> 6, k = i & 63;
      off = CP_TC_B3 + cp_tc_off(nn, k, 16);
      if (nn < 8) v = cp_bf16_bits(W3[k * 8 + nn]);
    }
    *reinterpret_cast<uint16_t*>(q + off) = v;
  }
}

// Elementwise transforms of the tensor-core path with the hardware approximations (lg2/ex2 and
// fast reciprocal; absolute errors of a few 1e-7 in z and ln J).  The log-Jacobian uses the same
// computed quantities as the map (z' = z e^s + t with ln J += s), so the weights stay consistent.
// Natural logarithm of a normal x, exponential of an x whose e^x may flush to zero when denormal, and
// quotient of normal values, from the flush-to-zero forms of the instructions: the range handling of the
// other forms (a compare, a scaling and its undoing around each) is for denormals, which these arguments
// never are (same bits; 100 of 1,276 instructions per tile and warp, 2^26 points 4.65 -> 4.54 ms).
__device__ __forceinline__ float cp_tc_ln(float x)
{
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y * 0.693147182f;
}
__device__ __forceinline__ float cp_tc_exp(float x)
{
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.44269502f));
  return y;
}
__device__ __forceinline__ float cp_tc_div(float a, float b)
{
  float y;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}
__device__ __forceinline__ float cp_tc_logit(float u, float& z)
{
  const float lu = cp_tc_ln(u), l1u = cp_tc_ln(1.f - u);
  z = lu - l1u;
  return -(lu + l1u);
}
__device__ __forceinline__ float cp_tc_sigmoid(float z, float& v)
{
  const float e = __expf(-fabsf(z));
  const float inv = cp_tc_div(1.f, 1.f + e);
  v = z >= 0.f ? inv : e * inv;
  return -fabsf(z) - 2.f * cp_tc_ln(1.f + e);
}
// CP_FLOW_S tanh(x / CP_FLOW_S) from one exponential
__device__ __forceinline__ float cp_tc_softclamp(float x)
{
  const float a = fabsf(x) * (2.f / CP_FLOW_S);
  const float t = cp_tc_exp(-a);
  return copysignf(CP_FLOW_S * cp_tc_div(1.f - t, 1.f + t), x);
}

struct CpTcPoint {
  float z0, z1, z2, ld;
};

__device__ __forceinline__ float cp_sel3(const CpTcPoint& t, int i) { return i == 0 ? t.z0 : (i == 1 ? t.z1 : t.z2); }

// this thread's row of the layer-1 input of coupling c, (in0, in1, 0 ... 0, 1, 1), to the A operand
__device__ __forceinline__ void cp_tc_write_in(uint32_t ta, int c, const CpTcPoint& t)
{
  const CpCoupling k = cp_coupling(c);
  const float in0 = cp_sel3(t, k.cin[0]);
  const float in1 = k.nin > 1 ? cp_sel3(t, k.cin[1]) : 0.f;
  const uint32_t r[8] = {cp_bf2(in0, in1), 0u, 0u, 0u, 0u, 0u, 0u, CP_TC_ONE2};
  cp_tc_st8(ta, r);
  cp_tc_wait_st();
}

// d = the tile's accumulator, a = its A operand; b64 / b16 = descriptors of the weight image base with
// the LBO of the N = 64 and N = 16 operands; an operand at byte offset o from the base adds o >> 4 to
// the start-address field (every shared address here is below 2^18, so the 14-bit field never
// carries).  bw = the coupling's image offset >> 4.
__device__ __forceinline__ void cp_tc_issue_l1(uint32_t d, uint32_t a, uint64_t b64, uint32_t bw)
{
  cp_tc_mma_ts(d, a, b64 + bw + (CP_TC_B1 >> 4), CP_TC_IDESC64, 0u);
}
__device__ __forceinline__ void cp_tc_issue_l2(uint32_t d, uint32_t a, uint32_t ones, uint64_t b64, uint32_t bw)
{
#pragma unroll
  for (int j = 0; j < 4; ++j)
    cp_tc_mma_ts(d, a + 8 * j, b64 + bw + ((CP_TC_B2 + j * 2048) >> 4), CP_TC_IDESC64, j > 0 ? 1u : 0u);
  cp_tc_mma_ts(d, ones, b64 + bw + (CP_TC_B2B >> 4), CP_TC_IDESC64, 1u);
}
__device__ __forceinline__ void cp_tc_issue_l3(uint32_t d, uint32_t a, uint64_t b16, uint32_t bw)
{
#pragma unroll
  for (int j = 0; j < 4; ++j)
    cp_tc_mma_ts(d, a + 8 * j, b16 + bw + ((CP_TC_B3 + j * 512) >> 4), CP_TC_IDESC16, j > 0 ? 1u : 0u);
}

// waits for the tile's MMAs; live turns false (for the whole warp) when the wait gives up, and then nothing is
// waited for any more: the warpgroup's tiles run out at once, with their results invalid
__device__ __forceinline__ void cp_tc_wait(uint32_t mbar, uint32_t& phase, volatile int* abort, bool& live)
{
  if (live && !__all_sync(0xffffffffu, cp_mbar_try(mbar, phase)))
    live = __all_sync(0xffffffffu, cp_mbar_wait_bounded(mbar, phase, abort)) && live;
  phase ^= 1u;
  cp_tc_fence_after();
}

// 32 accumulators of this thread's row -> ReLU -> 16 BF16 pairs
__device__ __forceinline__ void cp_tc_relu_pairs(const uint32_t (&r)[32], uint32_t (&w)[16])
{
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = cp_relu_bf2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}

// accumulator [row][0:64] -> ReLU -> BF16 pairs -> A operand (hidden unit k in column k / 2)
__device__ __forceinline__ void cp_tc_hidden(uint32_t taddr)
{
  uint32_t r0[32], r1[32], w[16];
  cp_tc_ld32_start(taddr, r0);
  cp_tc_ld32_start(taddr + 32, r1);
  cp_tc_ld32_done(r0);
  cp_tc_ld32_done(r1);
  cp_tc_relu_pairs(r0, w);
  cp_tc_st16(taddr + CP_TC_A, w);
  cp_tc_relu_pairs(r1, w);
  cp_tc_st16(taddr + CP_TC_A + 16, w);
  cp_tc_wait_st();
}

// The kernel body.  Sampling form (ACCEPT false): each point's (v, ln J) goes to out.  Production
// form (ACCEPT true, draws of stream 0): each point goes straight on, from registers, through the
// integrand and the accept step of the production pass (cp_unw_point, the code of k_unw_accept), and each
// CTA leaves its sums in its slot of L->slots; the record builder then runs unchanged.
template <bool ACCEPT>
__device__ __forceinline__ void cp_flow_tc_body(const uint4* __restrict__ img_g, const float* __restrict__ params,
                                                const double* __restrict__ edges, int nb, uint64_t seed, uint64_t point0,
                                                uint64_t n, uint32_t iter, uint32_t stream, float4* __restrict__ out,
                                                float* __restrict__ uout, int* __restrict__ status, int stall,
                                                const CpHadParams* P,
                                                const UnwLaunch* L)
{
  using Lay = CpTcLayout;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = cp_smem_u32(smem_raw);
  const uint32_t pad = ((raw + 1023u) & ~1023u) - raw;
  uint8_t* sm = smem_raw + pad;
  const uint32_t sbase = raw + pad;
  float2* sEdge = reinterpret_cast<float2*>(sm + Lay::EDGE);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + Lay::MISC);   // [0, 8) the tiles' MMAs, [8, 16) last commits
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + Lay::MISC + 128);
  int* abort_flags = reinterpret_cast<int*>(sm + Lay::MISC + 144);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), wg = warp >> 2, row = tid & 127;

  for (int e = tid; e < CP_TC_IMG / 16; e += Lay::THREADS) reinterpret_cast<uint4*>(sm)[e] = img_g[e];
  float* sB3 = reinterpret_cast<float*>(sm + Lay::B3);
  if (tid < CP_FLOW_NC * 8) sB3[tid] = params[(tid >> 3) * CP_FLOW_PER + CP_FLOW_B3 + (tid & 7)];
  for (int k = tid; k < 3 * nb; k += Lay::THREADS) {
    const int d = k / nb, b = k - d * nb;
    const double lo = edges[d * (nb + 1) + b], hi = edges[d * (nb + 1) + b + 1];
    sEdge[d * CP_MAX_BINS + b] = make_float2((float)lo, (float)(hi - lo));
  }
  double* sRed = reinterpret_cast<double*>(sm + Lay::RED);   // [4 CP_TC_WG warps][7]
  if (tid < CP_TC_WG) abort_flags[tid] = 0;
  if (tid == 0) {
    for (int i = 0; i < 16; ++i) cp_mbar_init(cp_smem_u32(&mbar[i]), 1);
    cp_mbar_init_fence();
  }
  if (warp == 0) {
    cp_tc_alloc(cp_smem_u32(tmem_slot), CP_TC_TMEM_COLS);
    cp_tc_relinquish();
  }
  cp_fence_proxy_async();
  cp_tc_fence_before();
  __syncthreads();
  cp_tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;
  if (wg == 0) {
    const uint32_t r[8] = {CP_TC_ONE2, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
    cp_tc_st8(tmem + CP_TC_ONES + lane_base, r);
    cp_tc_wait_st();
    cp_tc_fence_before();
  }
  __syncthreads();
  cp_tc_fence_after();
  const uint64_t tiles = (n + 127) / 128;
  const uint64_t stride = (uint64_t)gridDim.x * CP_TC_WG;
  volatile int* abort = abort_flags + wg;
  const uint32_t bar_id = 1 + wg;
  const uint64_t b64 = cp_tc_desc(sbase, 1024, 128), b16 = cp_tc_desc(sbase, 256, 128);
  const uint32_t td = tmem + (uint32_t)(wg * CP_TC_COLS), ta = td + CP_TC_A, mb = cp_smem_u32(&mbar[wg]);
  uint32_t ph = 0;
  bool live = stall != 1;     // MMAs are issued, and no wait of this warp has given up
  if (stall == 1) cp_mbar_wait_bounded(mb, 0u, abort);     // test hook: nothing is issued, so the wait expires
  // the warpgroup's rows of a step are written: its warps meet, one of them issues the next layer
  // (lay of coupling c) from warp-uniform operands
  auto publish = [&](int lay, int c) {
    cp_tc_fence_before();
    cp_bar_wg(bar_id);
    if ((warp & 3) == 0 && live) {
      cp_tc_fence_after();
      const uint32_t bw = (uint32_t)c * (CP_TC_PER >> 4);
      if (cp_elect()) {
        if (lay == 0) cp_tc_issue_l1(td, ta, b64, bw);
        else if (lay == 1) cp_tc_issue_l2(td, ta, tmem + CP_TC_ONES, b64, bw);
        else cp_tc_issue_l3(td, ta, b16, bw);
        cp_tc_commit(mb);
      }
      __syncwarp();
    }
  };
  CpTcPoint t;
  [[maybe_unused]] float u = 0.f;    // the accept draw
  [[maybe_unused]] CpUnwSums S;
  [[maybe_unused]] const float wmax = ACCEPT ? (float)L->wmax[0] : 0.f;
  // a tile's start: Philox words -> VEGAS map -> logit, layer-1 input (not published)
  auto start = [&](uint64_t qq, CpTcPoint& x, float& draw) {
    const uint64_t p = qq * 128 + row;
    uint32_t w[4] = {0x80000000u, 0x80000000u, 0x80000000u, 0u};
    if (p < n) cp_point_words(seed, point0 + p, iter, stream, w);
    if (ACCEPT || uout) draw = cp_u24(w[3]);
    float jv = 1.f, ld = 0.f, z[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      int bin;
      const float xv = cp_flow_vegas_in(sEdge + d * CP_MAX_BINS, nb, w[d], jv, bin);
      ld += cp_tc_logit(xv, z[d]);
    }
    x.z0 = z[0]; x.z1 = z[1]; x.z2 = z[2];
    x.ld = ld + __logf(jv);
  };
  uint64_t q = (uint64_t)wg * gridDim.x + blockIdx.x;
  if (q < tiles) {
    start(q, t, u);
    __syncwarp();
    cp_tc_write_in(ta + lane_base, 0, t);
    publish(0, 0);
  }
  for (; q < tiles; q += stride) {
    const uint64_t qn = q + stride;
    // unrolled: each coupling's input and transformed dimensions are compile-time constants
#pragma unroll
    for (int c = 0; c < CP_FLOW_NC; ++c) {
      // layer-1 output -> layer 2
      cp_tc_wait(mb, ph, abort, live);
      if (live) cp_tc_hidden(td + lane_base);
      publish(1, c);
      // layer-2 output -> layer 3
      cp_tc_wait(mb, ph, abort, live);
      if (live) cp_tc_hidden(td + lane_base);
      publish(2, c);
      // layer-3 output -> coupling update, next coupling's layer 1
      const CpCoupling k = cp_coupling(c);
      const bool last = c + 1 == CP_FLOW_NC;
      float b3[4];
#pragma unroll
      for (int j = 0; j < 2 * k.nt; ++j) b3[j] = sB3[8 * c + j];
      // the next tile's points are drawn while layer 3 runs
      CpTcPoint nx;
      float nu = 0.f;
      if (last && qn < tiles) start(qn, nx, nu);
      cp_tc_wait(mb, ph, abort, live);
      float o[4] = {0.f, 0.f, 0.f, 0.f};
      if (live) cp_tc_ld4(td + lane_base, o);
      if (last && qn < tiles) {
        if (live) cp_tc_write_in(ta + lane_base, 0, nx);
        publish(0, 0);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (j >= k.nt) break;
        const float sc = cp_tc_softclamp(o[j] + b3[j]), sh = o[k.nt + j] + b3[k.nt + j];
        const int d = k.tr[j];
        const float zn = fmaf(cp_sel3(t, d), cp_tc_exp(sc), sh);
        if (d == 0) t.z0 = zn;
        else if (d == 1) t.z1 = zn;
        else t.z2 = zn;
        t.ld += sc;
      }
      if (!last) {
        if (live) cp_tc_write_in(ta + lane_base, c + 1, t);
        publish(0, c + 1);
      } else {
        // the tile's points are done: their output runs beside the next tile's layer 1
        float v0, v1, v2;
        float ld = t.ld;
        ld += cp_tc_sigmoid(t.z0, v0);
        ld += cp_tc_sigmoid(t.z1, v1);
        ld += cp_tc_sigmoid(t.z2, v2);
        const uint64_t p = q * 128 + row;
        if constexpr (ACCEPT) {
          cp_unw_point(*P, P->cteq, *L, wmax, p, v0, v1, v2, expf(ld), u, S);
        } else {
          if (p < n) {
            out[p] = make_float4(v0, v1, v2, ld);
            if (uout) uout[p] = u;   // the accept draw, so the accept kernel need not redraw it
          }
        }
        if (qn < tiles) {
          t = nx;
          u = nu;
        }
      }
    }
  }
  // test hook: the last warp of a warpgroup gives up when the others are through (no arrival comes on this barrier)
  if (stall == 2 && (warp & 3) == 3) live = __all_sync(0xffffffffu, cp_mbar_wait_bounded(cp_smem_u32(&mbar[CP_TC_WG]), 0u, abort));
  // After an abort MMAs may still be in flight: every one this warpgroup issued has completed (bounded
  // wait) before the CTA releases its TMEM.
  if ((warp & 3) == 0 && stall != 1) {
    const uint32_t fin = cp_smem_u32(&mbar[8 + wg]);
    if (cp_elect()) cp_tc_commit(fin);
    __syncwarp();
    volatile int fin_abort = 0;
    live = __all_sync(0xffffffffu, cp_mbar_wait_bounded(fin, 0u, &fin_abort)) && live;
  }
  // every warp reports its own: no barrier follows its last wait, so another warp's flag may come too late to be seen
  if (!live && (tid & 31) == 0) *(volatile int*)status = 1;
  if constexpr (ACCEPT) {
    double v[7];
    cp_unw_warp_sums(S, v);
    if ((tid & 31) == 0)
      for (int k = 0; k < 7; ++k) sRed[warp * 7 + k] = v[k];
  }
  cp_tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    cp_tc_fence_after();
    cp_tc_dealloc(tmem, CP_TC_TMEM_COLS);
  }
  if constexpr (ACCEPT) {
    if (tid == 0) {   // the CTA's sums, warps in a fixed order
      double* slot = L->slots + (size_t)blockIdx.x * CP_UNW_SLOT;
      for (int k = 0; k < 7; ++k) {
        double acc = 0.0;
        for (int q = 0; q < 4 * CP_TC_WG; ++q) acc = (k == 2) ? fmax(acc, sRed[q * 7 + k]) : acc + sRed[q * 7 + k];
        slot[k] = acc;
      }
      slot[7] = 0.0;
    }
  }
}

__global__ void __launch_bounds__(CpTcLayout::THREADS, 1)
    k_flow_fwd_tc(const uint4* __restrict__ img_g, const float* __restrict__ params, const double* __restrict__ edges,
                  int nb, uint64_t seed, uint64_t point0, uint64_t n, uint32_t iter, uint32_t stream,
                  float4* __restrict__ out, float* __restrict__ uout, int* __restrict__ status, int stall)
{
  cp_flow_tc_body<false>(img_g, params, edges, nb, seed, point0, n, iter, stream, out, uout, status, stall,
                                   nullptr, nullptr);
}

// Production form: flow forward, integrand and accept step of the points [L.point0, L.point0 + L.n)
// in one pass (draws of stream 0, as k_unw_accept takes them), one CTA per SM.
__global__ void __launch_bounds__(CpTcLayout::THREADS, 1)
    k_flow_accept_tc(const uint4* __restrict__ img_g, const float* __restrict__ params,
                     const __grid_constant__ CpHadParams P, const __grid_constant__ UnwLaunch L,
                     int* __restrict__ status, int stall)
{
  cp_flow_tc_body<true>(img_g, params, L.edges, L.nb, L.seed, L.point0, L.n, L.iter, 0u, nullptr,
                                      nullptr, status, stall, &P, &L);
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
int cp_flow_tc_repack(cp_handle* h)
{
  k_flow_pack_tc<<<CP_FLOW_NC, 256, 0, h->stream>>>(h->d_flow, h->d_flow_tc);
  CP_LAUNCH_CHECK(h, "k_flow_pack_tc");
  return CP_OK;
}

int cp_flow_tc_alloc(cp_handle* h)
{
  if (!h->d_flow_tc) CP_CUDA(h, cudaMalloc(&h->d_flow_tc, CP_TC_IMG));
  CP_CUDA(h, cudaFuncSetAttribute(k_flow_fwd_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, CpTcLayout::SMEM));
  CP_CUDA(h, cudaFuncSetAttribute(k_flow_accept_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  CpTcLayout::SMEM));
  return CP_OK;
}

int cp_flow_tc_enqueue(cp_handle* h, uint64_t point0, uint64_t n, uint32_t iter, uint32_t stream, float4* out,
                       float* uout)
{
  if (h->flow_tc_stale) {
    const int rc = cp_flow_tc_repack(h);
    if (rc) return rc;
    h->flow_tc_stale = 0;
  }
  const uint64_t tiles = (n + 127) / 128;
  const int grid = (int)(tiles < (uint64_t)h->num_sms ? tiles : (uint64_t)h->num_sms);
  if (grid < 1) return CP_OK;
  k_flow_fwd_tc<<<grid, CpTcLayout::THREADS, CpTcLayout::SMEM, h->stream>>>(reinterpret_cast<const uint4*>(h->d_flow_tc), h->d_flow,
                                                                 h->d_edges,
                                                                 h->nb, h->cfg.seed, point0, n, iter, stream, out,
                                                                 uout, h->mail->status, h->flow_stall);
  CP_LAUNCH_CHECK(h, "k_flow_fwd_tc");
  return CP_OK;
}

// Enqueues the production form over the chunk L (its staging and range totals ready); *blocks =
// the CTAs launched, each of which writes its slot of L.slots.
int cp_flow_tc_accept_enqueue(cp_handle* h, const UnwLaunch& L, int* blocks)
{
  *blocks = 0;
  if (h->flow_tc_stale) {
    const int rc = cp_flow_tc_repack(h);
    if (rc) return rc;
    h->flow_tc_stale = 0;
  }
  const uint64_t tiles = (L.n + 127) / 128;
  const int grid = (int)(tiles < (uint64_t)h->num_sms ? tiles : (uint64_t)h->num_sms);
  if (grid < 1) return CP_OK;
  using Lay = CpTcLayout;
  k_flow_accept_tc<<<grid, Lay::THREADS, Lay::SMEM, h->stream>>>(reinterpret_cast<const uint4*>(h->d_flow_tc),
                                                                  h->d_flow, h->P, L, h->mail->status, h->flow_stall);
  CP_LAUNCH_CHECK(h, "k_flow_accept_tc");
  *blocks = grid;
  return CP_OK;
}

// Synchronises the handle's stream, then reads and clears the status words of the tensor-core
// kernels (mapped host memory): CP_ERR_TIMEOUT if a bounded wait expired since the last check.
int cp_flow_tc_status(cp_handle* h)
{
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  const bool wgrad = h->mail->status[1] != 0;
  if (!h->mail->status[0] && !wgrad) return CP_OK;
  h->mail->status[0] = h->mail->status[1] = 0;
  return cp_fail(h, CP_ERR_TIMEOUT, wgrad ? "flow training: a tensor-core or weight-copy wait expired (this training step is invalid)"
                                            : "k_flow_fwd_tc / k_flow_accept_tc: a tensor-core wait expired (results of this pass are invalid)");
}

// Test hook of the failure path: with on != 0 no layer is issued, so the first bounded
// wait of the epilogue expires (about one second of clock), the kernel raises its status word and
// releases its TMEM, and the call returns CP_ERR_TIMEOUT with the context still usable.  With on = 2 the layers
// are issued and the last warp of each warpgroup waits in vain after its last tile.  In training on = 1 leaves out the
// copies of the weights into shared memory, whose bounded waits expire.
extern "C" int cp_flow_test_stall(cp_handle* h, int on)
{
  CP_CHECK_HANDLE(h);
  h->flow_stall = on == 2 ? 2 : on != 0;
  return CP_OK;
}
