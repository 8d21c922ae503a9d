// cp_vegas.cu -- the fused hadronic VEGAS iteration and its FP64 reduction / refinement.
//
// One persistent kernel per iteration: every thread draws its points' Philox words, maps them
// through the VEGAS grid (edges staged in shared memory as FP32 (lo, width) pairs) and the
// analytic (tau, y, z) base map, evaluates the FP32 integrand in registers, and accumulates
//   sum w, sum w^2   Kahan-compensated FP32 per thread, compensated warp and block trees,
//   max w, n_bad     per thread, then warp / block,
//   sum w^2 per bin  warp-private shared-memory histograms, deterministic lane-order adds.
// Each block writes one FP64 slot; a second kernel, one cluster of blocks, reduces the slots in a fixed order (FP64)
// and its first block refines the grid in FP64, so iterations chain on the stream
// without host round trips (the reference round-trips through the host every iteration:
// cuPythia/11_vegas_importance/vegas.cu:107-124).
#include <cooperative_groups.h>

#include <mutex>

#include "cp_internal.cuh"

struct HadLaunch {
  uint64_t seed, point0, n;
  uint32_t iter, stream;
  int nb;
  const double* edges;
  double* slots;   // gridDim.x * (CP_SLOT_HEAD + 3 nb)
  float* w_out;    // optional per-point weights
  float* x_out;    // optional per-point mapped x (3 per point)
  unsigned long long* qhist;   // weight histogram (CP_QBINS), integer adds; or null: not wanted
  const float4* flow;          // flow output (v, ln J) per point, or null: map the Philox words
};

template <bool WRITE>
__global__ void __launch_bounds__(CP_THREADS, CP_MIN_BLOCKS) k_had_accum(const __grid_constant__ CpHadParams P,
                                                                          const __grid_constant__ HadLaunch L)
{
  __shared__ float2 sEdge[3][CP_MAX_BINS];
  __shared__ float sHist[CP_WARPS][3][CP_MAX_BINS];
  __shared__ float sRed[CP_WARPS][6];
  __shared__ unsigned sQ[CP_QBINS];
  const int nb = L.nb;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  cp_next_may_launch();
  for (int k = threadIdx.x; k < CP_WARPS * 3 * CP_MAX_BINS; k += CP_THREADS)
    (&sHist[0][0][0])[k] = 0.f;
  if (L.qhist)
    for (int k = threadIdx.x; k < CP_QBINS; k += CP_THREADS) sQ[k] = 0u;
  cp_wait_previous();   // the grid, and the slots and histogram that the pass before may still read
  for (int k = threadIdx.x; k < 3 * nb; k += CP_THREADS) {
    int d = k / nb, b = k - d * nb;
    const double* e = L.edges + d * (nb + 1);
    double lo = e[b], hi = e[b + 1];
    sEdge[d][b] = make_float2((float)lo, (float)(hi - lo));
  }
  __syncthreads();

  const float nbf = (float)nb;
  const uint64_t stride = (uint64_t)gridDim.x * CP_THREADS;
  const uint64_t gtid = (uint64_t)blockIdx.x * CP_THREADS + threadIdx.x;
  const uint64_t rounds = (L.n + stride - 1) / stride;
  float s1 = 0.f, c1 = 0.f, s2 = 0.f, c2 = 0.f, wmax = 0.f;
  uint32_t nbad = 0;
  float* const myHist[3] = {&sHist[warp][0][0], &sHist[warp][1][0], &sHist[warp][2][0]};

  for (uint64_t r = 0; r < rounds; ++r) {
    const uint64_t p = r * stride + gtid;
    const bool active = p < L.n;
    float w = 0.f;
    int bin[3] = {0, 0, 0};
    if (active) {
      float x[3], jv = 1.f;
      uint32_t wd[4];
      cp_point_words(L.seed, L.point0 + p, L.iter, L.stream, wd);
      if (L.flow) {
        // the flow already applied the VEGAS map and its own transform: x and the total ln J
        const float4 f = L.flow[p];
        x[0] = f.x; x[1] = f.y; x[2] = f.z;
        jv = expf(f.w);
#pragma unroll
        for (int d = 0; d < 3; ++d) bin[d] = (int)(((wd[d] >> 8) * (uint32_t)nb) >> 24);
      } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          float frac;
          cp_bin_frac(wd[d], nb, bin[d], frac);
          float2 e = sEdge[d][bin[d]];
          x[d] = fmaf(frac, e.y, e.x);
          jv *= nbf * e.y;
        }
      }
      w = cp_had_weight(P, P.cteq, x[0], x[1], x[2], nullptr) * jv;
      if (!(w >= 0.f) || isinf(w)) { ++nbad; w = 0.f; }
      cp_kahan(s1, c1, w);
      cp_kahan(s2, c2, w * w);
      wmax = fmaxf(wmax, w);
      if (L.qhist) {
        int qb = cp_qbin(w);
        if (qb >= 0) atomicAdd(&sQ[qb], 1u);
      }
      if (WRITE) {
        if (L.w_out) L.w_out[p] = w;
        if (L.x_out) { L.x_out[3 * p] = x[0]; L.x_out[3 * p + 1] = x[1]; L.x_out[3 * p + 2] = x[2]; }
      }
    }
    const float w2 = w * w;
    const float hv[3][1] = {{w2}, {w2}, {w2}};
    cp_warp_hist_add<3, 1>(myHist, 0, bin, hv);
  }

  // compensated warp trees: Kahan sum s with compensation -c is the pair (s, -c)
  float h1 = s1, l1 = -c1, h2 = s2, l2 = -c2;
  cp_warp_sum_comp(h1, l1);
  cp_warp_sum_comp(h2, l2);
  float wm = cp_warp_max(wmax);
  unsigned nb_w = __reduce_add_sync(0xffffffffu, nbad);
  if (lane == 0) {
    sRed[warp][0] = h1; sRed[warp][1] = l1; sRed[warp][2] = h2; sRed[warp][3] = l2;
    sRed[warp][4] = wm; sRed[warp][5] = __uint_as_float(nb_w);
  }
  __syncthreads();
  double* slot = L.slots + (size_t)blockIdx.x * (CP_SLOT_HEAD + 3 * nb);
  if (threadIdx.x == 0) {
    // block combine in warp order, FP32 compensated, then one FP64 store
    float bh1 = 0.f, bl1 = 0.f, bh2 = 0.f, bl2 = 0.f, bm = 0.f;
    unsigned bn = 0;
    for (int k = 0; k < CP_WARPS; ++k) {
      float s, e;
      cp_two_sum(bh1, sRed[k][0], s, e); bh1 = s; bl1 += sRed[k][1] + e;
      cp_two_sum(bh2, sRed[k][2], s, e); bh2 = s; bl2 += sRed[k][3] + e;
      bm = fmaxf(bm, sRed[k][4]);
      bn += __float_as_uint(sRed[k][5]);
    }
    slot[0] = (double)bh1 + (double)bl1;
    slot[1] = (double)bh2 + (double)bl2;
    slot[2] = (double)bm;
    slot[3] = (double)bn;
  }
  for (int k = threadIdx.x; k < 3 * nb; k += CP_THREADS) {
    int d = k / nb, b = k - d * nb;
    float s = 0.f;
    for (int q = 0; q < CP_WARPS; ++q) s += sHist[q][d][b];
    slot[CP_SLOT_HEAD + k] = (double)s;
  }
  if (L.qhist)
    for (int k = threadIdx.x; k < CP_QBINS; k += CP_THREADS)
      if (sQ[k]) atomicAdd(&L.qhist[k], (unsigned long long)sQ[k]);
}

// Smallest bin edge w such that at most (1 - q) n of the weights lie above it (q-quantile,
// rounded up to the bin's upper edge); stored as the unweighting threshold.  One block, four bins
// a thread: with S(b) the weights in bins >= b (integers, so exact in any order), the threshold
// bin is the largest b >= 1 with S(b) > (1 - q) n, or 0.  One thread walking the 4096 bins twice
// took 92 us, longer than a pass of a million points.
__global__ void __launch_bounds__(1024) k_quantile(const unsigned long long* __restrict__ qhist, double q, double* wmax,
                                                   double* host)
{
  static_assert(CP_QBINS == 4 * 1024, "four bins a thread");
  __shared__ unsigned long long sWarp[32];
  __shared__ int sBest;
  // thread t owns bins 4 (1023 - t) .. + 3, so an inclusive scan over threads is a sum from the top
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, b0 = 4 * (1023 - t);
  unsigned long long c[4], x = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) x += c[j] = qhist[b0 + j];
  if (t == 0) sBest = 0;
  const unsigned long long own = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sWarp[w] = x;
  __syncthreads();
  unsigned long long tot = 0, before = 0;
  for (int k = 0; k < 32; ++k) {
    const unsigned long long y = sWarp[k];
    if (k < w) before += y;
    tot += y;
  }
  const double allowed = (1.0 - q) * (double)tot;
  unsigned long long above = before + x - own;   // weights in bins above this thread's
  int best = 0;
#pragma unroll
  for (int j = 3; j >= 0; --j) {
    above += c[j];
    if (!best && (double)above > allowed) best = b0 + j;
  }
  best = __reduce_max_sync(0xffffffffu, best);
  if (lane == 0 && best) atomicMax(&sBest, best);
  __syncthreads();
  if (t == 0) {
    host[0] = wmax[0] = (double)cp_qbin_hi(sBest);
    host[1] = wmax[1] = q;
  }
}

// Shared-memory working set of one dimension's refinement: the histogram, the old edges, the
// smoothed histogram, the bins' shares and their running sum, and the two warps' parts of a sum.
struct CpRefineDim {
  double h[CP_MAX_BINS], e[CP_MAX_BINS + 1], r[CP_MAX_BINS], cum[CP_MAX_BINS + 1], part[2];
};

// the two warps of a dimension
#define CP_REFINE_WARPS 2
__device__ __forceinline__ void cp_refine_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// Lepage's refinement of one dimension (FP64) by two warps (so 50 bins are one round), from S.h and S.e:
// smooth (1,1)/(1,1,1)/(1,1), normalise, compress r = ((d - 1) / ln d)^alpha, and rebin to equal shares of
// sum r.  The new edge k lies in the first bin j with cum[j + 1] >= k rsum / nb, cum the
// running sum of r: a binary search.  The sum is formed by a tree, so over bins without a share it may fall by its
// rounding; what two edges look for lies further apart than that, so they keep their order, and an edge that
// falls on such a flat stretch may take either end of it, as with any other rounding of the sum.  It is all latency:
// the two sums over the bins are warp trees (serial on one thread: 2,200 of 6,500 cycles for 50 bins, now 700), and
// the usual alpha of 3/2 is a product and a square root instead of a power.
__device__ __forceinline__ void cp_refine_dim(CpRefineDim& S, double* __restrict__ edges, int nb, double alpha, int bar)
{
  const int t = threadIdx.x % (32 * CP_REFINE_WARPS), n = 32 * CP_REFINE_WARPS, lane = t & 31, w = t >> 5;
  double a = 0.0;
  for (int i = t; i < nb; i += n) {
    double s;
    if (i == 0) s = (S.h[0] + S.h[1]) / 2.0;
    else if (i == nb - 1) s = (S.h[nb - 2] + S.h[nb - 1]) / 2.0;
    else s = (S.h[i - 1] + S.h[i] + S.h[i + 1]) / 3.0;
    S.r[i] = s;
    a += s;
  }
  a = cp_warp_sum_d(a);
  if (lane == 0) S.part[w] = a;
  cp_refine_sync(bar);
  const double tot = S.part[0] + S.part[1];
  if (!(tot > 0.0)) return;
  double carry = 0.0;
  if (t == 0) S.cum[0] = 0.0;
  for (int i0 = 0; i0 < nb; i0 += n) {
    const int i = i0 + t;
    double ri = 0.0;
    if (i < nb) {
      const double di = S.r[i] / tot;
      if (di >= 1.0) {
        ri = 1.0;
      } else if (di > 0.0) {
        const double x = (di - 1.0) / log(di);
        ri = alpha == 1.5 ? x * sqrt(x) : pow(x, alpha);
      }
      S.r[i] = ri;
    }
    double c = ri;   // inclusive sum over the warp's bins
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, c, o);
      if (lane >= o) c += y;
    }
    cp_refine_sync(bar);   // the parts read before
    if (lane == 31) S.part[w] = c;
    cp_refine_sync(bar);
    if (w) c += S.part[0];
    if (i < nb) S.cum[i + 1] = carry + c;
    carry += S.part[0] + S.part[1];
  }
  cp_refine_sync(bar);
  const double step = S.cum[nb] / (double)nb;
  for (int k = 1 + t; k < nb; k += n) {
    const double need = step * (double)k;
    int j = 0, hi = nb - 1;
    while (j < hi) {
      const int m = (j + hi) >> 1;
      if (S.cum[m + 1] < need) j = m + 1;
      else hi = m;
    }
    double frac = S.r[j] > 0.0 ? (need - S.cum[j]) / S.r[j] : 0.0;
    frac = frac < 0.0 ? 0.0 : (frac > 1.0 ? 1.0 : frac);
    edges[k] = S.e[j] + frac * (S.e[j + 1] - S.e[j]);
  }
}

// Iteration record (one thread) and, if alpha > 0, the grid refinement (two warps a dimension, from
// S[d].h and S[d].e) of a pass with the sums head; blocks of at least 256 threads.
__device__ __forceinline__ void cp_pass_record_refine(CpRefineDim (&S)[3], const double* head, double* edges, int nb,
                                                      double n, double alpha, CpIterDev* rec)
{
  const int d = threadIdx.x / (32 * CP_REFINE_WARPS);
  if (threadIdx.x == 255 && rec) {
    const double sumw = head[0], sumw2 = head[1];
    const double mean = sumw / n;
    const double var = (sumw2 / n - mean * mean) / (n - 1.0);
    rec->sumw = sumw; rec->sumw2 = sumw2; rec->wmax = head[2]; rec->nbad = head[3]; rec->n = n;
    rec->sigma = mean; rec->err = sqrt(var > 0.0 ? var : 0.0);
  }
  if (alpha > 0.0 && d < 3) cp_refine_dim(S[d], edges + d * (nb + 1), nb, alpha, 1 + d);
}

__device__ __forceinline__ void cp_refine_load_edges(CpRefineDim (&S)[3], const double* __restrict__ edges, int nb)
{
  for (int k = threadIdx.x; k < 3 * (nb + 1); k += blockDim.x) S[k / (nb + 1)].e[k % (nb + 1)] = edges[k];
}

// The record and refinement from sums already reduced (over ranks).
__global__ void __launch_bounds__(256) k_refine(double* edges, const double* red, int nb, double n, double alpha,
                                                CpIterDev* rec)
{
  __shared__ CpRefineDim S[3];
  cp_refine_load_edges(S, edges, nb);
  for (int k = threadIdx.x; k < 3 * nb; k += blockDim.x) S[k / nb].h[k % nb] = red[CP_SLOT_HEAD + k];
  __syncthreads();
  cp_pass_record_refine(S, red, edges, nb, n, alpha, rec);
}

// The end of an iteration in one launch, by one cluster: the fixed-order reduction of the block slots, the
// sums of k_reduce_slots bit for bit, with the partial sums stored to the first block's shared memory, then
// there the iteration record and the refinement; on the way the weight histogram is cleared, if qclear is given.  Four warps take four columns: lane 4 o + c
// of warp w adds column c of the slots b = w + 4 o (mod 32), so a load of the warp covers whole sectors
// and 296 slots are two batches of loads.  It is latency from end to end, and a pass of a few thousand points waits
// for it longer than for its own kernel.  With a grid of 20 blocks, a ticket for the last of them, the sums read
// back through L2 and serial sums in the refinement, five iterations of 4,099 points took 137 us, then 128, and ten
// of a million 818, then 803.  The block is as small as that because the pass kernels on either side leave room for
// it, and it for them, so that chained launches take their places early (640 threads: 125 and 816 us).
#define CP_FINISH_BLOCKS 8
#define CP_FINISH_THREADS 320
#define CP_FINISH_LOADS 5
__global__ void __cluster_dims__(CP_FINISH_BLOCKS, 1, 1) __launch_bounds__(CP_FINISH_THREADS, 4)
    k_pass_finish(const double* __restrict__ slots, int nblocks, int width, double* red, double* edges, int nb, double n,
                  double alpha, CpIterDev* rec, unsigned long long* qclear)
{
  __shared__ CpRefineDim S[3];
  __shared__ double sPart[4][CP_SLOT_HEAD + 3 * CP_MAX_BINS], sHead[CP_SLOT_HEAD];
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = (int)cluster.block_rank(), lane = threadIdx.x & 31;
  cluster.barrier_arrive();
  cp_next_may_launch();
  cp_wait_previous();
  if (rank == 0) cp_refine_load_edges(S, edges, nb);
  double* const part0 = cluster.map_shared_rank(&sPart[0][0], 0);
  // the blocks of a cluster are placed together but need not have started together, and a block's shared memory
  // may be written only once it runs: a pass of one slot leaves most blocks nothing to load before they store
  cluster.barrier_wait();
  const int groups = (width + 3) / 4;
  for (int v = rank + CP_FINISH_BLOCKS * (threadIdx.x >> 5); v < 4 * groups; v += CP_FINISH_BLOCKS * (CP_FINISH_THREADS / 32)) {
    const int w = v & 3, k = 4 * (v >> 2) + (lane & 3);
    double acc = 0.0;
    if (k < width) {
      const double* col = slots + k;
      for (int b0 = w + 4 * (lane >> 2); b0 < nblocks; b0 += 32 * CP_FINISH_LOADS) {
        double x[CP_FINISH_LOADS];   // in flight at once, added in slot order (a slot past the last adds nothing)
#pragma unroll
        for (int i = 0; i < CP_FINISH_LOADS; ++i) x[i] = b0 + 32 * i < nblocks ? col[(size_t)(b0 + 32 * i) * width] : 0.0;
#pragma unroll
        for (int i = 0; i < CP_FINISH_LOADS; ++i) acc = k == 2 ? fmax(acc, x[i]) : acc + x[i];
      }
    }
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) {
      const double y = __shfl_xor_sync(0xffffffffu, acc, o);
      acc = k == 2 ? fmax(acc, y) : acc + y;
    }
    if (lane < 4 && k < width) part0[w * (CP_SLOT_HEAD + 3 * CP_MAX_BINS) + k] = acc;
  }
  if (qclear)
    for (int k = rank * CP_FINISH_THREADS + threadIdx.x; k < CP_QBINS; k += CP_FINISH_BLOCKS * CP_FINISH_THREADS) qclear[k] = 0ull;
  cluster.sync();
  if (rank != 0) return;
  for (int k = threadIdx.x; k < width; k += CP_FINISH_THREADS) {
    const double v = k == 2 ? fmax(fmax(sPart[0][k], sPart[2][k]), fmax(sPart[1][k], sPart[3][k]))
                            : (sPart[0][k] + sPart[2][k]) + (sPart[1][k] + sPart[3][k]);
    red[k] = v;
    const int q = k - CP_SLOT_HEAD;
    if (q < 0) sHead[k] = v;
    else S[q / nb].h[q % nb] = v;
  }
  __syncthreads();
  cp_pass_record_refine(S, sHead, edges, nb, n, alpha, rec);
}

// FP32 integrand at caller-supplied x
__global__ void __launch_bounds__(CP_THREADS, CP_MIN_BLOCKS) k_weight_at(const CpHadParams P, const CpCteqPoly* cteq_g, const float* __restrict__ x,
                            int64_t n, float* w)
{
  __shared__ CpCteqPoly sCteq[8];
  cp_stage_cteq(sCteq, cteq_g);
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    w[i] = cp_had_weight(P, sCteq, x[3 * i], x[3 * i + 1], x[3 * i + 2], nullptr);
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
// Blocks of a pass over n points: the resident blocks, fewer when the points do not fill them (a
// block without points would write and have reduced a slot of zeros).
static int had_blocks_for(const cp_handle* h, uint64_t n)
{
  const uint64_t want = (n + CP_THREADS - 1) / CP_THREADS;
  return want < (uint64_t)h->had_blocks ? (want > 0 ? (int)want : 1) : h->had_blocks;
}

// The pass kernel alone.  The weight histogram: added to (CP_HIST_ADD), cleared before (CP_HIST_NEW), or left alone.
enum { CP_HIST_NONE, CP_HIST_ADD, CP_HIST_NEW };
static int had_pass(cp_handle* h, uint64_t point0, uint64_t n, uint32_t iter, uint32_t stream,
                    float* w_out, float* x_out, int hist)
{
  const int blocks = had_blocks_for(h, n);
  int rc = cp_ensure_slots(h, (size_t)blocks * (CP_SLOT_HEAD + 3 * h->nb));
  if (rc) return rc;
  point0 += h->point_offset;
  HadLaunch L;
  L.seed = h->cfg.seed; L.point0 = point0; L.n = n; L.iter = iter; L.stream = stream;
  L.nb = h->nb; L.edges = h->d_edges; L.slots = h->d_slots; L.w_out = w_out; L.x_out = x_out;
  L.qhist = hist == CP_HIST_NONE ? nullptr : h->d_qhist;
  L.flow = nullptr;
  if (h->flow_on) {
    rc = cp_flow_buffer(h, n);
    if (rc) return rc;
    rc = cp_flow_forward_enqueue(h, point0, n, iter, stream, h->d_flow_buf, nullptr);
    if (rc) return rc;
    L.flow = h->d_flow_buf;
  }
  if (hist == CP_HIST_NEW) CP_CUDA(h, cudaMemsetAsync(h->d_qhist, 0, sizeof(unsigned long long) * CP_QBINS, h->stream));
  h->last_n = n;
  if (w_out || x_out) CP_CUDA(h, cp_launch_chained(k_had_accum<true>, blocks, CP_THREADS, h->stream, h->P, L));
  else CP_CUDA(h, cp_launch_chained(k_had_accum<false>, blocks, CP_THREADS, h->stream, h->P, L));
  return CP_OK;
}

// A pass and the reduction of its sums into d_red.
static int had_launch(cp_handle* h, uint64_t point0, uint64_t n, uint32_t iter, uint32_t stream,
                      float* w_out, float* x_out)
{
  int rc = had_pass(h, point0, n, iter, stream, w_out, x_out, CP_HIST_NEW);
  if (rc) return rc;
  const int wpb = 8, width = CP_SLOT_HEAD + 3 * h->nb;
  k_reduce_slots<0><<<(width + wpb - 1) / wpb, wpb * 32, 0, h->stream>>>(h->d_slots, had_blocks_for(h, n), width, h->d_red);
  CP_LAUNCH_CHECK(h, "k_reduce_slots");
  return CP_OK;
}

// An iteration: pass, reduction, record and refinement; clear: the weight histogram is cleared at its end.
static int had_iteration(cp_handle* h, uint64_t n, uint32_t iter, double alpha, CpIterDev* rec, int hist, int clear)
{
  int rc = had_pass(h, 0, n, iter, 0, nullptr, nullptr, hist);
  if (rc) return rc;
  CP_CUDA(h, cp_launch_chained(k_pass_finish, CP_FINISH_BLOCKS, CP_FINISH_THREADS, h->stream, h->d_slots, had_blocks_for(h, n),
                               CP_SLOT_HEAD + 3 * h->nb, h->d_red, h->d_edges, h->nb, (double)n, alpha, rec,
                               clear ? h->d_qhist : nullptr));
  return CP_OK;
}

static void fill_result(const CpIterDev& r, cp_result* out)
{
  out->sigma = r.sigma;
  out->sigma_err = r.err;
  out->sum_w = r.sumw;
  out->sum_w2 = r.sumw2;
  out->w_max = r.wmax;
  out->n_points = (uint64_t)r.n;
  out->n_bad = (uint64_t)r.nbad;
  out->eta = r.wmax > 0 ? r.sigma / r.wmax : 0.0;
}

int cp_had_launch_shape(cp_handle* h)
{
  int per_sm = 0;
  CP_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_had_accum<false>, CP_THREADS, 0));
  if (per_sm < 1) per_sm = 1;
  h->had_blocks = h->num_sms * per_sm;
  return CP_OK;
}

extern "C" int cp_vegas_iteration(cp_handle* h, uint64_t n_points, uint32_t iter, double alpha,
                                  cp_result* out)
{
  CP_CHECK_HANDLE(h);
  if (n_points < 2) return cp_fail(h, CP_ERR_INVALID, "cp_vegas_iteration: n_points < 2");
  int rc = cp_ensure_iters(h, 1);
  if (rc) return rc;
  rc = had_iteration(h, n_points, iter, alpha, h->h_iters, CP_HIST_NEW, 0);
  if (rc) return rc;
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  const CpIterDev& r = h->h_iters[0];
  if (h->flow_on && (rc = cp_flow_tc_status(h)) != CP_OK) return rc;
  if (out) fill_result(r, out);
  if (r.nbad > 0) return cp_fail(h, CP_ERR_NUMERIC, "non-finite or negative weights were zeroed");
  return CP_OK;
}

extern "C" int cp_integrate(cp_handle* h, int n_iter, uint64_t n_points, double alpha, int skip,
                            cp_result* per_iter, cp_result* combined)
{
  CP_CHECK_HANDLE(h);
  if (n_iter < 1 || n_points < 2) return cp_fail(h, CP_ERR_INVALID, "cp_integrate: bad sizes");
  int rc = cp_ensure_iters(h, n_iter);
  if (rc) return rc;
  // The weight histogram is the last pass's, so the others fill none (10 x 10^6 points: 803 -> 785 us); the first one's end
  // clears it.
  for (int it = 0; it < n_iter; ++it) {
    const int hist = it + 1 < n_iter ? CP_HIST_NONE : n_iter == 1 ? CP_HIST_NEW : CP_HIST_ADD;
    rc = had_iteration(h, n_points, (uint32_t)it, alpha, h->h_iters + it, hist, it == 0 && n_iter > 1);
    if (rc) return rc;
  }
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  const CpIterDev* recs = h->h_iters;
  if (h->flow_on && (rc = cp_flow_tc_status(h)) != CP_OK) return rc;
  double wsum = 0, w2 = 0, sw = 0, sw2 = 0, wmax = 0, nbad = 0, npts = 0;
  for (int it = 0; it < n_iter; ++it) {
    if (per_iter) fill_result(recs[it], per_iter + it);
    nbad += recs[it].nbad;
    if (it < skip) continue;
    double err = recs[it].err;
    if (err > 0) { wsum += recs[it].sigma / (err * err); w2 += 1.0 / (err * err); }
    sw += recs[it].sumw; sw2 += recs[it].sumw2; npts += recs[it].n;
    wmax = recs[it].wmax > wmax ? recs[it].wmax : wmax;
  }
  if (combined) {
    combined->sigma = w2 > 0 ? wsum / w2 : 0;
    combined->sigma_err = w2 > 0 ? 1.0 / sqrt(w2) : 0;
    combined->sum_w = sw; combined->sum_w2 = sw2; combined->w_max = wmax;
    combined->n_points = (uint64_t)npts; combined->n_bad = (uint64_t)nbad;
    combined->eta = wmax > 0 ? combined->sigma / wmax : 0;
  }
  if (nbad > 0) return cp_fail(h, CP_ERR_NUMERIC, "non-finite or negative weights were zeroed");
  return CP_OK;
}

extern "C" int cp_point_weights(cp_handle* h, uint64_t point0, uint64_t n, uint32_t iter,
                                float* w_dev, float* x_dev)
{
  CP_CHECK_HANDLE(h);
  if (!w_dev && !x_dev) return cp_fail(h, CP_ERR_INVALID, "cp_point_weights: no output");
  if (n == 0) return CP_OK;
  int rc = had_launch(h, point0, n, iter, 0, w_dev, x_dev);
  if (rc) return rc;
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_weight_at(cp_handle* h, const float* x, int64_t n, float* w)
{
  CP_CHECK_HANDLE(h);
  if (n < 0 || (n > 0 && (!x || !w))) return cp_fail(h, CP_ERR_INVALID, "cp_weight_at: bad args");
  if (n == 0) return CP_OK;
  int blocks = (int)((n + CP_THREADS - 1) / CP_THREADS);
  if (blocks > h->num_sms * 16) blocks = h->num_sms * 16;
  k_weight_at<<<blocks, CP_THREADS, 0, h->stream>>>(h->P, h->d_cteq, x, n, w);
  CP_LAUNCH_CHECK(h, "k_weight_at");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_last_histogram(cp_handle* h, double* out)
{
  CP_CHECK_HANDLE(h);
  if (!out) return cp_fail(h, CP_ERR_INVALID, "cp_last_histogram: null output");
  CP_CUDA(h, cudaMemcpyAsync(out, h->d_red, sizeof(double) * (CP_SLOT_HEAD + 3 * h->nb),
                             cudaMemcpyDeviceToHost, h->stream));
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_weight_quantile(cp_handle* h, double q, double* w_q)
{
  CP_CHECK_HANDLE(h);
  if (!(q > 0.0 && q < 1.0)) return cp_fail(h, CP_ERR_INVALID, "cp_weight_quantile: q must be in (0, 1)");
  if (h->last_n == 0) return cp_fail(h, CP_ERR_INVALID, "cp_weight_quantile: run an iteration first");
  k_quantile<<<1, 1024, 0, h->stream>>>(h->d_qhist, q, h->d_wmax, h->mail->wq);
  CP_LAUNCH_CHECK(h, "k_quantile");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  const double* v = h->mail->wq;
  h->wmax_host = v[0];   // production passes check the threshold without reading the device
  if (w_q) *w_q = v[0];
  return CP_OK;
}

// ------------------------------------------------------------------------------------------
// Distributed iteration: a pass over this handle's points into a caller buffer, and the
// refinement from sums the caller has reduced over ranks (sum over every entry except the
// maximum weight at index 2, which is reduced by max).
// ------------------------------------------------------------------------------------------
extern "C" int cp_vegas_accumulate(cp_handle* h, uint64_t n_points, uint32_t iter, double* sums_dev)
{
  CP_CHECK_HANDLE(h);
  if (n_points < 1 || !sums_dev) return cp_fail(h, CP_ERR_INVALID, "cp_vegas_accumulate: bad arguments");
  int rc = had_launch(h, 0, n_points, iter, 0, nullptr, nullptr);
  if (rc) return rc;
  CP_CUDA(h, cudaMemcpyAsync(sums_dev, h->d_red, sizeof(double) * (CP_SLOT_HEAD + 3 * h->nb), cudaMemcpyDeviceToDevice,
                             h->stream));
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  if (h->flow_on && (rc = cp_flow_tc_status(h)) != CP_OK) return rc;
  return CP_OK;
}

extern "C" int cp_vegas_refine_sums(cp_handle* h, const double* sums_dev, double n_total, double alpha, cp_result* out)
{
  CP_CHECK_HANDLE(h);
  if (!sums_dev || !(n_total >= 2)) return cp_fail(h, CP_ERR_INVALID, "cp_vegas_refine_sums: bad arguments");
  int rc = cp_ensure_iters(h, 1);
  if (rc) return rc;
  CP_CUDA(h, cudaMemcpyAsync(h->d_red, sums_dev, sizeof(double) * (CP_SLOT_HEAD + 3 * h->nb), cudaMemcpyDeviceToDevice,
                             h->stream));
  k_refine<<<1, 256, 0, h->stream>>>(h->d_edges, h->d_red, h->nb, n_total, alpha, h->h_iters);
  CP_LAUNCH_CHECK(h, "k_refine");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  const CpIterDev& r = h->h_iters[0];
  if (out) fill_result(r, out);
  if (r.nbad > 0) return cp_fail(h, CP_ERR_NUMERIC, "non-finite or negative weights were zeroed");
  return CP_OK;
}

extern "C" int cp_weight_histogram(cp_handle* h, unsigned long long* hist_dev)
{
  CP_CHECK_HANDLE(h);
  if (!hist_dev) return cp_fail(h, CP_ERR_INVALID, "cp_weight_histogram: null buffer");
  if (h->last_n == 0) return cp_fail(h, CP_ERR_INVALID, "cp_weight_histogram: run a pass first");
  CP_CUDA(h, cudaMemcpyAsync(hist_dev, h->d_qhist, sizeof(unsigned long long) * CP_QBINS, cudaMemcpyDeviceToDevice,
                             h->stream));
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  return CP_OK;
}

extern "C" int cp_weight_quantile_hist(cp_handle* h, const unsigned long long* hist_dev, double q, double* w_q)
{
  CP_CHECK_HANDLE(h);
  if (!hist_dev || !(q > 0.0 && q < 1.0)) return cp_fail(h, CP_ERR_INVALID, "cp_weight_quantile_hist: bad arguments");
  k_quantile<<<1, 1024, 0, h->stream>>>(hist_dev, q, h->d_wmax, h->mail->wq);
  CP_LAUNCH_CHECK(h, "k_quantile");
  CP_CUDA(h, cudaStreamSynchronize(h->stream));
  const double* v = h->mail->wq;
  h->wmax_host = v[0];
  if (w_q) *w_q = v[0];
  return CP_OK;
}

// ------------------------------------------------------------------------------------------
// Allocation-free VEGAS pass.
//
// For callers that must not allocate device memory: a host program that owns every device
// allocation (a caching allocator or memory pool whose accounting a cudaMalloc behind its back
// would break), a process held to a fixed device-memory budget, or a plugin such as a Pythia
// SigmaProcess running inside someone else's event loop, which cannot create and keep a handle
// with its own buffers.  This entry point creates no handle and calls no cudaMalloc / cudaFree:
// its scratch (the per-block partial sums and the weight histogram; the CTEQ5L coefficient
// records travel in the kernel's parameters) lives in the file-scope array below, which every GPU that loads this library keeps
// until the process exits.  The first call on a device looks up the array's address and the
// launch shape (later calls only re-check the address); make that first call before any stream
// capture.
//
// Limits: the partial sums hold at most CP_NOALLOC_MAX_BLOCKS blocks of CP_SLOT_HEAD + 3 *
// CP_MAX_BINS doubles, so n_bins above CP_MAX_BINS is rejected; the grid is capped at
// CP_NOALLOC_MAX_BLOCKS blocks (296 are used on a B200).  Total: 1,622,016 bytes per device.
// Every call shares the array and it keeps the last call's contents; each call clears the
// weight histogram and rewrites every partial-sum slot it reads.  Calls that overlap on the GPU (different streams, or several host threads) race on the
// array and must not be issued; calls in one stream are ordered and safe.
// ------------------------------------------------------------------------------------------
#define CP_NOALLOC_MAX_BLOCKS 512
#define CP_NOALLOC_SLOT_DOUBLES (CP_NOALLOC_MAX_BLOCKS * (CP_SLOT_HEAD + 3 * CP_MAX_BINS))
#define CP_NOALLOC_DOUBLES (CP_QBINS + CP_NOALLOC_SLOT_DOUBLES)

static __device__ __align__(256) double cp_noalloc_scratch[CP_NOALLOC_DOUBLES];

// Per-call set-up of the shared array, on the caller's stream: a cleared weight histogram.
__global__ void k_noalloc_setup(double* base)
{
  unsigned long long* qhist = reinterpret_cast<unsigned long long*>(base);
  for (int k = threadIdx.x; k < CP_QBINS; k += blockDim.x) qhist[k] = 0ull;
}

namespace {
struct NoallocDevice {
  double* scratch = nullptr;   // device address of cp_noalloc_scratch on this device
  int blocks = 0;
};
const int CP_NOALLOC_MAX_DEVICES = 64;
NoallocDevice g_noalloc[CP_NOALLOC_MAX_DEVICES];
std::mutex g_noalloc_mutex;
}  // namespace

extern "C" int cp_vegas_pass_noalloc(const cp_config* cfg, uint64_t n_points, uint32_t iter,
                                     const double* edges_dev, double* sums_dev, void* cuda_stream)
{
  if (!cfg || !edges_dev || !sums_dev) return CP_ERR_INVALID;
  if (cfg->n_bins < 2 || cfg->n_bins > CP_MAX_BINS) return CP_ERR_INVALID;   // beyond the scratch
  if (n_points < 2) return CP_ERR_INVALID;
  if (cfg->device < 0 || cfg->device >= CP_NOALLOC_MAX_DEVICES) return CP_ERR_INVALID;
  CpHadConfig hc{cfg->sqrt_s, cfg->pt_hat_min, cfg->alphas_mz, cfg->k_ren, cfg->k_fac,
                 cfg->convert2mb, cfg->n_quark_in, cfg->n_quark_new, cfg->proc_mask};
  CpHadParams P;
  if (cp_build_had_params(hc, P) || (cfg->proc_mask & ~CP_PROC_ALL) || cfg->proc_mask == 0)
    return CP_ERR_INVALID;
  int prev = -1;
  if (cudaGetDevice(&prev) != cudaSuccess) return CP_ERR_CUDA;
  if (prev != cfg->device && cudaSetDevice(cfg->device) != cudaSuccess) return CP_ERR_CUDA;
  cudaStream_t stream = (cudaStream_t)cuda_stream;
  int rc = CP_OK;
  NoallocDevice D;
  {
    // With the device current: the array's device address (looked up on every call, so a
    // reloaded module after a device reset is picked up) and, when it is new, the launch shape.
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    NoallocDevice& G = g_noalloc[cfg->device];
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, cp_noalloc_scratch) != cudaSuccess || !ptr) {
      rc = CP_ERR_CUDA;
    } else if (ptr != G.scratch) {
      int nsm = 0, per_sm = 0;
      if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, cfg->device) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_had_accum<false>, CP_THREADS, 0) != cudaSuccess) {
        rc = CP_ERR_CUDA;
      } else {
        const int blocks = nsm * (per_sm > 0 ? per_sm : 1);
        G.blocks = blocks < CP_NOALLOC_MAX_BLOCKS ? blocks : CP_NOALLOC_MAX_BLOCKS;
        G.scratch = (double*)ptr;
      }
    }
    D = G;
  }
  if (rc == CP_OK) {
    double* base = D.scratch;
    unsigned long long* qhist = reinterpret_cast<unsigned long long*>(base);
    double* slots = base + CP_QBINS;
    int nb = cfg->n_bins, width = CP_SLOT_HEAD + 3 * nb, max_col = 2;
    HadLaunch L;
    L.seed = cfg->seed; L.point0 = 0; L.n = n_points; L.iter = iter; L.stream = 0;
    L.nb = nb; L.edges = edges_dev;
    L.slots = slots; L.w_out = nullptr; L.x_out = nullptr; L.qhist = qhist; L.flow = nullptr;
    // Each launch's own return code is checked; an error the caller left pending from earlier,
    // unrelated work is neither reported as this call's nor cleared.
    void* a_setup[] = {&base};
    void* a_accum[] = {&P, &L};
    void* a_reduce[] = {&slots, &D.blocks, &width, &sums_dev, &max_col};
    if (cudaLaunchKernel((const void*)k_noalloc_setup, dim3(1), dim3(256), a_setup, 0, stream) != cudaSuccess ||
        cudaLaunchKernel((const void*)k_had_accum<false>, dim3(D.blocks), dim3(CP_THREADS), a_accum, 0, stream) !=
            cudaSuccess ||
        cudaLaunchKernel((const void*)k_reduce_slots<0>, dim3((width + 7) / 8), dim3(8 * 32), a_reduce, 0, stream) !=
            cudaSuccess)
      rc = CP_ERR_CUDA;
  }
  if (prev != cfg->device) cudaSetDevice(prev);
  return rc;
}
