// Exact angular top-k with the tensor cores as a filter (implementation 2; the reference's
// plain exact scan, memOptimizedLinearScan.cu:20-106): ids and distances are those of the FP32
// scan of scan_float.cu, bit for bit.
//
// Each point's cosine is first scored in BF16 (tc_filter.cu); only points whose score can
// belong to the top-k are scored with the reference's single-precision formula.  What makes
// that exact is a bound eps on |1 - s - D|, s the BF16 score and D the FP32 distance of a
// (query, point) pair.  With u = x / |x| and r(x) = |u - bf16 row of x|:
//   the rows' rounding    |s' - cos| <= r(x) (1 + r(q)) + r(q), s' the rows' exact product;
//   the rows themselves   r(x) is taken from the rows as built, whose FP32 normalisation is
//                         within 2^-18 of u;
//   the accumulation      of at most 128 products of magnitude <= 1 (in total, by
//                         Cauchy-Schwarz) in the tensor core: 2^-15 allowed, 64 times what
//                         eight FP32 additions with truncation lose (an allowance: how the
//                         tensor core adds is not documented);
//   the FP32 distance     within (2 d + 7) 2^-24 of 1 - cos (fp64_band in rerank.cu) while
//                         both norms are in [2^-40, 2^40], so that nothing over- or underflows.
// Let s_k be the k-th best score.  The k points that reach it have D <= 1 - s_k + eps, so every
// point of the exact top-k (by (D, id)) has D at most that and s >= s_k - 2 eps.  The filter's
// threshold is lowered by 2 eps, and a query whose survivors do not provably include that
// range -- a threshold above it, more survivors than fit, a norm out of range -- is scanned by
// the FP32 scan, from a list on the device.  A base with a row whose norm is out of range
// always takes the FP32 scan.
//
// r(x) is about 8e-4 for vectors of 100 comparable components, so 2 eps is about 0.004 and the
// candidates are a handful more than k.  Measured (100k x 100, 1,000 queries, k = 32): the
// FP32 scan 886 us, this 78; 1M x 100, one query 915 -> 100 us; 1.2M, 1,000 queries 6.62 -> 0.28
// ms.
#include <algorithm>

#include "index.h"
#include "launch_count.h"
#include "launch_next.cuh"
#include "profile.h"
#include "tc_filter.h"
#include "tc_ptx.cuh"

namespace lshg {

namespace {

constexpr float kNormMin = 9.094947e-13f, kNormMax = 1.0995116e12f;  // 2^-40, 2^40
// slack of eps besides the rows' residuals: 2^-15 + 2 * 2^-18 + (2 * 128 + 7) 2^-24 < 6e-5
constexpr float kScoreSlack = 8e-5f;

// Unit rows in BF16, zero-padded to 128 columns and rows_pad rows, as the tensor-core scan's
// (to_unit_bf16), with each row's residual |x / |x| - row|.  Base (stat): the largest residual
// (as ordered bits) and whether a row is out of range.  Queries (eps): the bound eps of the
// row against a base of largest residual *base_res, infinite for a row out of range.
__global__ void unit_rows_kernel(const float* __restrict__ x, int64_t n, int d, int64_t rows_pad,
                                 __nv_bfloat16* __restrict__ out, unsigned* stat, const float* base_res,
                                 float* __restrict__ eps, int* counters, int ncounters) {
  grid_ready();
  zero_counters(counters, ncounters);
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  float worst = 0.0f;
  bool bad = false;
  for (int64_t i = warp; i < rows_pad; i += nw) {
    float v[4];
    float ss = 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = c * 32 + lane;
      v[c] = (i < n && j < d) ? x[i * d + j] : 0.0f;
      ss = fmaf(v[c], v[c], ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const bool ok = ss >= kNormMin * kNormMin && ss <= kNormMax * kNormMax;  // false for NaN
    const float inv = ok ? rsqrtf(ss) : 0.0f;
    float rr = 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float u = ok ? v[c] * inv : 0.0f;
      const __nv_bfloat16 h = __float2bfloat16_rn(u);
      const float df = u - __bfloat162float(h);
      rr = fmaf(df, df, rr);
      out[i * tc::KD + c * 32 + lane] = h;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rr += __shfl_xor_sync(0xffffffffu, rr, o);
    if (i >= n) continue;
    const float r = sqrtf(rr) * 1.001f;  // above the rounding of the sum and the root
    worst = fmaxf(worst, r);
    bad |= !ok;
    if (eps && lane == 0) {
      const float R = *base_res;
      eps[i] = ok ? R + r + R * r + kScoreSlack : INFINITY;
    }
  }
  if (stat && lane == 0) {
    if (worst > 0.0f) atomicMax(stat, __float_as_uint(worst));  // nonnegative floats order as their bits
    if (bad) atomicExch(stat + 1, 1u);
  }
}

void launch_unit_rows(const float* x, int64_t n, int d, int64_t rows_pad, uint16_t* out, unsigned* stat,
                      const float* base_res, float* eps, int* counters, int ncounters, cudaStream_t s) {
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((rows_pad * 32 + 255) / 256, (int64_t)num_sms() * 8));
  launch_next(unit_rows_kernel, blocks, 256, 0, s, x, n, d, rows_pad, reinterpret_cast<__nv_bfloat16*>(out), stat,
              base_res, eps, counters, ncounters);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

// Bases below kExactFilterMinBase points and batches below kExactFilterMinPairs (query, point)
// pairs stay with the FP32 scan: the filter's eight launches take 39 to 52 us whatever the sizes.
// FP32 scan and filter, us, k = 10: one query on 20,000 x 100 53 / 41, two on 8,192 53 / 40, four
// on 4,096 67 / 40; below the line one on 8,192 and on 4,096 46.  At 16 dimensions the FP32 scan is
// shorter for one query up to 60,000 points (20,000: 30 / 40) and longer from four on (4,096: 48 / 39).
constexpr int64_t kExactFilterMinBase = 4096;
constexpr int64_t kExactFilterMinPairs = 16384;
// The base from which a query re-scores 256 candidates at most instead of 128 (k <= 32): queries with
// more go to the FP32 scan, and a large base has more points within 2 eps of the k-th.  1.2M x 32,
// 1,000 queries, k = 10: with 128 places 595 us, with 256 261; 100k x 100, k = 32: 81 and
// 90.
constexpr int64_t kExactFewCandidatesBase = 1 << 18;
// The largest base that is filtered at few dimensions: on a sphere of d - 1 dimensions the points
// within 2 eps of the k-th fill a fixed share of it, more than the places hold beyond about these
// sizes, and the batch is then scanned twice.  Uniform points, filtered / FP32, us: d = 3, 20,000
// points, 16 queries 106 / 90, 1,000 154 / 242; 100,000 points 213 / 149; d = 4, 100,000 190 / 149
// and 303 / 638, 1M, one 329 / 214; d = 5, 1M, one 103 / 220, 1,000 656 / 2,922, 3M, one 703 /
// 588; d = 6, 3M, one 180 / 612.  Below d = 3 every size lost (d = 2, 100,000 points, 200 queries
// 339 / 259).
int64_t exact_filter_max_base(int d) {
  return d < 3 ? 0 : d == 3 ? 1 << 15 : d == 4 ? 1 << 17 : d == 5 ? 1 << 20 : INT_MAX;
}

}  // namespace

void derive_exact(Index& I, cudaStream_t s) {
  if (I.dist != DIST_ANGULAR || I.d > tc::KD || I.n < kExactFilterMinBase || I.n > exact_filter_max_base(I.d)) return;
  const int64_t npad = (int64_t)ceil_div(I.n, tc::FILTER_TN) * tc::FILTER_TN;
  unsigned bad = 0;
  try {
    I.ebf.alloc((size_t)npad * tc::KD, s);
    I.ebf_res.alloc(2, s);
  } catch (const Error& e) {  // no room for the filter's rows: the FP32 scan needs none
    if (e.status != LSHG_ERR_OUT_OF_MEMORY) throw;
    cudaGetLastError();
    I.ebf.release();
    return;
  }
  LSHG_CUDA(cudaMemsetAsync(I.ebf_res.ptr, 0, I.ebf_res.bytes(), s));
  unsigned* stat = reinterpret_cast<unsigned*>(I.ebf_res.ptr);
  launch_unit_rows(I.x.ptr, I.n, I.d, npad, I.ebf.ptr, stat, nullptr, nullptr, nullptr, 0, s);
  LSHG_CUDA(cudaMemcpyAsync(&bad, stat + 1, sizeof(bad), cudaMemcpyDeviceToHost, s));
  LSHG_CUDA(cudaStreamSynchronize(s));
  if (bad) {
    I.ebf.release();
    I.ebf_res.release();
  }
}

bool query_exact_filtered(Index& I, const float* q, int nq, int k, lshg_point* out, cudaStream_t s) {
  using namespace tc;
  if (!I.ebf.ptr || k > 128 || (int64_t)nq * I.n < kExactFilterMinPairs) return false;
  const int CT = k <= 32 && I.n < kExactFewCandidatesBase ? 128 : 256;
  const int64_t qpad = (int64_t)ceil_div(nq, BM) * BM, npad = (int64_t)ceil_div(I.n, FILTER_TN) * FILTER_TN;
  FilterPlan plan = plan_filter(I.n, std::max(k, 16), nq);
  // test hook: every query through the listed FP32 scan
  if (const char* e = getenv("LSHG_TC_FORCE_FALLBACK"); e && e[0] == '1') plan.cap = 0;
  int C = 32;
  while (C < k) C <<= 1;
  const int64_t room = listed_scan_room(nq, C, (int64_t)nq * plan.cap);
  try {
    DevBuf<uint16_t> qbf((size_t)qpad * KD, s);
    DevBuf<float> eps((size_t)nq, s), tau((size_t)nq, s), qnorm((size_t)nq, s);
    DevBuf<int> cnt((size_t)nq + 1 + nq, s);  // [0, nq): survivors; [nq]: listed; then the list
    // survivors, then (the re-rank reads `best`) the lists of the FP32 scan
    DevBuf<uint64_t> cand((size_t)room, s), best((size_t)nq * CT, s);
    int* ovf = cnt.ptr + nq;
    launch_unit_rows(q, nq, I.d, qpad, qbf.ptr, nullptr, I.ebf_res.ptr, eps.ptr, cnt.ptr, nq + 1, s);
    const FilterMaps maps = make_filter_maps(qbf.ptr, qpad, I.ebf.ptr, npad, I.d, false);
    launch_filter_scan(maps, plan, nq, I.n, I.d, (int)(qpad / BM), tau.ptr, cnt.ptr, cand.ptr, I.error_word(s), s,
                       eps.ptr);
    launch_exact_select(cnt.ptr, cand.ptr, nq, plan.cap, (int)std::min<int64_t>(k, I.n), CT,
                        plan.M > 0 ? tau.ptr : nullptr, eps.ptr, best.ptr, ovf, tau.ptr, s);
    launch_rerank(best.ptr, nq, CT, I.x.ptr, I.n, I.d, I.xnorm.ptr, q, nullptr, DIST_ANGULAR, k, out, s,
                  I.error_word(s), false, nullptr, nullptr, qnorm.ptr);
    launch_scan_float_listed(I.xt.ptr, I.n, I.d, I.xnorm.ptr, q, nq, qnorm.ptr, DIST_ANGULAR, ovf, tau.ptr, C, cand.ptr,
                             room, k, out, s);
  } catch (const Error& e) {
    if (e.status != LSHG_ERR_OUT_OF_MEMORY) throw;
    cudaGetLastError();  // temporaries that do not fit: the FP32 scan needs fewer
    return false;
  }
  return true;
}

}  // namespace lshg
