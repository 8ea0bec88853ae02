// Exact generalized-Jaccard top-k through 8-bit rows (implementation 2; the reference's plain exact
// scan, memOptimizedLinearScan.cu:20-106, with generalizedJaccard, distanceFunctions.cuh:10-21):
// ids and distances are those of the FP32 scan of scan_float.cu, bit for bit.
//
// The FP32 scan pays two minima or maxima (half rate) and two additions a dimension of every
// pair.  Here every pair is first bounded from 8-bit codes, four dimensions an instruction: with
// the codes u = rint(s (x - lo)) of [lo, lo + 255 / s], the base's range,
// sum min(u_q, u_x) = (sum u_q + sum u_x - sum |u_q - u_x|) / 2, and the distance lies between the
// bounds of rerank_bounds.cu (the same residuals and allowance for FP32 arithmetic).  Two passes:
//   thresholds  the smallest upper bound of every 32 points of every S-th tile; T[q] = the k-th
//               smallest of these (k different points have at most it), so the k-th smallest
//               distance is at most T;
//   candidates  points whose lower bound is at most T -- every point of the top-k -- are listed
//               (at most 512 or 1,024 a query) and scored with the reference's formula (launch_rerank).
// Queries with more candidates, or with a negative or non-finite value, are scanned by the FP32
// scan from a list on the device, starting from T.  A base with such a value, or whose rows lie too
// close for the codes (crowded_rows_kernel), always takes it.
//
// scan kernel: a CTA takes 64 queries and a run of 128-point tiles, warp w queries 8w .. 8w + 7,
// lane l points 4l .. 4l + 3: 32 sums a thread, three shared 16-byte loads a four-dimension step.
// Measured (60,013 x 100, 129 queries, k = 10): the FP32 scan 413 us, this 85 (the two passes 15 + 27,
// the re-rank 14; the rest is launches and latency); 1M x 100, one query 2,140 -> 117, 100 queries, k =
// 32, 2,640 -> 631.  Both passes are bounded by the integer ALU (77 and 83% busy, memory idle).  With
// the divisions of every bound in place of the linear form below the second pass took 49 us against 31.
#include <algorithm>

#include "index.h"
#include "launch_count.h"
#include "launch_next.cuh"
#include "profile.h"
#include "tc_filter.h"

namespace lshg {

namespace {

constexpr int kTile = 128;
constexpr int kQB = 64;
constexpr int kMinDim = 16;   // 8-bit codes of fewer dimensions leave too many candidates
constexpr int kMaxDim = 128;  // the listed FP32 scan's shared memory
constexpr int kMinBase = 4096;
constexpr int64_t kMinPairs = 16384;
// Group maxima a query at most: groups span several tiles on bases that have more.  (1.2M points, k
// = 32, had 37,500, 150 KB a query, which also took the threshold select's slowest form; any group
// bounds as well, and with 48 groups or more for each of the k the threshold hardly moves.)
constexpr int kMaxGroups = 6144;

__device__ __forceinline__ unsigned code(float v, float s) {
  return (unsigned)__float2int_rn(fminf(fmaxf(v * s, 0.0f), 255.0f));
}

__device__ __forceinline__ unsigned sad4(unsigned a, unsigned b, unsigned c) {  // c + sum |a_i - b_i|
  unsigned r;
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

__device__ __forceinline__ float delta(int d) { return (2.0f * d + 7.0f) * 1.2e-7f + 2e-6f; }

// ROWS rows a block: their codes as [wd][ROWS] words (byte j of word w = dimension 4w + j), and for
// each row (2 s S, U - 2 s E, U + 2 s E, 0): S its sum, U its codes' sum + s lo d, E its share of what the
// codes and the FP32 sums hide.  With these of a query and a point added and A = sum |u_q - u_x|,
// A_lo = (P - A) / 2 s and A_hi = (Q - A) / 2 s bound the sum of minima.  bad[i] = 1 for a row without
// bounds.
// A warp a row, its (at most four) loads in flight together; queries' few blocks take 32 warps
// (one row after another by 8 warps: 17 us of a batch of 129).
template <int ROWS, int THREADS>
__global__ void __launch_bounds__(THREADS)
    code_tiles_kernel(const float* __restrict__ x, int64_t n, int d, int wd, float lo, float s,
                      uint32_t* __restrict__ out, float4* __restrict__ tails, int* __restrict__ bad, int* counters, int ncounters) {
  grid_ready();
  zero_counters(counters, ncounters);
  extern __shared__ uint32_t rows[];  // [ROWS][wd | 1]
  const int pitch = wd | 1, lane = threadIdx.x & 31;
  const int64_t row0 = (int64_t)blockIdx.x * ROWS;
  const float inv = 1.0f / s;
  for (int r = threadIdx.x >> 5; r < ROWS; r += THREADS / 32) {
    const int64_t i = row0 + r;
    uint8_t* codes = reinterpret_cast<uint8_t*>(rows + r * pitch);
    float v[kMaxDim / 32];
#pragma unroll
    for (int t = 0; t < kMaxDim / 32; ++t) v[t] = i < n && 32 * t + lane < d ? x[i * d + 32 * t + lane] : 0.0f;
    float sum = 0.0f, err = 0.0f;
    unsigned total = 0;
    bool wrong = false;
#pragma unroll
    for (int t = 0; t < kMaxDim / 32; ++t) {
      const int c = 32 * t + lane;
      unsigned u = 0;
      if (c < d) {
        wrong |= !(v[t] >= 0.0f && v[t] <= 1e18f);
        u = code(v[t] - lo, s);
        total += u;
        sum += v[t];
        err += fabsf(v[t] - (lo + (float)u * inv));
      }
      if (c < 4 * wd) codes[c] = (uint8_t)u;
    }
    total = __reduce_add_sync(0xffffffffu, total);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      err += __shfl_xor_sync(0xffffffffu, err, o);
    }
    wrong = __any_sync(0xffffffffu, wrong) || !(sum > 1e-6f && 2.0f * s * sum < 1e30f);
    if (lane == 0) {
      const float e = 2.0f * s * (err * 1.0001f + sum * 2e-5f);
      const float u = (float)total + s * lo * (float)d;
      tails[row0 + r] = make_float4(2.0f * s * sum, u - e, u + e, 0.0f);
      if (bad && i < n) bad[i] = wrong ? 1 : 0;
    }
  }
  __syncthreads();
  uint32_t* dst = out + (int64_t)blockIdx.x * wd * ROWS;
  for (int i = threadIdx.x; i < wd * ROWS; i += THREADS) dst[i] = rows[(i % ROWS) * pitch + i / ROWS];
}

// Tiles 0, stride, 2 stride, ... (ntiles of them; tile i below is the i-th).
// MODE 0: gmax[q][4 i + g] = -(smallest upper bound of tile i's 32 points of group g).
// MODE 2: the same with groups over the tiles i gt .. i gt + gt - 1 (tiles_per_split is a multiple of gt).
// MODE 1: points with a lower bound <= T = -tau[q] appended to cand[q][0..cap) (cnt[q] counts
// all).  The sums start at 2^23 as a float's bits, so they are read as floats without conversions.
template <int MODE>
__global__ void __launch_bounds__(256, 4)
    jaccard_scan_kernel(const uint32_t* __restrict__ xt, const float4* __restrict__ xtail, int64_t n, int wd, int d,
                        const uint32_t* __restrict__ qt, const float4* __restrict__ qtail,
                        const int* __restrict__ qbad, int nq, int ntiles, int tiles_per_split, int stride, int gt,
                        float* __restrict__ gmax, const float* __restrict__ tau, int* __restrict__ cnt,
                        uint64_t* __restrict__ cand, int cap) {
  grid_ready();
  constexpr unsigned kOne = 0x4b000000u;  // 2^23
  extern __shared__ __align__(16) uint32_t sm[];
  uint32_t* xs = sm;               // [wd][128]
  uint32_t* qs = sm + wd * kTile;  // [wd][64]
  __shared__ float2 xl[kTile], ql[kQB];
  __shared__ float runs[MODE == 2 ? kQB : 1][4];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int q0 = blockIdx.x * kQB;
  const int t0 = blockIdx.y * tiles_per_split, t1 = min(ntiles, t0 + tiles_per_split);
  for (int i = tid; i < wd * kQB / 4; i += 256)
    reinterpret_cast<uint4*>(qs)[i] = reinterpret_cast<const uint4*>(qt + (int64_t)blockIdx.x * wd * kQB)[i];
  if (tid < kQB) {
    const int q = q0 + tid;
    const float4 v = qtail[q];
    if (MODE != 1) {
      ql[tid] = make_float2(v.x, v.y);
    } else {
      // 1 - A_hi / (S - A_hi) - delta <= T  <=>  A_hi >= S c / (1 + c), c = 1 - delta - T
      //                                    <=>  A <= Q - (2 s S) c / (1 + c);
      // two units for the roundings at 2^23
      float r = 0.0f, lim = -INFINITY;
      if (q < nq && !qbad[q]) {
        const float c = 1.0f - delta(d) + tau[q];
        r = -c / (1.0f + c);
        lim = v.z + r * v.x + (8388608.0f + 2.0f);
        if (!(tau[q] > -2.0f)) { r = 0.0f; lim = INFINITY; }  // no threshold
      }
      ql[tid] = make_float2(r, lim);
    }
  }
  for (int t = t0; t < t1; ++t) {
    __syncthreads();  // the previous tile has been read
    const int64_t row0 = (int64_t)t * stride * kTile;
    for (int i = tid; i < wd * kTile / 4; i += 256)
      reinterpret_cast<uint4*>(xs)[i] = __ldg(reinterpret_cast<const uint4*>(xt + row0 * wd) + i);
    if (tid < kTile) {
      const float4 v = __ldg(xtail + row0 + tid);
      xl[tid] = make_float2(v.x, MODE != 1 ? v.y : v.z);
    }
    __syncthreads();
    if (q0 + 8 * w >= nq) continue;  // no query of this warp: it only copies
    unsigned acc[8][4];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = kOne;
#pragma unroll 2
    for (int j = 0; j < wd; ++j) {
      const uint4 xv = *reinterpret_cast<const uint4*>(xs + j * kTile + 4 * lane);
      const uint4 qa = *reinterpret_cast<const uint4*>(qs + j * kQB + 8 * w);
      const uint4 qb = *reinterpret_cast<const uint4*>(qs + j * kQB + 8 * w + 4);
      const unsigned xb[4] = {xv.x, xv.y, xv.z, xv.w};
      const unsigned qv[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = sad4(xb[b], qv[a], acc[a][b]);
    }
    const int64_t left = n - row0 - 4 * lane;  // points of this thread that exist
    float2 xv[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) xv[b] = xl[4 * lane + b];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const float2 qv = ql[8 * w + a];
      const int q = q0 + 8 * w + a;
      if (MODE != 1) {
        float best = 0.0f;  // the largest A_lo / S
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const float A = __uint_as_float(acc[a][b]) - 8388608.0f;
          const float R = __fdividef(qv.y + xv[b].y - A, qv.x + xv[b].x);
          if (b < left) best = fmaxf(best, R);
        }
        best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, 1));
        best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, 2));
        best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, 4));
        // a group without points bounds nothing
        if ((lane & 7) == 0 && q < nq) {
          float up = left > 0 ? __fdividef(best, 1.0f - best) - 1.0f - delta(d) : -INFINITY;
          if (MODE == 0) {
            gmax[(int64_t)q * 4 * ntiles + 4 * t + (lane >> 3)] = up;
          } else {
            float* run = &runs[8 * w + a][lane >> 3];  // this thread's own
            const int in = t % gt;
            if (in) up = fmaxf(up, *run);
            *run = up;
            if (in == gt - 1 || t == ntiles - 1)
              gmax[(int64_t)q * 4 * ((ntiles + gt - 1) / gt) + 4 * (t / gt) + (lane >> 3)] = up;
          }
        }
      } else {
        unsigned hits = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (__uint_as_float(acc[a][b]) <= fmaf(qv.x, xv[b].x, xv[b].y) + qv.y && b < left) hits |= 1u << b;
        if (hits) {  // q < nq: the limit is -inf beyond
          int pos;
          const unsigned who = __activemask();
          if (__popc(who) <= 8) {
            pos = atomicAdd(cnt + q, __popc(hits));
            // a query past its places is scanned in full: its other points need not be looked for
            if (pos >= cap) ql[8 * w + a] = make_float2(0.0f, -INFINITY);
          } else {
            // One addition for the lanes that are here together: a query that ties with much of the base
            // takes its places in the first tiles of every CTA at the same time (60,000 rows of 16, a
            // third of them copies of each of 500 queries: the pass 348 us with an addition a lane, 39
            // this way).
            int before = 0, sum = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              const unsigned mk = __ballot_sync(who, hits >> b & 1u);
              before += __popc(mk & ((1u << lane) - 1u));
              sum += __popc(mk);
            }
            const int first = __ffs(who) - 1;
            const int base = __shfl_sync(who, lane == first ? atomicAdd(cnt + q, sum) : 0, first);
            pos = base + before;  // after the points of the lanes below
            if (base + sum > cap) ql[8 * w + a] = make_float2(0.0f, -INFINITY);
          }
          for (unsigned h = hits; h; h &= h - 1, ++pos)
            if (pos < cap) cand[(int64_t)q * cap + pos] = make_key(0.0f, (int)(row0 + 4 * lane + __ffs(h) - 1));
        }
      }
    }
  }
}

// Rows i of 64 spread over the base that have more than `most` of 256 other points, spread as well,
// within the codes' resolution: a lower bound of their distance at most the row's upper bound to itself.
constexpr int kProbeRows = 64, kProbePoints = 256;
__global__ void __launch_bounds__(kProbePoints)
    crowded_rows_kernel(const uint32_t* __restrict__ xt, const float4* __restrict__ xtail, int64_t n, int wd, int most,
                        int* __restrict__ crowded) {
  grid_ready();
  const int64_t step = n / kProbePoints;
  const int64_t i = (2 * blockIdx.x + 1) * n / (2 * kProbeRows) + step / 2;
  const unsigned t = threadIdx.x;
  const int64_t j = t * n / kProbePoints + ((t + 1) * 2654435761u >> 8) % (unsigned)step;  // no period
  const uint32_t *ci = xt + i / kTile * wd * kTile + i % kTile, *cj = xt + j / kTile * wd * kTile + j % kTile;
  unsigned A = 0;
  for (int w = 0; w < wd; ++w) A = sad4(ci[w * kTile], cj[w * kTile], A);
  const float4 vi = xtail[i], vj = xtail[j];
  const bool near = i != j && (vi.z + vj.z - (float)A) / (vi.x + vj.x) >= vi.y / vi.x;
  const int cnt = __syncthreads_count(near);
  if (t == 0 && cnt > most) atomicAdd(crowded, 1);
}

// Queries to scan in full: more candidates than places, fewer than k, or no bounds.  The re-rank has
// nothing of them to do: their candidates are emptied, and tau becomes the full scan's distance limit T.
__global__ void list_hard_kernel(const int* __restrict__ cnt, const int* __restrict__ bad, int nq, int k,
                                 int cap, uint64_t* __restrict__ cand, int* __restrict__ list,
                                 float* __restrict__ tau) {
  grid_ready();
  const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (q >= nq) return;
  const int c = cnt[q];
  const bool hard = bad[q] || c > cap || c < k;
  for (int i = lane + (hard ? 0 : c); i < cap; i += 32) cand[(int64_t)q * cap + i] = kEmptyKey;
  if (hard && lane == 0) {
    list[1 + atomicAdd(list, 1)] = q;
    tau[q] = bad[q] || c < k ? INFINITY : -tau[q];
  }
}

size_t tile_smem(int wd, int rows) { return (size_t)rows * (wd | 1) * 4; }

}  // namespace

void derive_jaccard_scan(Index& I, cudaStream_t s) {
  if (I.p.framework != 0 || I.dist != DIST_JACCARD || I.d < kMinDim || I.d > kMaxDim || I.n < kMinBase) return;
  float lo, hi;
  if (!base_range(I.x.ptr, I.n * I.d, &lo, &hi, s)) return;
  const int wd = ceil_div(I.d, 4), tiles = ceil_div(I.n, kTile);
  try {
    I.jq.alloc((size_t)tiles * wd * kTile, s);
    I.jq_tail.alloc((size_t)tiles * kTile, s);
  } catch (const Error& e) {  // no room for the codes: the FP32 scan needs none
    if (e.status != LSHG_ERR_OUT_OF_MEMORY) throw;
    cudaGetLastError();
    I.jq.release();
    return;
  }
  I.jq_lo = lo;
  I.jq_scale = 255.0f / std::max(hi - lo, 1e-6f * hi);
  const size_t smem = tile_smem(wd, kTile);
  launch_next(code_tiles_kernel<kTile, 256>, tiles, 256, smem, s, I.x.ptr, I.n, I.d, wd, I.jq_lo, I.jq_scale, I.jq.ptr,
              I.jq_tail.ptr, nullptr, nullptr, 0);
  count_launch();
  LSHG_CHECK_LAUNCH();
  // A base whose rows mostly have more points within the codes' resolution than a query has places --
  // 60,013 rows that differ by less than a code, or copies of ten -- would be scanned twice: 1,000
  // queries, k = 32, filtered and rescanned 1,512 and 1,308 us, the FP32 scan alone 1,106 and 978.
  DevBuf<int> crowded(1, s);
  LSHG_CUDA(cudaMemsetAsync(crowded.ptr, 0, sizeof(int), s));
  const int most = (int)std::max<int64_t>(2, (int64_t)1024 * kProbePoints / I.n);
  launch_next(crowded_rows_kernel, kProbeRows, kProbePoints, 0, s, I.jq.ptr, I.jq_tail.ptr, I.n, wd, most, crowded.ptr);
  count_launch();
  LSHG_CHECK_LAUNCH();
  int h = 0;
  LSHG_CUDA(cudaMemcpyAsync(&h, crowded.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
  LSHG_CUDA(cudaStreamSynchronize(s));
  if (2 * h > kProbeRows) {
    I.jq.release();
    I.jq_tail.release();
  }
}

bool query_jaccard_filtered(Index& I, const float* q, int nq, int k, lshg_point* out, cudaStream_t s) {
  const int wd = ceil_div(I.d, 4), tiles = ceil_div(I.n, kTile), qblocks = ceil_div(nq, kQB);
  if (!I.jq.ptr || k > std::min(128, tiles) || (int64_t)nq * I.n < kMinPairs) return false;
  const int cap = k <= 64 ? 512 : 1024;  // candidates a query, re-scored
  // Every S-th tile for the thresholds: the bounds pass about 5 S k candidates (60,013 sparse rows of
  // 100: 150 at S k = 32, at most 255), within the places, and never fewer than 4 k groups.
  const int S = std::max(1, std::min({8, cap / 16 / k, tiles / k})), stiles = ceil_div(tiles, S);
  const int gt = ceil_div(4 * (int64_t)stiles, kMaxGroups), groups = 4 * ceil_div(stiles, gt);
  int C = 32;
  while (C < k) C <<= 1;
  const int64_t room = listed_scan_room(nq, C, (int64_t)nq * cap);
  try {
    DevBuf<uint32_t> qt((size_t)qblocks * wd * kQB, s);
    DevBuf<float4> qtail((size_t)qblocks * kQB, s);
    DevBuf<int> ctl((size_t)3 * nq + 1, s);  // [0, nq): candidates; [nq]: listed, then their list; then no bounds
    DevBuf<float> gmax((size_t)nq * groups, s), tau((size_t)nq, s);
    DevBuf<uint64_t> cand((size_t)room, s);  // candidates, then the lists of the FP32 scan
    int *cnt = ctl.ptr, *list = ctl.ptr + nq, *bad = ctl.ptr + 2 * nq + 1;
    const size_t qsm = tile_smem(wd, kQB);
    launch_next(code_tiles_kernel<kQB, 1024>, qblocks, 1024, qsm, s, q, nq, I.d, wd, I.jq_lo, I.jq_scale, qt.ptr,
                qtail.ptr, bad, cnt, nq + 1);
    count_launch();
    LSHG_CHECK_LAUNCH();
    // two rounds of four CTAs an SM where there are tiles enough, at least two tiles each
    auto split = [&](int nt) {
      return ceil_div(nt, std::max(1, std::min(ceil_div(nt, 2), ceil_div(num_sms() * 8, qblocks))));
    };
    const int tps0 = ceil_div(split(stiles), gt) * gt, tps = split(tiles);
    const dim3 grid0(qblocks, ceil_div(stiles, tps0)), grid(qblocks, ceil_div(tiles, tps));
    const size_t smem = (size_t)wd * (kTile + kQB) * 4;
    auto bounds = gt == 1 ? jaccard_scan_kernel<0> : jaccard_scan_kernel<2>;
    raise_smem_limit(bounds, smem);
    raise_smem_limit(jaccard_scan_kernel<1>, smem);
    {
      ProfScope _ps("jaccard_bounds", s);
      launch_next(bounds, grid0, 256, smem, s, I.jq.ptr, I.jq_tail.ptr, I.n, wd, I.d, qt.ptr, qtail.ptr, bad, nq,
                                                      stiles, tps0, S, gt, gmax.ptr, nullptr, nullptr, nullptr, 0);
      count_launch();
      LSHG_CHECK_LAUNCH();
    }
    tc::launch_tau_select(gmax.ptr, nq, groups, k, 0.0f, tau.ptr, s);
    {
      ProfScope _ps("jaccard_filter", s);
      launch_next(jaccard_scan_kernel<1>, grid, 256, smem, s, I.jq.ptr, I.jq_tail.ptr, I.n, wd, I.d, qt.ptr, qtail.ptr, bad, nq,
                                                     tiles, tps, 1, 1, nullptr, tau.ptr, cnt, cand.ptr, cap);
      count_launch();
      LSHG_CHECK_LAUNCH();
    }
    launch_next(list_hard_kernel, ceil_div(nq, 8), 256, 0, s, cnt, bad, nq, (int)std::min<int64_t>(k, I.n), cap,
                cand.ptr, list, tau.ptr);
    count_launch();
    LSHG_CHECK_LAUNCH();
    launch_rerank(cand.ptr, nq, cap, I.x.ptr, I.n, I.d, nullptr, q, nullptr, DIST_JACCARD, k, out, s, I.error_word(s));
    launch_scan_float_listed(I.xt.ptr, I.n, I.d, nullptr, q, nq, nullptr, DIST_JACCARD, list, tau.ptr, C, cand.ptr,
                             room, k, out, s);
  } catch (const Error& e) {
    if (e.status != LSHG_ERR_OUT_OF_MEMORY) throw;
    cudaGetLastError();  // temporaries that do not fit: the FP32 scan needs fewer
    return false;
  }
  return true;
}

}  // namespace lshg
