// Re-rank of long candidate lists through quantised rows: which of a query's candidates can be in
// its top-k is decided from 8-bit copies of the rows and bounds on what they hide, and only those
// are scored from the FP32 rows (launch_rerank), so the results are those of scoring every
// candidate (rerank.cu, restating candidateSetScan, candidateSetScanner.cuh:10-32; for LSH
// tables lsh.cu's scoring of the distinct candidates).
//
// Generalized Jaccard.  A row x >= 0 is kept as u = rint(s x) (s = 255 / the base's largest
// value, one scale for all rows) with its sum S(x) and its residual e(x) = sum |x - u / s|.  For a
// query quantised the same way, M = sum min(u_q, u_x) / s is an integer sum, and
//     |sum min(q, x) - M| <= sum max(|q - u_q / s|, |x - u_x / s|) <= e(q) + e(x) = E.
// sum max = S(q) + S(x) - sum min, so the similarity A / (S - A) rises with A = sum min and
// M - E, M + E bound the distance from above and below.
//
// Angular.  A row is kept as c = rint(s u), u = x / |x| and s = 127 / max |u_j| (a scale a row),
// with 1 / s and r(x) = |u - c / s|.  The query has 16-bit codes (its residual, half of E with
// 8-bit ones, all but goes away: a SimHash list of 1,024 keeps 120 candidates, not 300), split
// into two 8-bit halves.  The cosine is within E = r(q) + r(x) + r(q) r(x) of c_q . c_x / (s_q
// s_x), an integer dot product.
//
// delta covers the FP32 arithmetic of the reference's formulas ((2 d + 3) and (2 d + 7) 2^-24,
// fp64_band, while norms are in [2^-40, 2^40]) and of this kernel's (a quotient within 2^-21,
// sums within d 2^-24).  With T the k-th smallest upper bound of the list, every candidate of
// the top-k has a lower bound of at most T.  Lists with more than kKeep such candidates, and
// queries whose values have no such bounds, are scored in full (from a list on the device).
//
// A row of 100 dimensions is 128 bytes here against 400 (angular, 128 dimensions: 160 against
// 512), and about 60 of 4,096 Jaccard candidates, 130 of 1,900 of an LSH query, are left at k =
// 32.  Eight lanes read a row, 16 bytes each.  The Jaccard kernel is bounded by its instructions
// (minima as packed 16-bit pairs: 1.15 ms, 28 a row), the LSH lists' by instructions and gathers
// together (600k x 128: 75% of the issue slots, waiting for rows otherwise): bounds of 4
// bytes a candidate and 48 registers let five CTAs share an SM (8 bytes and 58: 0.66 ms).
// Measured (10,000 queries): Jaccard, C = 4,096,
// 500k x 100: partition, gather of every row and select 2.77 ms; this way 0.74 + 0.15 ms.
// LSH tables, 1M x 128: scoring 1.31 ms; this way 0.48 + 0.18.  SimHash, C = 1,024, 1.2M x 100: 0.75
// ms; 0.32 + 0.15.
#include <algorithm>

#include "common.cuh"
#include "index.h"
#include "kernels.h"
#include "launch_count.h"
#include "launch_next.cuh"
#include "profile.h"

namespace lshg {

namespace {

constexpr int kMaxJaccardDim = 120;  // 8 bytes of a 128-byte row hold S and e
constexpr int kMaxAngularDim = 128;
constexpr float kQueryLevels = 127.0f * 256.0f;  // 16-bit codes whose rounded upper half is 8-bit
constexpr float kNormMin = 9.094947e-13f, kNormMax = 1.0995116e12f;  // 2^-40, 2^40
constexpr int kKeep = kBoundsKeep;  // candidates a query passed on
constexpr int kBoundThreads = 256;
// Smaller batches are scored in full: their rows' gather is no longer than one more launch (one
// JL query, C = 1,024: 543 us in full, 556 through bounds).
constexpr int64_t kBoundsMinCandidates = 16384;

int jaccard_pitch(int d) { return (d + 8 + 31) / 32 * 32; }
int angular_pitch(int d) { return (d + 15) / 16 * 16; }

// stat[0]: bits of the largest value; stat[1]: 1 when a value is negative or not finite; stat[2]:
// complement of the bits of the smallest value.
__global__ void base_range_kernel(const float* __restrict__ x, int64_t total, unsigned* stat) {
  float m = 0.0f, lo = INFINITY;
  bool bad = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = fabsf(x[i]) == 0.0f ? 0.0f : x[i];  // -0: its bits are not ordered
    if (v >= 0.0f && v <= 1e18f) m = fmaxf(m, v), lo = fminf(lo, v);
    else bad = true;
  }
  const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  const unsigned wl = __reduce_max_sync(0xffffffffu, ~__float_as_uint(lo));
  const bool wb = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(stat, w);
    atomicMax(stat + 2, wl);
    if (wb) atomicExch(stat + 1, 1u);
  }
}

__device__ __forceinline__ unsigned quantise(float v, float s) { return (unsigned)__float2int_rn(fminf(v * s, 255.0f)); }

// One warp a row: codes, then in the row's last 8 bytes S (float), the codes' sum (16 bits) and e
// (the upper 16 bits of a float, rounded up).
__global__ void quantise_rows_kernel(const float* __restrict__ x, int64_t n, int d, int pitch, float s,
                                     uint8_t* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const float inv = 1.0f / s;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
    float sum = 0.0f, err = 0.0f;
    unsigned codes = 0;
    uint8_t* row = out + i * pitch;
    for (int c = lane; c < pitch - 8; c += 32) {
      const float v = c < d ? x[i * d + c] : 0.0f;
      const unsigned u = quantise(v, s);
      row[c] = (uint8_t)u;
      sum += v;
      codes += u;
      err += fabsf(v - (float)u * inv);
    }
    codes = __reduce_add_sync(0xffffffffu, codes);  // at most 120 * 255
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      err += __shfl_xor_sync(0xffffffffu, err, o);
    }
    if (lane == 0)
      *reinterpret_cast<uint2*>(row + pitch - 8) =
          make_uint2(__float_as_uint(sum), ((__float_as_uint(err) + 0xffffu) & 0xffff0000u) | codes);
  }
}

__device__ __forceinline__ int dot16(const uint4& r, const unsigned (&w)[4]) {
  return __dp4a((int)r.x, (int)w[0],
                __dp4a((int)r.y, (int)w[1], __dp4a((int)r.z, (int)w[2], __dp4a((int)r.w, (int)w[3], 0))));
}

// A row's angular quantisation to codes of magnitude at most `levels`: its values (four a lane), v *
// unit = the unit vector's, and the codes rint(v * mul), each worth inv.  Computed by a whole warp;
// ok: the norm is in range.
struct AngularScale {
  float unit, mul, inv;
  bool ok;
};
__device__ __forceinline__ AngularScale angular_scale(const float* __restrict__ row, int d, int lane, float levels,
                                                      float (&v)[4]) {
  float ss = 0.0f, m = 0.0f;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int j = c * 32 + lane;
    v[c] = j < d ? row[j] : 0.0f;
    ss = fmaf(v[c], v[c], ss);
    m = fmaxf(m, fabsf(v[c]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  AngularScale a;
  a.ok = ss >= kNormMin * kNormMin && ss <= kNormMax * kNormMax;  // false for NaN
  a.unit = a.ok ? rsqrtf(ss) : 0.0f;
  const float top = m * a.unit;  // the largest component: at least 1 / sqrt(128) where ok
  a.inv = a.ok ? top / levels : 0.0f;
  a.mul = a.ok ? a.unit * (levels / top) : 0.0f;
  return a;
}

// Angular rows, a warp each: codes (zeros past d), and 1 / s and r (rounded up, the FP32
// normalisation's 2^-18 included) in tails[i].  A row out of range raises *bad.
__global__ void quantise_angular_kernel(const float* __restrict__ x, int64_t n, int d, int pitch,
                                        int8_t* __restrict__ out, float2* __restrict__ tails, unsigned* bad) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  bool wrong = false;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
    float v[4];
    const AngularScale a = angular_scale(x + i * d, d, lane, 127.0f, v);
    wrong |= !a.ok;
    float rr = 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = c * 32 + lane;
      const int u = __float2int_rn(v[c] * a.mul);
      const float df = v[c] * a.unit - (float)u * a.inv;
      rr = fmaf(df, df, rr);
      if (j < pitch) out[i * pitch + j] = (int8_t)u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rr += __shfl_xor_sync(0xffffffffu, rr, o);
    if (lane == 0) tails[i] = make_float2(a.inv, sqrtf(rr) * 1.001f + 4e-6f);
  }
  if (wrong) atomicExch(bad, 1u);
}

// near[b]: of kProbePoints points spread over the base (all of a smaller one), those within the codes'
// resolution of row b of kProbeRows: a distance that the residuals of both may hide.
constexpr int kProbeRows = 64, kProbePoints = 8192;
__global__ void __launch_bounds__(256) near_rows_kernel(const uint8_t* __restrict__ rows,
                                                        const float2* __restrict__ tails, int64_t n, int pitch,
                                                        int points, unsigned* __restrict__ near) {
  const int64_t step = n / points;  // at least 1
  const int64_t i = (2 * blockIdx.x + 1) * n / (2 * kProbeRows);
  const unsigned t = blockIdx.y * blockDim.x + threadIdx.x;
  bool in = false;
  if ((int)t < points) {
    const int64_t j = t * n / points + ((t + 1) * 2654435761u >> 8) % (unsigned)step;  // no period
    int dot = 0;
    for (int w = 0; w < pitch / 4; ++w)
      dot = __dp4a(*reinterpret_cast<const int*>(rows + i * pitch + 4 * w),
                   *reinterpret_cast<const int*>(rows + j * pitch + 4 * w), dot);
    const float2 ti = tails[i], tj = tails[j];
    in = i != j && 1.0f - (float)dot * (ti.x * tj.x) <= ti.y + tj.y;
  }
  const int c = __syncthreads_count(in);
  if (threadIdx.x == 0 && c) atomicAdd(near + blockIdx.x, (unsigned)c);
}

// Bounds are kept as 16-bit steps of a distance in [-0.0625, 2.0625), rounded outwards (a step is
// 3.2e-5, a tenth of the narrowest bounds); kEmptyStep: none.
constexpr float kBase = -0.0625f, kStepsPer = 65000.0f / 2.125f;
constexpr int kEmptyStep = 0xffff;
__device__ __forceinline__ uint32_t step_down(float d) {
  return (uint32_t)fminf(fmaxf(floorf((d - kBase) * kStepsPer) - 1.0f, 0.0f), 65000.0f);
}
__device__ __forceinline__ uint32_t step_up(float d) {
  return (uint32_t)fminf(fmaxf(ceilf((d - kBase) * kStepsPer) + 1.0f, 0.0f), 65001.0f);
}

// One block a query; see the header.  The candidates: cand[qi][0..C) keys, or (LIST) ids
// list[qi][0..C) of which ccnt[qi] are there (a query with more than C is another kernel's).
// kept: [nq][kKeep] keys (ids of the candidates that can be in the top-k, then empty keys);
// listed: count, then the queries to score in full.  s: the Jaccard scale; tails: angular.
template <int DIST, int C, bool LIST>
__global__ void __launch_bounds__(kBoundThreads, 5) bounds_kernel(
    const uint64_t* __restrict__ cand, const int* __restrict__ list, int list_cap, const int* __restrict__ ccnt,
    const uint8_t* __restrict__ rows, const float2* __restrict__ tails, int pitch, float s, int64_t n, int d,
    const float* __restrict__ q, int k, uint64_t* __restrict__ kept, int* __restrict__ listed) {
  grid_ready();
  constexpr bool JAC = DIST == DIST_JACCARD;
  constexpr int W = kBoundThreads / 32, PER = C / kBoundThreads;
  extern __shared__ uint32_t bnd[];  // [C] lower bound << 16 | upper bound, in steps of 1 / kStepsPer from kBase
  __shared__ int wcnt[2][W];
  __shared__ int total;
  const int qi = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int have = LIST ? ccnt[qi] : C;  // candidates
  const float* qr = q + (int64_t)qi * d;
  // the query's scale, sum and residual (every warp computes them)
  float inv, sq = 0.0f, eq = 0.0f, mul = s;
  bool bad = false;
  if (JAC) {
    inv = 1.0f / s;
    for (int c = lane; c < d; c += 32) {
      const float v = qr[c];
      bad |= !(v >= 0.0f && v <= 1e18f);
      sq += v;
      eq += fabsf(v - (float)quantise(v, s) * inv);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      eq += __shfl_xor_sync(0xffffffffu, eq, o);
    }
  } else {
    float v[4];
    const AngularScale a = angular_scale(qr, d, lane, kQueryLevels, v);
    bad = !a.ok;
    inv = a.inv;
    mul = a.mul;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float df = v[c] * a.unit - (float)__float2int_rn(v[c] * a.mul) * a.inv;
      eq = fmaf(df, df, eq);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) eq += __shfl_xor_sync(0xffffffffu, eq, o);
    eq = sqrtf(eq) * 1.001f + 4e-6f;
  }
  if (LIST && have > list_cap) {  // block-uniform
    for (int i = tid; i < kKeep; i += kBoundThreads) kept[(int64_t)qi * kKeep + i] = kEmptyKey;
    return;
  }
  if (__any_sync(0xffffffffu, bad)) {  // the same in every warp
    for (int i = tid; i < kKeep; i += kBoundThreads) kept[(int64_t)qi * kKeep + i] = kEmptyKey;
    if (tid == 0) listed[1 + atomicAdd(listed, 1)] = qi;
    return;
  }
  const int part = lane & 7, parts = pitch / 16;  // 16-byte part of a row
  unsigned qw[4];                                 // this lane's 16 query codes
  unsigned ql[4];                                 // angular: their lower halves
  int uq = 0;                                     // Jaccard: the sum of all the query's codes
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    qw[e] = ql[e] = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = part * 16 + 4 * e + j;
      if (c < d) {  // codes past d: 0, as in the rows
        if (JAC) {
          const unsigned u = quantise(qr[c], s);
          qw[e] |= u << (8 * j);
          uq += (int)u;
        } else {
          const int u = __float2int_rn(qr[c] * mul), hi8 = (u + 128) >> 8;
          qw[e] |= ((unsigned)hi8 & 0xffu) << (8 * j);
          ql[e] |= ((unsigned)(u - hi8 * 256) & 0xffu) << (8 * j);
        }
      }
    }
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) uq += __shfl_xor_sync(0xffffffffu, uq, o);
  const float delta = (2.0f * d + 7.0f) * 1.2e-7f + 2e-6f;
  if (tid == 0) total = 0;
  // Bounds: a warp takes 16 candidates at a time, 8 lanes a row and four rows a load.  The sum of
  // minima is (sum u_q + sum u_x - sum |u_q - u_x|) / 2, and four bytes' absolute differences are
  // one instruction.  The four loads' sums are reduced together (four shuffles), which leaves
  // row `t` of its group in the lanes with part >> 1 == t.
  constexpr int U = 4;
  const int grp = lane >> 3, own = part >> 1;
  const bool tail = part == parts - 1;
  const int end = LIST ? (have + 15) & ~15 : C;  // at most C (a multiple of 256)
  for (int c0 = warp * 4 * U; c0 < end; c0 += W * 4 * U) {
    int id[U];
    uint4 r[U];
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const int i = c0 + 4 * t + grp;
      if (LIST) {
        id[t] = i < have ? list[(int64_t)qi * list_cap + i] : -1;
      } else {
        const uint64_t key = cand[(int64_t)qi * C + i];
        id[t] = key == kEmptyKey ? -1 : key_id(key);
      }
      if (id[t] >= n) id[t] = -1;
    }
#pragma unroll
    for (int t = 0; t < U; ++t) {
      r[t] = make_uint4(0, 0, 0, 0);
      if (id[t] >= 0 && part < parts)
        r[t] = __ldg(reinterpret_cast<const uint4*>(rows + (int64_t)id[t] * pitch) + part);
    }
    const int oid = own == 0 ? id[0] : own == 1 ? id[1] : own == 2 ? id[2] : id[3];
    uint2 rt = make_uint2(0, 0);  // the own row's sum or scale, and its residual
    if (oid >= 0)
      rt = JAC ? __ldg(reinterpret_cast<const uint2*>(rows + (int64_t)oid * pitch + pitch - 8))
               : __ldg(reinterpret_cast<const uint2*>(tails + oid));
    unsigned sad[U];  // or the dot products
#pragma unroll
    for (int t = 0; t < U; ++t) {
      if (JAC)
        sad[t] = __vsadu4(r[t].x, qw[0]) + __vsadu4(r[t].y, qw[1]) + __vsadu4(tail ? 0u : r[t].z, qw[2]) +
                 __vsadu4(tail ? 0u : r[t].w, qw[3]);
      else  // |sum| <= 128 * 127 * 32512 < 2^31
        sad[t] = (unsigned)(dot16(r[t], qw) * 256 + dot16(r[t], ql));
    }
    // lanes with bit 2 of the part keep loads 2 and 3, then bit 1 the odd one, then bit 0 is summed
    const bool up = part & 4, odd = part & 2;
    unsigned x0 = up ? sad[2] : sad[0], x1 = up ? sad[3] : sad[1];
    x0 += __shfl_xor_sync(0xffffffffu, up ? sad[0] : sad[2], 4);
    x1 += __shfl_xor_sync(0xffffffffu, up ? sad[1] : sad[3], 4);
    unsigned x = odd ? x1 : x0;
    x += __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    if (!(part & 1)) {
      float l, h;
      if (JAC) {
        const float sx = __uint_as_float(rt.x), ex = __uint_as_float(rt.y & 0xffff0000u);
        const float S = sq + sx, M = (float)((uq + (int)(rt.y & 0xffffu) - (int)x) >> 1) * inv;
        const float E = (eq + ex) * 1.0001f + S * 2e-5f;
        const float ah = fminf(M + E, 0.5f * S), al = fmaxf(M - E, 0.0f);
        l = 1.0f - __fdividef(ah, S - ah) - delta;
        h = 1.0f - __fdividef(al, S - al) + delta;
        if (!(S > 1e-6f && S < 1e30f)) {  // no bound: always scored
          l = -1.0f;
          h = 4.0f;
        }
      } else {
        const float ex = __uint_as_float(rt.y);
        const float D = 1.0f - (float)(int)x * (inv * __uint_as_float(rt.x));
        const float E = (eq + ex + eq * ex) * 1.0001f + delta;
        l = D - E;
        h = D + E;
      }
      // rounded outwards; 0xffff in both: an empty place
      bnd[c0 + 4 * own + grp] = oid < 0 ? 0xffffffffu : step_down(l) << 16 | step_up(h);
    }
  }
  __syncthreads();
  // T: the k-th smallest upper bound, by bisection over the steps
  int v[PER];
  int mn = kEmptyStep, mx = 0;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    v[e] = kEmptyStep;
    if (e * kBoundThreads >= end) continue;  // block-uniform, here and below
    if (e * kBoundThreads + tid < end) v[e] = (int)(bnd[e * kBoundThreads + tid] & 0xffffu);
    if (v[e] < kEmptyStep) {
      mn = min(mn, v[e]);
      mx = max(mx, v[e]);
    }
  }
  auto count_le = [&](int t, int buf) {
    int c = 0;
#pragma unroll
    for (int e = 0; e < PER; ++e)
      if (e * kBoundThreads < end) c += v[e] <= t ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) wcnt[buf][warp] = c;
    __syncthreads();
    return __reduce_add_sync(0xffffffffu, lane < W ? wcnt[buf][lane] : 0);
  };
  mn = __reduce_min_sync(0xffffffffu, mn);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) {
    wcnt[0][warp] = mn;
    wcnt[1][warp] = mx;
  }
  __syncthreads();
  mn = __reduce_min_sync(0xffffffffu, lane < W ? wcnt[0][lane] : kEmptyStep);
  mx = __reduce_max_sync(0xffffffffu, lane < W ? wcnt[1][lane] : 0);
  __syncthreads();
  int T = kEmptyStep - 1;  // fewer than k candidates: all of them
  if (mn <= mx && count_le(mx, 0) >= k) {  // block-uniform
    T = mx;
    int a = mn - 1;  // count(<= a) < k <= count(<= T)
    for (int it = 1; T - a > 1; ++it) {
      const int mid = (a + T) >> 1;
      if (count_le(mid, it & 1) >= k) T = mid;
      else a = mid;
    }
  }
  // the candidates whose lower bound reaches T, in any order
  uint64_t* dst = kept + (int64_t)qi * kKeep;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    if (e * kBoundThreads >= end) continue;
    const int i = e * kBoundThreads + tid;
    const bool in = i < end && (int)(bnd[i] >> 16) <= T;
    const unsigned mk = __ballot_sync(0xffffffffu, in);
    int base = 0;
    if (lane == 0 && mk) base = atomicAdd(&total, __popc(mk));
    base = __shfl_sync(0xffffffffu, base, 0) + __popc(mk & ((1u << lane) - 1u));
    if (in && base < kKeep)
      dst[base] = LIST ? make_key(0.0f, list[(int64_t)qi * list_cap + i]) : cand[(int64_t)qi * C + i];
  }
  __syncthreads();
  const int got = total;
  if (got > kKeep) {  // scored in full: no place here
    for (int i = tid; i < kKeep; i += kBoundThreads) dst[i] = kEmptyKey;
    if (tid == 0) listed[1 + atomicAdd(listed, 1)] = qi;
  } else {
    for (int i = got + tid; i < kKeep; i += kBoundThreads) dst[i] = kEmptyKey;
  }
}

}  // namespace

namespace {

template <int DIST, int C, bool LIST>
void launch_bounds(const uint64_t* cand, const int* list, int list_cap, const int* ccnt, const uint8_t* rows,
                   const float2* tails, int pitch, float scale, int64_t n, int d, const float* q, int nq, int k,
                   uint64_t* kept, int* listed, cudaStream_t s) {
  ProfScope _ps("rerank_bounds", s);
  constexpr int smem = C * (int)sizeof(uint32_t);
  auto kern = bounds_kernel<DIST, C, LIST>;
  raise_smem_limit(kern, smem);
  launch_next(kern, nq, kBoundThreads, smem, s, cand, list, list_cap, ccnt, rows, tails, pitch, scale, n, d, q, k,
              kept, listed);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

void derive_jaccard(Index& I, cudaStream_t s) {
  float lo, hi;
  if (!base_range(I.x.ptr, I.n * I.d, &lo, &hi, s)) return;  // no such bounds: every candidate is scored
  I.xq8.alloc((size_t)I.n * jaccard_pitch(I.d), s);
  I.xq8_scale = 255.0f / hi;
  quantise_rows_kernel<<<(int)std::min<int64_t>((I.n * 32 + 255) / 256, (int64_t)num_sms() * 16), 256, 0, s>>>(
      I.x.ptr, I.n, I.d, jaccard_pitch(I.d), I.xq8_scale, I.xq8.ptr);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

void derive_angular(Index& I, cudaStream_t s) {
  const int pitch = angular_pitch(I.d);
  DevBuf<unsigned> stat(1 + kProbeRows, s);  // a row without bounds; the probe's counts
  LSHG_CUDA(cudaMemsetAsync(stat.ptr, 0, stat.bytes(), s));
  I.xq8.alloc((size_t)I.n * pitch, s);
  I.xq8_tail.alloc((size_t)I.n, s);
  quantise_angular_kernel<<<(int)std::min<int64_t>((I.n * 32 + 255) / 256, (int64_t)num_sms() * 16), 256, 0, s>>>(
      I.x.ptr, I.n, I.d, pitch, reinterpret_cast<int8_t*>(I.xq8.ptr), I.xq8_tail.ptr, stat.ptr);
  count_launch();
  LSHG_CHECK_LAUNCH();
  const int points = (int)std::min<int64_t>(kProbePoints, I.n);
  near_rows_kernel<<<dim3(kProbeRows, ceil_div(points, 256)), 256, 0, s>>>(I.xq8.ptr, I.xq8_tail.ptr, I.n, pitch, points,
                                                                          stat.ptr + 1);
  count_launch();
  LSHG_CHECK_LAUNCH();
  unsigned h[1 + kProbeRows];
  LSHG_CUDA(cudaMemcpyAsync(h, stat.ptr, sizeof(h), cudaMemcpyDeviceToHost, s));
  LSHG_CUDA(cudaStreamSynchronize(s));
  // A row without bounds, or a base whose rows mostly have more points within the codes' resolution
  // than a query may keep: every candidate is scored.  Bounds on top of that took a fifth more
  // (300,000 x 128, 32 tables, clusters of 1,500 within 0.013, 2,000 queries: 607 us without, 727
  // with).
  int crowded = 0;
  for (int b = 0; b < kProbeRows; ++b) crowded += (int64_t)h[1 + b] * I.n > (int64_t)kKeep * points ? 1 : 0;
  if (h[0] || 2 * crowded > kProbeRows) {
    I.xq8.release();
    I.xq8_tail.release();
  }
}

}  // namespace

bool base_range(const float* x, int64_t total, float* lo, float* hi, cudaStream_t s) {
  DevBuf<unsigned> stat(3, s);
  LSHG_CUDA(cudaMemsetAsync(stat.ptr, 0, stat.bytes(), s));
  base_range_kernel<<<(int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, (int64_t)num_sms() * 8)), 256, 0,
                      s>>>(x, total, stat.ptr);
  count_launch();
  LSHG_CHECK_LAUNCH();
  unsigned h[3];
  LSHG_CUDA(cudaMemcpyAsync(h, stat.ptr, sizeof(h), cudaMemcpyDeviceToHost, s));
  LSHG_CUDA(cudaStreamSynchronize(s));
  h[2] = ~h[2];
  memcpy(hi, &h[0], 4);
  memcpy(lo, &h[2], 4);
  return !h[1] && *hi > 1e-18f;
}

void derive_rerank_bounds(Index& I, cudaStream_t s) {
  const bool linear = I.p.framework == 0 && I.C >= 1024;
  const bool tables = I.p.framework == 1 && !(I.p.runWithSketchedData && I.sk_kind) && I.d % 4 == 0;
  try {
    if (linear && I.dist == DIST_JACCARD && (I.sk_kind == 4 || I.sk_kind == 5 || I.sk_kind == 10) &&
        I.d <= kMaxJaccardDim)
      derive_jaccard(I, s);
    else if (I.dist == DIST_ANGULAR && I.d <= kMaxAngularDim &&
             ((linear && (I.sk_kind == 3 || I.sk_kind == 6)) || tables))
      derive_angular(I, s);
  } catch (const Error& e) {  // no room for the copy: every candidate is scored
    if (e.status != LSHG_ERR_OUT_OF_MEMORY) throw;
    cudaGetLastError();
    I.xq8.release();
    I.xq8_tail.release();
  }
}

bool rerank_by_bounds(Index& I, const uint64_t* cand, int nq, int C, const float* q, const float* qnorm, int k,
                      lshg_point* out, cudaStream_t s) {
  if (!I.xq8.ptr || k > 128 || (C != 1024 && C != 2048 && C != 4096) || I.p.opt.fp64_recheck > 0 ||
      (int64_t)nq * C < kBoundsMinCandidates)
    return false;
  if (const char* e = getenv("LSHG_TEST_ROW_WAIT_STALL"); e && e[0] == '1') return false;  // a hook of the full re-rank
  DevBuf<uint64_t> kept;
  DevBuf<int> listed;
  try {
    kept.alloc((size_t)nq * kKeep, s);
    listed.alloc((size_t)nq + 1, s);
  } catch (const Error& e) {
    if (e.status != LSHG_ERR_OUT_OF_MEMORY) throw;
    cudaGetLastError();
    return false;
  }
  LSHG_CUDA(cudaMemsetAsync(listed.ptr, 0, sizeof(int), s));
#define LSHG_RB(DV, CV, PITCH)                                                                                      \
  launch_bounds<DV, CV, false>(cand, nullptr, 0, nullptr, I.xq8.ptr, I.xq8_tail.ptr, PITCH, I.xq8_scale, I.n, I.d, q, \
                               nq, k, kept.ptr, listed.ptr, s)
  if (I.dist == DIST_JACCARD) {
    if (C == 1024) LSHG_RB(DIST_JACCARD, 1024, jaccard_pitch(I.d));
    else if (C == 2048) LSHG_RB(DIST_JACCARD, 2048, jaccard_pitch(I.d));
    else LSHG_RB(DIST_JACCARD, 4096, jaccard_pitch(I.d));
  } else {
    if (C == 1024) LSHG_RB(DIST_ANGULAR, 1024, angular_pitch(I.d));
    else if (C == 2048) LSHG_RB(DIST_ANGULAR, 2048, angular_pitch(I.d));
    else LSHG_RB(DIST_ANGULAR, 4096, angular_pitch(I.d));
  }
#undef LSHG_RB
  launch_rerank(kept.ptr, nq, kKeep, I.x.ptr, I.n, I.d, I.xnorm.ptr, q, qnorm, I.dist, k, out, s, I.error_word(s));
  launch_rerank_listed(cand, C, I.x.ptr, I.n, I.d, I.xnorm.ptr, q, qnorm, I.dist, listed.ptr, nq, k, out, s,
                       I.error_word(s));
  return true;
}

void launch_list_bounds(const int* list, int cap, const int* ccnt, const uint8_t* rows, const float2* tails, int64_t n,
                        int d, const float* q, int nq, int k, uint64_t* kept, int* listed, cudaStream_t s) {
  LSHG_REQUIRE(cap <= kListBounds && d <= kMaxAngularDim, "list bounds: list or rows too long");
  launch_bounds<DIST_ANGULAR, kListBounds, true>(nullptr, list, cap, ccnt, rows, tails, angular_pitch(d), 1.0f, n, d, q,
                                                 nq, k, kept, listed, s);
}

}  // namespace lshg
