// Generalized-Jaccard re-rank of long candidate lists through quantised rows: which of a query's
// C candidates can be in its top-k is decided from 8-bit copies of the rows and bounds on what
// they hide, and only those are scored from the FP32 rows (launch_rerank), so the results are
// those of scoring every candidate (rerank.cu, restating candidateSetScan,
// candidateSetScanner.cuh:10-32).
//
// A row x >= 0 is kept as u = rint(s x) (s = 255 / the base's largest value, one scale for all
// rows) with its sum S(x) and its residual e(x) = sum |x - u / s|.  For a query quantised the same
// way, M = sum min(u_q, u_x) / s is an integer sum, and
//     |sum min(q, x) - M| <= sum max(|q - u_q / s|, |x - u_x / s|) <= e(q) + e(x) = E.
// sum max = S(q) + S(x) - sum min, so the similarity A / (S - A) rises with A = sum min and
// M - E, M + E bound the distance from above and below; delta covers the FP32 arithmetic of
// the reference's sums and quotient ((2 d + 3) 2^-24, fp64_band) and of this kernel's (a quotient
// within 2^-21, sums within d 2^-24).  With T
// the k-th smallest upper bound of the list, every candidate of the top-k has a lower bound
// of at most T.  Lists with more than kKeep such candidates, and queries with a negative or
// non-finite value, are scored in full (from a list on the device).
//
// A row of 100 dimensions is 128 bytes here (with its S and e) against 400, and about 60 of
// 4,096 candidates are left at k = 32.  Eight lanes read a row, 16 bytes each.  The kernel is
// bounded by its instructions (minima as packed 16-bit pairs: 1.15 ms, 28 a row).  Measured (10,000 queries, C = 4,096, 500k x 100): partition,
// gather of every row and select 2.77 ms; this way 0.74 + 0.15 ms.
#include <algorithm>

#include "common.cuh"
#include "index.h"
#include "kernels.h"
#include "launch_count.h"
#include "profile.h"

namespace lshg {

namespace {

constexpr int kMaxBoundsDim = 120;  // 8 bytes of a 128-byte row hold S and e
constexpr int kKeep = 256;          // candidates a query passed on
constexpr int kBoundThreads = 256;
constexpr int kMaxBoundsC = 4096;

int bounds_pitch(int d) { return (d + 8 + 31) / 32 * 32; }

// stat[0]: bits of the largest value; stat[1]: 1 when a value is negative or not finite.
__global__ void base_max_kernel(const float* __restrict__ x, int64_t total, unsigned* stat) {
  float m = 0.0f;
  bool bad = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = x[i];
    if (v >= 0.0f && v <= 1e18f) m = fmaxf(m, v);
    else bad = true;
  }
  const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  const bool wb = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(stat, w);
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

// One block a query; see the header.  kept: [nq][kKeep] keys (ids of the candidates that can be in
// the top-k, then empty keys); listed: count, then the queries to score in full.
template <int C>
__global__ void __launch_bounds__(kBoundThreads) jaccard_bounds_kernel(
    const uint64_t* __restrict__ cand, const uint8_t* __restrict__ rows, int pitch, float s, int64_t n, int d,
    const float* __restrict__ q, int k, uint64_t* __restrict__ kept, int* __restrict__ listed) {
  constexpr int W = kBoundThreads / 32, PER = C / kBoundThreads;
  __shared__ float lo[C], hi[C];
  __shared__ int wcnt[2][W];
  __shared__ float wmm[2][W];
  __shared__ int total;
  const int qi = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float inv = 1.0f / s;
  // the query: this lane's 16 codes as 16-bit pairs, sum and residual (every warp computes them)
  const float* qr = q + (int64_t)qi * d;
  float sq = 0.0f, eq = 0.0f;
  bool bad = false;
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
  if (__any_sync(0xffffffffu, bad)) {  // the same in every warp
    for (int i = tid; i < kKeep; i += kBoundThreads) kept[(int64_t)qi * kKeep + i] = kEmptyKey;
    if (tid == 0) listed[1 + atomicAdd(listed, 1)] = qi;
    return;
  }
  const int part = lane & 7, parts = pitch / 16;  // 16-byte part of a row
  unsigned qw[4];                                 // this lane's 16 query codes
  int uq = 0;                                     // and the sum of all the query's
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    qw[e] = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = part * 16 + 4 * e + j;
      if (c < d) {  // codes past d: 0, as in the rows
        const unsigned u = quantise(qr[c], s);
        qw[e] |= u << (8 * j);
        uq += (int)u;
      }
    }
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) uq += __shfl_xor_sync(0xffffffffu, uq, o);
  const float delta = (2.0f * d + 3.0f) * 1.2e-7f + 1e-6f;
  if (tid == 0) total = 0;
  // Bounds: a warp takes 16 candidates at a time, 8 lanes a row and four rows a load.  The sum of
  // minima is (sum u_q + sum u_x - sum |u_q - u_x|) / 2, and four bytes' absolute differences are
  // one instruction.  The four loads' sums are reduced together (four shuffles), which leaves
  // row `t` of its group in the lanes with part >> 1 == t.
  constexpr int U = 4;
  const int grp = lane >> 3, own = part >> 1;
  const bool tail = part == parts - 1;
  for (int c0 = warp * 4 * U; c0 < C; c0 += W * 4 * U) {
    int id[U];
    uint4 r[U];
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const uint64_t key = cand[(int64_t)qi * C + c0 + 4 * t + grp];
      id[t] = key == kEmptyKey ? -1 : key_id(key);
      if (id[t] >= n) id[t] = -1;
    }
#pragma unroll
    for (int t = 0; t < U; ++t) {
      r[t] = make_uint4(0, 0, 0, 0);
      if (id[t] >= 0 && part < parts)
        r[t] = __ldg(reinterpret_cast<const uint4*>(rows + (int64_t)id[t] * pitch) + part);
    }
    const int oid = own == 0 ? id[0] : own == 1 ? id[1] : own == 2 ? id[2] : id[3];
    uint2 rt = make_uint2(0, 0);  // the own row's last 8 bytes
    if (oid >= 0) rt = __ldg(reinterpret_cast<const uint2*>(rows + (int64_t)oid * pitch + pitch - 8));
    unsigned sad[U];
#pragma unroll
    for (int t = 0; t < U; ++t)
      sad[t] = __vsadu4(r[t].x, qw[0]) + __vsadu4(r[t].y, qw[1]) + __vsadu4(tail ? 0u : r[t].z, qw[2]) +
               __vsadu4(tail ? 0u : r[t].w, qw[3]);
    // lanes with bit 2 of the part keep loads 2 and 3, then bit 1 the odd one, then bit 0 is summed
    const bool up = part & 4, odd = part & 2;
    unsigned x0 = up ? sad[2] : sad[0], x1 = up ? sad[3] : sad[1];
    x0 += __shfl_xor_sync(0xffffffffu, up ? sad[0] : sad[2], 4);
    x1 += __shfl_xor_sync(0xffffffffu, up ? sad[1] : sad[3], 4);
    unsigned x = odd ? x1 : x0;
    x += __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    if (!(part & 1)) {
      const float sx = __uint_as_float(rt.x), ex = __uint_as_float(rt.y & 0xffff0000u);
      const float S = sq + sx, M = (float)((uq + (int)(rt.y & 0xffffu) - (int)x) >> 1) * inv;
      const float E = (eq + ex) * 1.0001f + S * 2e-5f;
      const float ah = fminf(M + E, 0.5f * S), al = fmaxf(M - E, 0.0f);
      float l = 1.0f - __fdividef(ah, S - ah) - delta, h = 1.0f - __fdividef(al, S - al) + delta;
      if (!(S > 1e-6f && S < 1e30f)) {  // no bound: always scored
        l = -INFINITY;
        h = INFINITY;
      }
      if (oid < 0) l = h = INFINITY;  // an empty place
      lo[c0 + 4 * own + grp] = l;
      hi[c0 + 4 * own + grp] = h;
    }
  }
  __syncthreads();
  // T: an upper bound of the k-th smallest upper bound, by bisection (count(<= T) >= k)
  float v[PER];
  float mn = INFINITY, mx = -INFINITY;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    v[e] = hi[e * kBoundThreads + tid];
    if (v[e] < INFINITY) {
      mn = fminf(mn, v[e]);
      mx = fmaxf(mx, v[e]);
    }
  }
  auto count_le = [&](float t, int buf) {
    int c = 0;
#pragma unroll
    for (int e = 0; e < PER; ++e) c += v[e] <= t ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) wcnt[buf][warp] = c;
    __syncthreads();
    int sum = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) sum += wcnt[buf][w];
    return sum;
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (lane == 0) {
    wmm[0][warp] = mn;
    wmm[1][warp] = mx;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < W; ++w) {
    mn = fminf(mn, wmm[0][w]);
    mx = fmaxf(mx, wmm[1][w]);
  }
  float T = INFINITY;
  if (mn <= mx && count_le(mx, 0) >= k) {  // block-uniform
    T = mx;
    float a = mn;
    for (int it = 1; it <= 12 && a < T; ++it) {
      const float mid = a + 0.5f * (T - a);
      if (!(mid > a && mid < T)) break;
      if (count_le(mid, it & 1) >= k) T = mid;
      else a = mid;
    }
  }
  // the candidates whose lower bound reaches T, in any order
  uint64_t* dst = kept + (int64_t)qi * kKeep;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int i = e * kBoundThreads + tid;
    const bool in = lo[i] <= T && lo[i] < INFINITY;
    const unsigned mk = __ballot_sync(0xffffffffu, in);
    int base = 0;
    if (lane == 0 && mk) base = atomicAdd(&total, __popc(mk));
    base = __shfl_sync(0xffffffffu, base, 0) + __popc(mk & ((1u << lane) - 1u));
    if (in && base < kKeep) dst[base] = cand[(int64_t)qi * C + i];
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

void derive_rerank_bounds(Index& I, cudaStream_t s) {
  if (I.p.framework != 0 || I.dist != DIST_JACCARD || !(I.sk_kind == 4 || I.sk_kind == 5 || I.sk_kind == 10) ||
      I.d > kMaxBoundsDim || I.C < 1024)
    return;
  DevBuf<unsigned> stat(2, s);
  LSHG_CUDA(cudaMemsetAsync(stat.ptr, 0, stat.bytes(), s));
  const int64_t total = I.n * I.d;
  base_max_kernel<<<(int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, (int64_t)num_sms() * 8)), 256, 0,
                    s>>>(I.x.ptr, total, stat.ptr);
  count_launch();
  LSHG_CHECK_LAUNCH();
  unsigned h[2];
  LSHG_CUDA(cudaMemcpyAsync(h, stat.ptr, sizeof(h), cudaMemcpyDeviceToHost, s));
  LSHG_CUDA(cudaStreamSynchronize(s));
  float mx;
  memcpy(&mx, &h[0], 4);
  if (h[1] || !(mx > 1e-18f)) return;  // no such bounds: every candidate is scored
  const int pitch = bounds_pitch(I.d);
  try {
    I.xq8.alloc((size_t)I.n * pitch, s);
  } catch (const Error&) {  // no room for the copy: every candidate is scored
    cudaGetLastError();
    return;
  }
  I.xq8_scale = 255.0f / mx;
  quantise_rows_kernel<<<(int)std::min<int64_t>((I.n * 32 + 255) / 256, (int64_t)num_sms() * 16), 256, 0, s>>>(
      I.x.ptr, I.n, I.d, pitch, I.xq8_scale, I.xq8.ptr);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

bool rerank_by_bounds(Index& I, const uint64_t* cand, int nq, int C, const float* q, int k, lshg_point* out,
                      cudaStream_t s) {
  if (!I.xq8.ptr || k > 128 || (C != 1024 && C != 2048 && C != 4096) || I.p.opt.fp64_recheck > 0) return false;
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
  const int pitch = bounds_pitch(I.d);
  {
    ProfScope _ps("rerank_bounds", s);
    if (C == 1024)
      jaccard_bounds_kernel<1024><<<nq, kBoundThreads, 0, s>>>(cand, I.xq8.ptr, pitch, I.xq8_scale, I.n, I.d, q, k,
                                                               kept.ptr, listed.ptr);
    else if (C == 2048)
      jaccard_bounds_kernel<2048><<<nq, kBoundThreads, 0, s>>>(cand, I.xq8.ptr, pitch, I.xq8_scale, I.n, I.d, q, k,
                                                               kept.ptr, listed.ptr);
    else
      jaccard_bounds_kernel<4096><<<nq, kBoundThreads, 0, s>>>(cand, I.xq8.ptr, pitch, I.xq8_scale, I.n, I.d, q, k,
                                                               kept.ptr, listed.ptr);
    count_launch();
    LSHG_CHECK_LAUNCH();
  }
  launch_rerank(kept.ptr, nq, kKeep, I.x.ptr, I.n, I.d, nullptr, q, nullptr, DIST_JACCARD, k, out, s, I.error_word(s));
  launch_rerank_listed(cand, C, I.x.ptr, I.n, I.d, q, listed.ptr, nq, k, out, s);
  return true;
}

}  // namespace lshg
