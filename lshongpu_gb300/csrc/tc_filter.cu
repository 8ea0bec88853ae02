// Threshold-filter tensor-core scan: the kernels behind implementation 8's main path.
//
// Selecting the top-CT cosine scores of every query out of a Q x N BF16 GEMM is done in
// two GEMM passes that share one persistent tcgen05 pipeline (tc_filter_kernel):
//
//   pass 0 (MODE_GROUPMAX) runs on a strided subsample of the base tiles (every S-th) and
//     writes, per query row, the maximum score of every GW-column group of every sampled
//     tile.  Each group maximum is the score of a real base point, so the CT-th largest
//     of them, tau[q] (tau_select_kernel), is a lower bound of the query's true CT-th best
//     score: every point of the exact top-CT has score >= tau[q].
//   pass 1 (MODE_FILTER) runs on the whole base.  The epilogue compares each score with
//     its row's tau; the (rare) survivors are staged per row in shared memory and moved
//     to the query's candidate array in global memory with one atomicAdd a batch (at the
//     end of each work unit, or when the 16-entry staging is full).  There is no per-row
//     selection state on chip, so the common case is a 64-wide maximum and a warp vote.
//
// cand_select_kernel then sorts each query's survivors and keeps the first CT keys
// (score descending, ties by lower id) -- exactly the top-CT by tensor-core score.  A query
// with more survivors than the candidate array holds (possible only with massive ties,
// e.g. duplicated points or a zero query) is listed for the exact per-row list kernel in
// tc_scan.cu, which runs on the device-side list without a host round trip.
//
// Work decomposition of tc_filter_kernel: persistent, one CTA per SM, in clusters of CL = 2
// CTAs (1 for batches of one query tile).  A unit is (CL query tiles, chunk of CH consecutive
// base positions); units are numbered chunk-major and dealt round-robin to the clusters.  At
// any moment the clusters therefore work on the same one or two chunks for different query
// tiles, so each base tile is read from HBM about once and served from L2.  The two CTAs of a
// cluster are an MMA pair (tcgen05 cta_group::2): each holds a query tile of its own and half
// of every base tile, and the even one issues the MMAs of both.  A CTA on its own would read
// 84 KB of operands from shared memory and write 56 KB of base tile into it for the 896
// cycles of MMA of a 128 x 256 tile at d = 100 -- 1,094 cycles at 128 bytes a cycle; in a
// pair it is 56 + 28 KB.  A CTA keeps its query tile, and its staged survivors, when its next
// unit has the same one.
//
// Tiles are 128 queries x 256 base points (tcgen05.mma M = 128, N = 256).  A row is KC chunks
// of 128 bytes -- 64 BF16 columns (KC = 1 for d <= 64, else 2) or 128 E4M3 ones -- and a ring
// stage one chunk of a base tile (32 KB, or a pair's 16 KB each), given back as soon as its K steps are done.  Warp
// roles (640 threads): warp 0 TMA producer, warp 1 MMA issuer, warp 2 TMEM allocator (2
// accumulators x 256 columns = 512), warp 3 idle, warps 4-19 the epilogue: warpgroup g (warps
// 4+4g .. 7+4g) reads TMEM columns [64g, 64g+64) of every accumulator, thread (warp & 3) *
// 32 + lane owns query row = TMEM lane.  Every mbarrier wait is bounded; a CTA that times
// out raises the error flag, drains its own copies and MMAs, frees TMEM and returns; the
// CTAs of a cluster leave together.
//
// Measured (10,000 queries, 1.2M x 100): prepass 128 -> 104 us, filter pass 1.90 -> 1.73 ms.
// Copies and MMAs alone are MMA-bound in a pair (1.13 ms of MMAs; 1.40 ms in single CTAs);
// the filter pass is bounded by its epilogue: reading a tile's scores, their maxima and, in
// 42% of a warp's pieces, a survivor.
#include "index.h"
#include "launch_count.h"
#include "launch_next.cuh"
#include "profile.h"
#include "select.cuh"
#include "tc_filter.h"
#include "tc_ptx.cuh"

namespace lshg {
namespace tc {

namespace {

constexpr int F_THREADS = 640;
constexpr int TN = FILTER_TN;        // base points a tile = UMMA N
constexpr int F_CHUNK = 128;         // bytes of a row in one K chunk (one 128-byte swizzle row)
constexpr int F_A_CHUNK = BM * F_CHUNK;  // 16 KB of a query tile
constexpr int F_NACC = 2;            // TMEM accumulators of TN columns
constexpr int F_TMEM_COLS = F_NACC * TN;  // 512 = all of TMEM (one CTA per SM)
constexpr int F_EPI_WARPS = 16;      // four warpgroups, one 64-column piece each
constexpr int kTauRegs = 80;  // group maxima a lane holds in the register threshold select
constexpr int kTauBlockRegs = 24;  // and a thread of the block form: 6,144 maxima
// and its smaller form, 1,408 maxima (59 registers, four blocks an SM).  One query on 1.2M points, the
// batch: 87 us with 44, 89 with 40, 90 with 48.
constexpr int kTauRegsFew = 44;

// Shared-memory layout of a CTA in a cluster of CL: CL buffers of its query tile (rows of KC
// chunks; a pair loads its next query tiles while these are in use, a CTA alone has but one
// query tile), the ring of its shares of base chunks, and the survivor staging (SBUF entries
// of (score, id) a row and warpgroup).
template <int KC, int CL>
struct FLayout {
  static constexpr int AB = CL;
  static constexpr int A_BYTES = KC * F_A_CHUNK;
  static constexpr int B_BYTES = TN / CL * F_CHUNK;  // 32 KB, or 16 KB of a pair's
  static constexpr int STAGES = CL == 2 ? 6 : 4;
  static constexpr int SBUF = 16;
  static constexpr int A_OFF = 0;
  static constexpr int B_OFF = AB * A_BYTES;
  static constexpr int S_OFF = B_OFF + STAGES * B_BYTES;  // [4][SBUF][BM] entries of 8 bytes
  static constexpr int BAR_OFF = S_OFF + 4 * SBUF * BM * 8;
  static constexpr int SMEM = BAR_OFF + 256 + 1024;  // + barriers + 1 KB alignment slack
  static_assert(SMEM <= 232448, "shared memory per CTA");
  static_assert(8 * (2 * STAGES + 2 * AB + 2 * F_NACC + 1) + 8 <= 256, "barrier area");
};

struct FilterArgs {
  int nq;
  int64_t n;
  int QT;        // query tiles
  int QP;        // groups of CL of them
  int NP;        // base positions scanned (tiles NP of them, base tile = p * dstride)
  int dstride;
  int CH;        // positions per unit
  int NCH;       // chunks = ceil(NP / CH)
  float* gmax;   // MODE_GROUPMAX: [nq][M] group maxima
  int M;
  const float* tau;  // MODE_FILTER: per-query threshold (nullptr = keep everything)
  int* cnt;          // survivors per query
  uint64_t* cand;    // [nq][cap] survivor keys
  int cap;
  int ksteps;    // MMA K steps covering the data dimension (K = 16 BF16 or 32 E4M3 a step)
  int hi_bytes;  // bytes a row loaded of the second chunk of a base tile (what its K steps read)
  int* err;
};

// Move a row's staged survivors to the query's candidate array: one atomicAdd reserves the
// slots.
__device__ __forceinline__ void f_flush(int* cnt, uint64_t* dst, int cap, uint32_t at0, uint32_t at) {
  if (at > at0) {
    int pos = atomicAdd(cnt, (int)((at - at0) / (BM * 8u)));
#pragma unroll 1
    for (uint32_t e = at0; e < at; e += BM * 8u, ++pos) {
      uint32_t v, id;
      asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v), "=r"(id) : "r"(e));
      if (pos < cap) dst[pos] = make_key(-__uint_as_float(v), (int)id);
    }
  }
}

// F8: E4M3 operands (kind::f8f6f4), one chunk; otherwise BF16 in KC chunks.  mapB's boxes
// hold a CTA's share (TN / CL rows) of a chunk, mapBhi's of the trimmed second chunk.
template <int MODE, int GW, bool F8, int KC, int CL>
__global__ void __launch_bounds__(F_THREADS, 1)
    tc_filter_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                     const __grid_constant__ CUtensorMap mapBhi, const FilterArgs a) {
  grid_ready();
  using LY = FLayout<KC, CL>;
  constexpr int SBUF = LY::SBUF, F_STAGES = LY::STAGES, AB = LY::AB;
  static_assert(MODE == MODE_GROUPMAX || GW == 64, "the filter reads whole 64-column pieces");
  static_assert(GW == 64 || GW == 8, "group width");
  static_assert(!F8 || KC == 1, "an E4M3 row is one chunk");
  const int U = a.NCH * a.QP;
  const int cid = blockIdx.x / CL, ncl = gridDim.x / CL;  // cluster, clusters
  if (cid >= U) return;  // no unit for this cluster: leave before any barrier or TMEM use

  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t s0 = smem_u32(sm);
  const uint32_t bar0 = s0 + LY::BAR_OFF;
  auto FULL = [&](int s) { return bar0 + 8u * s; };
  auto EMPTY = [&](int s) { return bar0 + 8u * (F_STAGES + s); };
  auto A_FULL = [&](int s) { return bar0 + 8u * (2 * F_STAGES + s); };
  auto A_EMPTY = [&](int s) { return bar0 + 8u * (2 * F_STAGES + AB + s); };
  auto ACC_FULL = [&](int b) { return bar0 + 8u * (2 * F_STAGES + 2 * AB + b); };
  auto ACC_EMPTY = [&](int b) { return bar0 + 8u * (2 * F_STAGES + 2 * AB + F_NACC + b); };
  const uint32_t DONE = bar0 + 8u * (2 * F_STAGES + 2 * AB + 2 * F_NACC);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + LY::BAR_OFF + 8 * (2 * F_STAGES + 2 * AB + 2 * F_NACC + 1));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform for the compiler too
  const int lane = threadIdx.x & 31;
  const int rank = CL > 1 ? (int)cluster_rank() : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < F_STAGES; ++s) {
      mbar_init(FULL(s), 1);
      mbar_init(EMPTY(s), 1);
    }
    for (int s = 0; s < AB; ++s) {
      mbar_init(A_FULL(s), 1);
      mbar_init(A_EMPTY(s), 1);
    }
    for (int b = 0; b < F_NACC; ++b) {
      mbar_init(ACC_FULL(b), 1);
      mbar_init(ACC_EMPTY(b), CL * F_EPI_WARPS);  // a pair's even CTA waits for both
    }
    mbar_init(DONE, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) tmem_alloc<CL>(smem_u32(tmem_slot), F_TMEM_COLS);
  tc_fence_before();
  if (CL > 1) cluster_sync();  // the peer's barriers are initialised before anything arrives on them
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      // a pair's bytes are counted on its even CTA's barriers, where the MMAs are issued
      auto load = [&](uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
        if (CL > 1) tma_load_2d_pair(dst, map, x, y, cluster_addr(bar, 0));
        else tma_load_2d(dst, map, x, y, bar);
      };
      int it = 0, na = 0;  // base chunks and query tiles issued
      int have = -1;       // group whose query tile was issued last
      bool ok = true;
      for (int u = cid; u < U && ok; u += ncl) {
        const int qp = u % a.QP, c = u / a.QP;
        const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
        if (qp != have) {  // (a tile past the last one, where the tiles do not fill the cluster, reads as zeros)
          const int ab = na % AB;
          if (!mbar_wait(A_EMPTY(ab), ((na / AB) & 1) ^ 1, abort_flag)) break;
          if (rank == 0) mbar_expect_tx(A_FULL(ab), CL * LY::A_BYTES);
#pragma unroll
          for (int kc = 0; kc < KC; ++kc)
            load(s0 + LY::A_OFF + ab * LY::A_BYTES + kc * F_A_CHUNK, &mapA, kc * KHALF, (CL * qp + rank) * BM,
                 A_FULL(ab));
          ++na;
          have = qp;
        }
        for (int p = p0; p < p1 && ok; ++p) {
          const int row = p * a.dstride * TN + rank * (TN / CL);  // this CTA's share of the tile
#pragma unroll
          for (int kc = 0; kc < KC; ++kc) {
            const int st = it % F_STAGES, rd = it / F_STAGES;
            if (!mbar_wait(EMPTY(st), (rd & 1) ^ 1, abort_flag)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(FULL(st), TN * (kc == 0 ? F_CHUNK : a.hi_bytes));
            load(s0 + LY::B_OFF + st * LY::B_BYTES, kc == 0 ? &mapB : &mapBhi, kc * KHALF, row, FULL(st));
            ++it;
          }
        }
      }
      // drain: every copy has landed and every stage has been given back before the CTA may
      // exit (a pair's odd CTA sees its copies' end only by the stages that come back)
      for (int j = max(0, it - F_STAGES); j < it; ++j) {
        if (rank == 0) mbar_wait(FULL(j % F_STAGES), (j / F_STAGES) & 1, abort_flag, true);
        mbar_wait(EMPTY(j % F_STAGES), (j / F_STAGES) & 1, abort_flag, true);
      }
      if (rank == 0)
        for (int j = max(0, na - AB); j < na; ++j) mbar_wait(A_FULL(j % AB), (j / AB) & 1, abort_flag, true);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (a pair's: its even CTA) ----------------
    const uint32_t leader = elect_one();  // the warp stays converged (see elect_one)
    constexpr uint32_t idesc = F8 ? idesc_e4m3(CL * BM, TN) : idesc_bf16(CL * BM, TN);
    auto commit = [&](uint32_t bar) {
      if (CL > 1) umma_commit_pair(bar, leader);
      else umma_commit(bar, leader);
    };
    // A tile's MMAs take 896 cycles at d = 100 and this warp issues nothing else meanwhile, so
    // its own time a tile has to stay below that: running stage and parity instead of
    // divisions, descriptors by 32-bit additions.
    const uint32_t a_lo0 = smem_desc_lo(s0 + LY::A_OFF), b_lo0 = smem_desc_lo(s0 + LY::B_OFF);
    int st = 0, na = 0, b = 0;
    uint32_t ph = 0, acc_ph = 1;
    int have = -1;
    bool ok = rank == 0;
    for (int u = cid; u < U && ok; u += ncl) {
      const int qp = u % a.QP, c = u / a.QP;
      const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
      if (qp != have) {
        if (!mbar_wait_warp(A_FULL(na % AB), (na / AB) & 1, abort_flag)) break;
        tc_fence_after();
        ++na;
        have = qp;
      }
      const int ab = (na - 1) % AB;
      const uint32_t a_lo = a_lo0 + (uint32_t)ab * (LY::A_BYTES >> 4);
      for (int p = p0; p < p1; ++p) {
        if (!mbar_wait_warp(ACC_EMPTY(b), acc_ph, abort_flag)) { ok = false; break; }
        const uint32_t d_tmem = tmem + (uint32_t)(b * TN);
#pragma unroll
        for (int kc = 0; kc < KC; ++kc) {
          if (!mbar_wait_warp(FULL(st), ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t b_lo = b_lo0 + (uint32_t)st * (LY::B_BYTES >> 4);
          // rows are zero past the data dimension: steps beyond it would add exact zeros
#pragma unroll
          for (int kk = 0; kk < F_CHUNK / 32; ++kk) {  // 32 bytes a step
            const uint64_t ad = smem_desc_of(a_lo + kc * (F_A_CHUNK >> 4) + 2 * kk), bd = smem_desc_of(b_lo + 2 * kk);
            if (4 * kc + kk >= a.ksteps) continue;
            if (F8) umma_e4m3<CL>(d_tmem, ad, bd, idesc, (kc > 0 || kk > 0) ? 1u : 0u, leader);
            else umma_bf16<CL>(d_tmem, ad, bd, idesc, (kc > 0 || kk > 0) ? 1u : 0u, leader);
          }
          commit(EMPTY(st));
          if (++st == F_STAGES) {
            st = 0;
            ph ^= 1u;
          }
        }
        if (!ok) break;
        commit(ACC_FULL(b));
        b ^= 1;
        if (b == 0) acc_ph ^= 1u;
      }
      // the query tile is free once this unit's MMAs complete
      if (u + ncl < U && (u + ncl) % a.QP != qp) commit(A_EMPTY(ab));
    }
    // drain: all issued MMAs complete before TMEM is released
    if (rank == 0) commit(DONE);
    mbar_wait(DONE, 0, abort_flag, true);
    __syncwarp();
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    const int g = (warp - 4) >> 2;               // warpgroup: columns [64g, 64g+64) of every accumulator
    const int r = (warp & 3) * 32 + lane;        // query row within the tile = TMEM lane
    const uint32_t tbase = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * 64);
    // Survivors are staged per row in shared memory as (score, id) -- this thread's own
    // column of the warpgroup's [SBUF][BM] array, so no synchronisation is needed -- and
    // reach the query's global array in batches: one atomicAdd a flush instead of one a
    // survivor, and the ordering keys are built only then.  A warp flushes when one of its
    // rows runs out of room and when its next unit has another query tile.
    const uint32_t at0 = s0 + LY::S_OFF + (uint32_t)(g * SBUF * BM + r) * 8u;
    const uint32_t at_end = at0 + (uint32_t)SBUF * (BM * 8u);
    uint32_t at = at0;
    int ia = 0;
    bool ok = true;
    for (int u = cid; u < U && ok; u += ncl) {
      const int qp = u % a.QP, c = u / a.QP;
      const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
      const int q = (CL * qp + rank) * BM + r;
      float tau = INFINITY;
      if (MODE == MODE_FILTER && q < a.nq) tau = a.tau ? a.tau[q] : -INFINITY;
      auto flush = [&] {
        f_flush(a.cnt + q, a.cand + (int64_t)q * a.cap, a.cap, at0, at);
        at = at0;
      };
      for (int p = p0; p < p1; ++p) {
        const int b = ia % F_NACC, ub = ia / F_NACC;
        // warp-uniform, so that a warp which gives up leaves its votes together
        if (!mbar_wait_warp(ACC_FULL(b), ub & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        uint32_t v[64];
        tmem_ld64(tbase + (uint32_t)(b * TN), v);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {  // scores are in registers: the MMA may reuse the buffer
          if (CL > 1) mbar_arrive_cluster(cluster_addr(ACC_EMPTY(b), 0));
          else mbar_arrive(ACC_EMPTY(b));
        }
        ++ia;
        const int64_t cbase = (int64_t)p * a.dstride * TN + g * 64;  // base id of v[0]
        const int piece = 4 * p + g;  // index of this 64-column piece among the row's sampled pieces
        if (cbase + 64 > a.n) {  // last base tile: padding rows become NaN, which no maximum or compare takes
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (cbase + j >= a.n) v[j] = 0x7fc00000u;
        }
        float m[8];
#pragma unroll
        for (int gg = 0; gg < 8; ++gg) m[gg] = max8(v, gg);
        const float tm = max3f(max3f(m[0], m[1], m[2]), max3f(m[3], m[4], m[5]), fmaxf(m[6], m[7]));
        if (MODE == MODE_GROUPMAX) {
          if (q < a.nq) {
            if (GW == 64) {
              a.gmax[(int64_t)q * a.M + piece] = tm;
            } else {
              float4* dst = reinterpret_cast<float4*>(a.gmax + (int64_t)q * a.M + 8 * piece);
              dst[0] = make_float4(m[0], m[1], m[2], m[3]);
              dst[1] = make_float4(m[4], m[5], m[6], m[7]);
            }
          }
        } else if (__any_sync(0xffffffffu, tm >= tau)) {
          const int ibase = (int)cbase;  // ids fit in 32 bits (n < 2^31)
          unsigned lm = 0;
#pragma unroll
          for (int gg = 0; gg < 8; ++gg) lm |= m[gg] >= tau ? (1u << gg) : 0u;
          const unsigned hm = __reduce_or_sync(0xffffffffu, lm);
#pragma unroll
          for (int gg = 0; gg < 8; ++gg) {
            if (!(hm & (1u << gg))) continue;
            int ng = 0;  // this lane's survivors in the group
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) ng += __uint_as_float(v[8 * gg + jj]) >= tau ? 1 : 0;
            if (at + (uint32_t)ng * (BM * 8u) > at_end) flush();
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              const float sc = __uint_as_float(v[8 * gg + jj]);
              if (sc >= tau) {
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(v[8 * gg + jj]), "r"(ibase + 8 * gg + jj) : "memory");
                at += BM * 8u;
              }
            }
          }
        }
      }
      if (MODE == MODE_FILTER && (!ok || u + ncl >= U || (u + ncl) % a.QP != qp)) flush();
    }
  }

  tc_fence_before();
  if (CL > 1) cluster_sync();  // both CTAs are done with TMEM and with each other's barriers
  else __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc<CL>(tmem, F_TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(a.err, 2);
  if (CL > 1) cluster_sync();  // a pair leaves together
}

// Descending scan of one warp's 256-bin histogram: digit = the bin where the count of keys
// in bins >= digit first reaches kk, rem = kk minus the count in the bins above it.  Lane l
// owns bins 255-8l .. 248-8l.  False (digit, rem untouched) when the bins hold fewer than
// kk keys.
__device__ __forceinline__ bool digit_of_rank(const unsigned* hist, int kk, int lane, int& digit, int& rem) {
  unsigned own = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) own += hist[255 - 8 * lane - j];
  unsigned incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (__shfl_sync(0xffffffffu, incl, 31) < (unsigned)kk) return false;
  const unsigned hit = __ballot_sync(0xffffffffu, incl >= (unsigned)kk);
  const int L = __ffs(hit) - 1;
  int dg = 0, rm = 0;
  if (lane == L) {
    unsigned acc = incl - own;
    for (int j = 0; j < 8; ++j) {
      const int d = 255 - 8 * lane - j;
      const unsigned h = hist[d];
      if (acc + h >= (unsigned)kk) {
        dg = d;
        rm = kk - (int)acc;
        break;
      }
      acc += h;
    }
  }
  digit = __shfl_sync(0xffffffffu, dg, L);
  rem = __shfl_sync(0xffffffffu, rm, L);
  return true;
}

// The threshold a query filters with: t - margin, lowered by 2 eps[q] where given (+inf, no
// survivor, when that is not finite).
__device__ __forceinline__ float lowered_tau(float t, float margin, const float* __restrict__ eps, int q) {
  if (!eps) return t - margin;
  const float e = eps[q];
  return e < 1e30f ? t - margin - 2.0f * e : INFINITY;
}

// tau[q] = (CT-th largest of the row's M group maxima) - margin, or -inf when the row has
// fewer than CT finite-or-infinite (non-NaN) maxima.  One warp per query: a 4-pass
// 8-bit radix select on order-preserving keys, histogram in shared memory.
__global__ void __launch_bounds__(256) tau_select_kernel(const float* __restrict__ gmax, int nq, int M, int CT,
                                                          float margin, float* __restrict__ tau,
                                                          const float* __restrict__ eps) {
  grid_ready();
  __shared__ unsigned hist[8][256];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = blockIdx.x * 8 + w;
  if (q >= nq) return;  // warp-uniform; only __syncwarp below
  const float* row = gmax + (int64_t)q * M;
  uint32_t prefix = 0, pmask = 0;
  int kk = CT;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int i = lane; i < 256; i += 32) hist[w][i] = 0;
    __syncwarp();
    for (int i = lane; i < M; i += 32) {
      const float f = row[i];
      if (f != f) continue;  // NaN maxima are not scores
      const uint32_t key = float_to_ordered(f);
      if ((key & pmask) == prefix) atomicAdd(&hist[w][(key >> shift) & 255u], 1u);
    }
    __syncwarp();
    int digit = 0, rem = 0;
    if (!digit_of_rank(hist[w], kk, lane, digit, rem)) {  // fewer than CT usable maxima (first pass only)
      if (lane == 0) tau[q] = lowered_tau(-INFINITY, margin, eps, q);
      return;
    }
    prefix |= (uint32_t)digit << shift;
    pmask |= 255u << shift;
    kk = rem;
    __syncwarp();
  }
  if (lane == 0) tau[q] = lowered_tau(ordered_to_float(prefix), margin, eps, q);
}

// tau_select_kernel for rows of at most 32 * R maxima (a multiple of 4), read once into
// registers by 16-byte loads.  It
// returns a lower bound of the CT-th largest maximum (minus the margin), which is all the
// filter needs -- a lower threshold only keeps more survivors, and the candidates
// selected from them are the same: a bisection on the order-preserving key between the
// row's smallest and largest maximum above -inf keeps lo with at least CT keys >= lo (so
// lo never passes the CT-th largest) and stops at 1/65536 of the range; each probe is a
// compare a key and one warp reduction (no histogram atomics, whose bins the clustered
// keys share).  With fewer than CT maxima above -inf (NaN is not a score) the CT-th
// largest is -inf, and so is tau, as in the exact select.
template <int R>
__global__ void __launch_bounds__(256) tau_select_reg_kernel(const float* __restrict__ gmax, int nq, int M, int CT,
                                                              float margin, float* __restrict__ tau,
                                                              const float* __restrict__ eps) {
  grid_ready();
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (q >= nq) return;  // warp-uniform
  // all R/4 16-byte loads issued before any is used (M % 4 == 0: rows are 16-byte aligned)
  const float4* row = reinterpret_cast<const float4*>(gmax + (int64_t)q * M);
  float4 raw[R / 4];
#pragma unroll
  for (int j = 0; j < R / 4; ++j) {
    const int i4 = j * 32 + lane;
    raw[j] = 4 * i4 < M ? __ldg(row + i4) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
  }
  uint32_t key[R];  // ordered keys; 0 = no value (no float but a NaN maps to 0)
  int valid = 0;
  uint32_t kmax = 0u, kmin = 0xffffffffu;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const float4 r4 = raw[j / 4];
    const float f = (j & 3) == 0 ? r4.x : (j & 3) == 1 ? r4.y : (j & 3) == 2 ? r4.z : r4.w;
    key[j] = (f == f && f != -INFINITY) ? float_to_ordered(f) : 0u;
    if (key[j]) {
      ++valid;
      kmax = max(kmax, key[j]);
      kmin = min(kmin, key[j]);
    }
  }
  if (__reduce_add_sync(0xffffffffu, valid) < CT) {
    if (lane == 0) tau[q] = lowered_tau(-INFINITY, margin, eps, q);
    return;
  }
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  uint64_t lo = kmin, hi = (uint64_t)kmax + 1;  // count(>= lo) >= CT > count(>= hi)
  const uint64_t stop = ((hi - lo) >> 16) + 1;
  while (hi - lo > stop) {  // warp-uniform
    const uint32_t mid = (uint32_t)(lo + ((hi - lo) >> 1));
    int c = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) c += key[j] >= mid ? 1 : 0;  // empty slots (0) never count: mid >= kmin >= 1
    if (__reduce_add_sync(0xffffffffu, c) >= CT) lo = mid;
    else hi = mid;
  }
  if (lane == 0) tau[q] = lowered_tau(ordered_to_float((uint32_t)lo), margin, eps, q);
}

// The same by a block a query, for rows of up to 256 * R maxima (a multiple of 4): long rows of
// 8-point maxima (10,000 rows of 4,480: the histogram form above 188 us, this 122).
template <int R>
__global__ void __launch_bounds__(256) tau_select_block_kernel(const float* __restrict__ gmax, int M, int CT,
                                                                float margin, float* __restrict__ tau,
                                                                const float* __restrict__ eps) {
  grid_ready();
  __shared__ unsigned part[3][2][8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = blockIdx.x;
  const float4* row = reinterpret_cast<const float4*>(gmax + (int64_t)q * M);
  uint32_t key[R];  // ordered keys; 0 = no value
  unsigned valid = 0, kmax = 0u, kmin = 0xffffffffu;
#pragma unroll
  for (int j = 0; j < R / 4; ++j) {
    const int i4 = j * 256 + tid;
    const float4 r = 4 * i4 < M ? __ldg(row + i4) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    const float f[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t k = (f[e] == f[e] && f[e] != -INFINITY) ? float_to_ordered(f[e]) : 0u;
      key[4 * j + e] = k;
      if (k) {
        ++valid;
        kmax = max(kmax, k);
        kmin = min(kmin, k);
      }
    }
  }
  valid = __reduce_add_sync(0xffffffffu, valid);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  if (lane == 0) {
    part[0][0][warp] = valid;
    part[1][0][warp] = kmax;
    part[2][0][warp] = kmin;
  }
  __syncthreads();
  valid = __reduce_add_sync(0xffffffffu, lane < 8 ? part[0][0][lane] : 0u);
  kmax = __reduce_max_sync(0xffffffffu, lane < 8 ? part[1][0][lane] : 0u);
  kmin = __reduce_min_sync(0xffffffffu, lane < 8 ? part[2][0][lane] : 0xffffffffu);
  if ((int)valid < CT) {  // block-uniform
    if (tid == 0) tau[q] = lowered_tau(-INFINITY, margin, eps, q);
    return;
  }
  uint64_t lo = kmin, hi = (uint64_t)kmax + 1;  // count(>= lo) >= CT > count(>= hi)
  const uint64_t stop = ((hi - lo) >> 12) + 1;  // 1/4096 of the range: a few survivors more
  for (int it = 1; hi - lo > stop; ++it) {  // block-uniform; one barrier a step, buffers in turn
    const uint32_t mid = (uint32_t)(lo + ((hi - lo) >> 1));
    int c = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) c += key[j] >= mid ? 1 : 0;  // empty slots (0) never count: mid >= kmin >= 1
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) part[0][it & 1][warp] = (unsigned)c;
    __syncthreads();
    if ((int)__reduce_add_sync(0xffffffffu, lane < 8 ? part[0][it & 1][lane] : 0u) >= CT) lo = mid;
    else hi = mid;
  }
  if (tid == 0) tau[q] = lowered_tau(ordered_to_float((uint32_t)lo), margin, eps, q);
}

// The 32*E smallest of c keys, ascending (element e * 32 + lane), by one warp: sort each chunk
// and merge it into the running result.
template <int E>
__device__ __forceinline__ void warp_top(const uint64_t* __restrict__ src, int c, int lane, uint64_t (&best)[E]) {
  constexpr int CT = 32 * E;
#pragma unroll
  for (int e = 0; e < E; ++e) best[e] = kEmptyKey;
  for (int base = 0; base < c; base += CT) {
    uint64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int i = base + e * 32 + lane;
      x[e] = i < c ? src[i] : kEmptyKey;
    }
    warp_bitonic<E>(x, lane, false);
    // best ascending, x ascending: min(best[i], x[CT-1-i]) is bitonic and holds the CT
    // smallest of the union
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint64_t r = __shfl_sync(0xffffffffu, x[E - 1 - e], 31 - lane);
      best[e] = best[e] < r ? best[e] : r;
    }
    warp_bitonic<E>(best, lane, true);
  }
}

// Per query (one warp): the CT = 32*E smallest keys of the survivors -- sort each chunk of
// CT keys and merge it into the running result with a bitonic "min + merge" step.  Lists
// queries whose survivors overflowed the candidate array (ovf[0] = count, ovf[1..] = ids).
template <int E>
__global__ void __launch_bounds__(256) cand_select_kernel(const int* __restrict__ cnt,
                                                           const uint64_t* __restrict__ cand, int cap, int need,
                                                           int nq, uint64_t* __restrict__ out,
                                                           int* __restrict__ ovf, const uint16_t* __restrict__ rows,
                                                           uint16_t* __restrict__ gathered) {
  grid_ready();
  constexpr int CT = 32 * E;
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (q >= nq) return;  // warp-uniform
  const int c = cnt[q];
  uint64_t* dst = out + (int64_t)q * CT;
  if (c > cap || c < need) {
#pragma unroll
    for (int e = 0; e < E; ++e) dst[e * 32 + lane] = kEmptyKey;
    int at = 0;
    if (lane == 0) {
      at = atomicAdd(ovf, 1);
      ovf[1 + at] = q;
    }
    at = __shfl_sync(0xffffffffu, at, 0);
    // its row for the list kernel (rows past the count are never read out)
    if (gathered)
      reinterpret_cast<uint2*>(gathered + (int64_t)at * KD)[lane] =
          reinterpret_cast<const uint2*>(rows + (int64_t)q * KD)[lane];
    return;
  }
  uint64_t best[E];
  warp_top<E>(cand + (int64_t)q * cap, c, lane, best);
#pragma unroll
  for (int e = 0; e < E; ++e) dst[e * 32 + lane] = best[e];
}

// launch_exact_select: keys order by score, so the sorted top-CT gives the k-th best score and
// the candidates are a prefix of it.
template <int E>
__global__ void __launch_bounds__(256) exact_select_kernel(const int* __restrict__ cnt,
                                                            const uint64_t* __restrict__ cand, int cap, int k, int nq,
                                                            const float* tau, const float* __restrict__ eps,
                                                            uint64_t* __restrict__ out, int* __restrict__ ovf,
                                                            float* lim) {
  grid_ready();
  constexpr int CT = 32 * E;
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (q >= nq) return;  // warp-uniform
  const int c = cnt[q];
  const float e2 = 2.0f * eps[q];
  uint64_t* dst = out + (int64_t)q * CT;
  bool listed = c > cap || c < k || !(e2 < 1e30f);
  uint64_t best[E];
#pragma unroll
  for (int e = 0; e < E; ++e) best[e] = kEmptyKey;
  float cut = 0.0f;
  // a score that k points reach (none: -inf); it bounds their distances by 1 - reach + eps
  const float t = tau ? tau[q] : -INFINITY;
  float reach = c >= k ? t : -INFINITY;
  if (!listed) {
    warp_top<E>(cand + (int64_t)q * cap, c, lane, best);
    uint64_t kth = kEmptyKey, last = kEmptyKey;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint64_t v = __shfl_sync(0xffffffffu, best[e], (k - 1) & 31);
      if (e == (k - 1) >> 5) kth = v;
      last = best[e];
    }
    last = __shfl_sync(0xffffffffu, last, 31);
    reach = -key_dist(kth);
    cut = reach - e2;  // scores from here up
    listed = (tau && t > cut) || (last != kEmptyKey && c > CT && -key_dist(last) >= cut);
  }
#pragma unroll
  for (int e = 0; e < E; ++e)
    dst[e * 32 + lane] = !listed && best[e] != kEmptyKey && -key_dist(best[e]) >= cut ? best[e] : kEmptyKey;
  __syncwarp();  // every lane has read tau[q], which may be lim[q]
  if (listed && lane == 0) {
    ovf[1 + atomicAdd(ovf, 1)] = q;
    lim[q] = e2 < 1e30f ? 1.0f - reach + 0.5f * e2 + 1e-6f : INFINITY;
  }
}

// Merge the list kernel's per-CTA partial lists of every listed query and write the
// result over the query's row of `out`.  The split arithmetic repeats the list kernel's
// (tc_list_geometry).
__global__ void merge_fallback_kernel(const uint64_t* __restrict__ part, const int* __restrict__ ovf, int NT,
                                      int grid, int CT, uint64_t* __restrict__ out) {
  grid_ready();
  extern __shared__ uint64_t ms[];
  const int cntq = ovf[0];
  if (cntq == 0) return;
  const ListGeometry geo = tc_list_geometry(cntq, NT, grid);
  for (int i = blockIdx.x; i < cntq; i += gridDim.x) {
    const int qt = i / BM;
    const int first = (int)(((int64_t)qt * NT) / geo.per);
    const int last = (int)(((int64_t)qt * NT + NT - 1) / geo.per);
    const uint64_t* src = part + (int64_t)i * geo.maxp * CT;
    for (int j = threadIdx.x; j < CT; j += blockDim.x) ms[j] = src[j];
    __syncthreads();
    for (int s = 1; s <= last - first; ++s) {
      const uint64_t* lst = src + (int64_t)s * CT;
      for (int j = threadIdx.x; j < CT; j += blockDim.x) {
        const uint64_t b = lst[CT - 1 - j];
        if (b < ms[j]) ms[j] = b;
      }
      __syncthreads();
      block_bitonic_merge(ms, CT);
    }
    const int q = ovf[1 + i];
    for (int j = threadIdx.x; j < CT; j += blockDim.x) out[(int64_t)q * CT + j] = ms[j];
    __syncthreads();
  }
}

template <int MODE, int GW, bool F8, int KC, int CL>
void run_filter_as(const FilterMaps& m, FilterArgs a, int clusters, const char* name, cudaStream_t s) {
  // chunk size: long enough to amortise the query-tile switch (at most 32 tiles), short
  // enough for >= 16 units per cluster so the last unit leaves little imbalance
  const int64_t work = (int64_t)a.NP * a.QP;
  a.CH = (int)std::max<int64_t>(1, std::min<int64_t>(32, (work + 16 * clusters - 1) / (16 * clusters)));
  a.NCH = ceil_div(a.NP, a.CH);
  const int grid = CL * std::min(clusters, a.NCH * a.QP);
  auto kern = tc_filter_kernel<MODE, GW, F8, KC, CL>;
  constexpr int smem = FLayout<KC, CL>::SMEM;
  raise_smem_limit(kern, smem);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(F_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2]{};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = CL;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CL > 1 ? 2 : 1;
  ProfScope _ps(name, s);
  LSHG_CUDA(cudaLaunchKernelEx(&cfg, kern, m.a, m.b, m.bhi, a));
  count_launch();
}

template <int MODE, int GW, bool F8, int KC>
void run_filter(const FilterMaps& m, FilterArgs a, const char* name, cudaStream_t s) {
  a.QP = ceil_div(a.QT, m.cl);
  const int G = std::max(1, num_sms() / m.cl);
  // Clusters in a multiple of the groups keep one query tile each for the whole scan: nothing
  // is reloaded and the staging is flushed when it is full, not every unit (100k x 100, 1,000
  // queries: units of two tiles).  Worth up to 6% of the SMs.
  const int keep = a.QP <= G ? G / a.QP * a.QP : 0;
  const int clusters = keep * 100 >= G * 94 ? keep : G;
  if (m.cl == 2) run_filter_as<MODE, GW, F8, KC, 2>(m, a, clusters, name, s);
  else run_filter_as<MODE, GW, F8, KC, 1>(m, a, clusters, name, s);
}

template <int MODE, int GW>
void run_filter_fmt(const FilterMaps& m, const FilterArgs& a, const char* name, cudaStream_t s) {
  if (m.e4m3) run_filter<MODE, GW, true, 1>(m, a, name, s);
  else if (a.ksteps <= 4) run_filter<MODE, GW, false, 1>(m, a, name, s);
  else run_filter<MODE, GW, false, 2>(m, a, name, s);
}

}  // namespace

// Prepass parameters in units of TN-point tiles.  Large bases sample every S-th tile
// (S <= 16) and take tau at rank r = CT/S + 4 sqrt(CT/S) + 8 of the sample's 64-column
// maxima: the query's CT-th best point puts about CT/S points of the sample above it, so
// tau stays at or below that point unless the count exceeds its mean by four standard
// deviations, and about r * S points survive (CT * S with r = CT).  A query with fewer
// than CT survivors is rescanned exactly by the list kernel (cand_select lists it), so
// the rank only trades survivors against fallbacks.  Among the S that leave at least 4 r
// maxima a row, so that the r-th largest is a tight bound, the plan takes the cheapest, by
// what each part took at 1.2M x 10,000 and 100k x 1,000: 0.9 us a sampled tile of an SM, 3.2 ps
// a maximum of the threshold select, 0.12 ns a survivor (its way through the filter and the
// candidate select).  10,000 queries on 1.2M points: S = 16 prepass, threshold, filter and
// select 104 + 39 + 1,730 + 60 us, S = 8 199 + 75 + 1,630 + 44; 1,000 on 100k: S = 16 10 +
// 10 + 48 + 18 us, S = 1 25 + 17 + 33 + 9.
FilterPlan plan_filter(int64_t n, int CT, int nq) {
  FilterPlan p{};
  const int NT = ceil_div(n, TN);
  p.NT = NT;
  p.rank = CT;
  if (NT >= CT) {  // 64-column maxima: 4 a tile
    p.GW = 64;
    p.S = 1;
    const int QT = ceil_div(nq, BM);
    double best = 0.0;
    for (int S : {16, 8, 4, 2, 1}) {
      const double m = (double)CT / S;
      const int r = S == 1 ? CT : std::min(CT, (int)std::ceil(m + 4.0 * std::sqrt(m) + 8.0));
      const int NS = ceil_div(NT, S);
      if (S > 1 && NS < r) continue;
      const double cost = 0.9e-6 * ceil_div((int64_t)NS * QT, num_sms()) + 3.2e-12 * (double)nq * 4 * NS +
                          0.12e-9 * (double)nq * r * S;
      if (best == 0.0 || cost < best) {
        best = cost;
        p.S = S;
        p.rank = r;
      }
    }
    p.NS = ceil_div(NT, p.S);
    p.M = 4 * p.NS;
    p.cap = std::max(1024, 4 * p.rank * p.S);
  } else if (NT * 32 >= 4 * CT) {  // 8-column maxima: 32 a tile
    p.GW = 8;
    p.S = 1;
    p.NS = NT;
    p.M = 32 * NT;
    p.cap = std::max(1024, 4 * CT);
  } else {  // a few thousand points: keep every one
    p.GW = 0;
    p.S = 1;
    p.NS = 0;
    p.M = 0;
    p.cap = NT * TN;
  }
  p.cap = std::min<int64_t>(p.cap, (int64_t)NT * TN);
  return p;
}

FilterMaps make_filter_maps(const void* q, int64_t qrows, const void* base, int64_t brows, int d, bool e4m3) {
  FilterMaps m{};
  m.e4m3 = e4m3;
  // clusters of two query tiles share each base tile's fetch; one tile alone would leave the
  // second CTA without work
  m.cl = qrows > BM ? 2 : 1;
  m.hi_cols = std::max(8, std::min(KHALF, 16 * tc_ksteps(d) - KHALF));
  if (e4m3) {
    m.a = make_map_e4m3(q, qrows, BM);
    m.b = make_map_e4m3(base, brows, TN / m.cl);
    m.bhi = m.b;
  } else {
    m.a = make_map(q, qrows);
    m.b = make_map(base, brows, TN / m.cl);
    m.bhi = make_map(base, brows, TN / m.cl, m.hi_cols);
  }
  return m;
}

void launch_filter_scan(const FilterMaps& m, const FilterPlan& plan, int nq, int64_t n, int d, int QT, float* tau,
                        int* cnt, uint64_t* cand, int* err, cudaStream_t s, const float* eps) {
  FilterArgs a{};
  a.hi_bytes = m.hi_cols * 2;
  a.nq = nq;
  a.ksteps = m.e4m3 ? tc_ksteps_e4m3(d) : tc_ksteps(d);
  // scores of E4M3 codes carry the factor kE4M3Scale^2
  const float margin = m.e4m3 ? kTauMargin * kE4M3Scale * kE4M3Scale : kTauMargin;
  a.n = n;
  a.QT = QT;
  a.err = err;
  if (plan.M > 0) {
    DevBuf<float> gmax((size_t)nq * plan.M, s);
    a.NP = plan.NS;
    a.dstride = plan.S;
    a.gmax = gmax.ptr;
    a.M = plan.M;
    if (plan.GW == 64) run_filter_fmt<MODE_GROUPMAX, 64>(m, a, "tc_prepass", s);
    else run_filter_fmt<MODE_GROUPMAX, 8>(m, a, "tc_prepass", s);
    launch_tau_select(gmax.ptr, nq, plan.M, plan.rank, margin, tau, s, eps);
  }
  a.gmax = nullptr;
  a.M = 0;
  a.NP = plan.NT;
  a.dstride = 1;
  a.tau = plan.M > 0 ? tau : nullptr;
  a.cnt = cnt;
  a.cand = cand;
  a.cap = plan.cap;
  run_filter_fmt<MODE_FILTER, 64>(m, a, "tc_filter", s);
}

void launch_tau_select(const float* gmax, int nq, int M, int rank, float margin, float* tau, cudaStream_t s,
                       const float* eps) {
  ProfScope _ps("tc_tau_select", s);
  // the register slots a lane walks in every bisection step: as few as cover M
  if (M <= 32 * kTauRegsFew && M % 4 == 0)
    launch_next(tau_select_reg_kernel<kTauRegsFew>, ceil_div(nq, 8), 256, 0, s, gmax, nq, M, rank, margin, tau, eps);
  else if (M <= 32 * kTauRegs && M % 4 == 0)
    launch_next(tau_select_reg_kernel<kTauRegs>, ceil_div(nq, 8), 256, 0, s, gmax, nq, M, rank, margin, tau, eps);
  else if (M <= 256 * kTauBlockRegs && M % 4 == 0)
    launch_next(tau_select_block_kernel<kTauBlockRegs>, nq, 256, 0, s, gmax, M, rank, margin, tau, eps);
  else
    launch_next(tau_select_kernel, ceil_div(nq, 8), 256, 0, s, gmax, nq, M, rank, margin, tau, eps);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

void launch_cand_select(const int* cnt, const uint64_t* cand, int nq, int cap, int need, int CT, uint64_t* out,
                        int* ovf, const uint16_t* rows, uint16_t* gathered, cudaStream_t s) {
  ProfScope _ps("tc_cand_select", s);
  if (CT == 32) launch_next(cand_select_kernel<1>, ceil_div(nq, 8), 256, 0, s, cnt, cand, cap, need, nq, out, ovf,
                            rows, gathered);
  else if (CT == 64) launch_next(cand_select_kernel<2>, ceil_div(nq, 8), 256, 0, s, cnt, cand, cap, need, nq, out,
                                 ovf, rows, gathered);
  else if (CT == 128) launch_next(cand_select_kernel<4>, ceil_div(nq, 8), 256, 0, s, cnt, cand, cap, need, nq, out,
                                  ovf, rows, gathered);
  else throw Error(LSHG_ERR_INVALID_ARGUMENT, "tensor-core scan: candidate count must be 32, 64 or 128");
  count_launch();
  LSHG_CHECK_LAUNCH();
}

void launch_exact_select(const int* cnt, const uint64_t* cand, int nq, int cap, int k, int CT, const float* tau,
                         const float* eps, uint64_t* out, int* ovf, float* lim, cudaStream_t s) {
  ProfScope _ps("exact_select", s);
  if (CT == 128) launch_next(exact_select_kernel<4>, ceil_div(nq, 8), 256, 0, s, cnt, cand, cap, k, nq, tau, eps,
                             out, ovf, lim);
  else if (CT == 256) launch_next(exact_select_kernel<8>, ceil_div(nq, 8), 256, 0, s, cnt, cand, cap, k, nq, tau,
                                  eps, out, ovf, lim);
  else throw Error(LSHG_ERR_INVALID_ARGUMENT, "exact scan: candidate count must be 128 or 256");
  count_launch();
  LSHG_CHECK_LAUNCH();
}

void launch_merge_fallback(const uint64_t* part, const int* ovf, int nq, int NT, int grid, int CT, uint64_t* out,
                           cudaStream_t s) {
  const size_t smem = (size_t)CT * 8;
  launch_next(merge_fallback_kernel, std::min(nq, num_sms() * 4), 128, smem, s, part, ovf, NT, grid, CT, out);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

}  // namespace tc
}  // namespace lshg
