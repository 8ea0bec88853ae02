// Tensor-core sketch scan: the Hamming distance of bit sketches as a +-1 E2M1 (FP4) GEMM
// (implementations 3 and 5 -- SimHash and one-bit weighted MinHash -- in place of the
// XOR/popcount scan of scan_bits.cu for batches that fill the tensor cores; the
// reference's scanHammingDistance, sketchedDistanceScanners.cuh:14-100, and its one-bit
// scanJaccardDistance, :194-274).
//
// Bit b of a sketch becomes the E2M1 value 1 - 2b: +1.0 (0x2) or -1.0 (0xA), two to a byte.
// For two sketches of B = 32 * words bits the dot product of those rows is (#equal bits) -
// (#different bits) = B - 2 * hamming.  Every product is +-1, every block scale 1.0 and
// every partial sum an integer of magnitude <= B <= 1024, which FP32 holds exactly, so the
// accumulator gives hamming = (B - dot) / 2 exactly, and the top-C by (hamming, id) equals
// the popcount scan's.  The one-bit Jaccard distance 1 - (B - hamming) / B orders points the
// same way.  Rows are padded to whole 128-byte chunks (256 bits) with 0x0 (+0.0), which adds
// nothing.
//
// Selection, as in the threshold-filter scan of tc_filter.cu, in two GEMM passes:
//   prepass  on every S-th base tile writes each query's group maxima of the score (the
//            best score of each 56- or 8-point group of a sampled tile); tau[q] = the
//            r-th largest of them (launch_tau_select).  With S = 1, r = C and every point
//            of the exact top-C scores >= tau.  With S > 1, r = C/S + 4 sqrt(C/S) + 8 -- the
//            C-th best point of the base would put about C/S points of the sample above
//            it, so tau stays at or below it unless that count exceeds its mean by four
//            standard deviations -- and about r * S ~ 1.5 C points survive instead of C * S;
//   filter   on the whole base keeps the points whose score reaches tau[q], staged per row
//            in shared memory and moved to the query's candidate array with one atomicAdd
//            a batch;
//   select   keeps each query's first C survivors by (score desc, id asc): bisection
//            over the integer scores and over the ids at the C-th score by a block, or a warp
//            sort for C <= 128 and many queries.
//            A query with fewer than C survivors (tau above its C-th best score: the
//            sample was unrepresentative) or more than its array holds (massive ties) is
//            listed and rescanned exactly by the popcount scan on the device, so the result
//            is always the exact top-C.
//
// tc_hamming_kernel: persistent, one CTA per SM, 640 threads, in clusters of CL = 2 CTAs (1
// for batches of one query tile).  A unit is (CL query tiles of 128 rows, chunk of up to 36
// consecutive base tiles of 224 points), numbered chunk-major so that all SMs stream the
// same base tiles at a time (each read from HBM about once a batch, then from L2).  The two
// CTAs of a cluster are an MMA pair (tcgen05 cta_group::2): each keeps its query tile in shared
// memory for the unit (KC chunks of 128 rows x 128 bytes) and streams its half of the base
// tile through a ring of one-chunk stages (112 rows x 128 bytes); the even one issues the MMAs
// of both.  A CTA on its own reads 11 KB of operands from shared memory an MMA of 112 cycles and
// writes 28 KB of base tile every four -- 160 bytes a cycle of the 128 there are -- and takes
// 112 KB a tile from L2; in a pair both halve on the base tile's side.
// Warp 0 issues the TMA copies, warp 1 the MMAs (tcgen05.mma kind::mxf4 with block scales
// of 1.0, M = 128, N = 224, K = 64 each; 4 a chunk), warp 2 owns the 512 TMEM columns, warps
// 4-19 are the epilogue (warpgroup g reads columns [56g, 56g + 56), one query row a thread).
// N = 224 leaves TMEM columns [224, 256) beside the two accumulators (at 0 and 256) for the
// scale factors, which are filled once with the UE8M0 code of 1.0 (0x7f), so their layout
// does not matter.  Every mbarrier wait is bounded (2 s); a CTA that times out raises
// error 2, drains its copies and MMAs, frees TMEM and returns; the CTAs of a cluster leave
// together.
//
// Measured (filter pass; 10,000 queries): 1.2M points of 1,024 bits 7.52 -> 2.96 ms (8.3
// PFLOP/s of +-1 products; 2.5 ms is the MMAs alone), 500k points of 256 bits at C = 4,096
// 4.79 -> 1.79 ms (bounded by the 1.3% survivors: without any the same pass takes 0.67 ms);
// before: E4M3 rows (twice the bytes, half the MMA rate), a query tile a CTA with its own
// copy of every base tile, MMAs issued from a diverged warp, branches around each store.  The
// pair's MMAs against two CTAs that multicast the base tile to each other: 3.25 -> 2.96 ms.
//
// tc_signs_kernel: the same pipeline with BF16 operands and one query tile for the SimHash
// projections (below).
#include "index.h"
#include "launch_count.h"
#include "launch_next.cuh"
#include "profile.h"
#include "select.cuh"
#include "tc_filter.h"
#include "tc_ptx.cuh"

#include <cuda_bf16.h>

namespace lshg {

int launch_scan_bits_listed(const uint32_t* xst, int64_t n, int wp, int words, int sbytes, const uint32_t* qs, int nq,
                            int op, int C, const int* list, uint64_t* out, uint64_t* scratch, int room,
                            cudaStream_t s);

namespace tc {

namespace {

constexpr int H_THREADS = 640;
constexpr int HN = 224;           // base points a tile (UMMA N): 4 warpgroups x 7 groups of 8 columns
constexpr int HW = HN / 4;        // columns a warpgroup reads
constexpr int H_CHUNK = 128;      // bytes of a row in one K chunk (one 128-byte swizzle row): 256 bits
constexpr int H_TMEM_COLS = 512;  // accumulators at columns 0 and 256, scale factors at [224, 256)
constexpr int H_ACC_COL = 256;
constexpr int H_SF_COL = HN;
constexpr int H_MAX_CH = 36;      // base tiles a unit: 36 * 224 column offsets fit the staging's 13 bits
constexpr int H_EPI_WARPS = 16;
// Batches whose base tiles are expanded from packed sketches: those that leave half of the epilogue
// warps without query rows to read.  They are bounded by the base's bytes where it does not fit in L2
// (16 queries of 1,024 bits: 1.2M points, filter pass 97 -> 82 us, batch 185 -> 165; 400k, batch 163 ->
// 145; 256 bits, 1.2M, 161 -> 151), and as fast either way where it does (100k: 87 and 87).
constexpr int H_BITS_MAX_Q = 64;
constexpr int H_SEL_MAX = 16384;  // survivor slots a query of a filtered base, at most
constexpr int PN = 256;           // planes a tile of the projections' GEMM (UMMA N)
constexpr int P_NACC = 2;         // its TMEM accumulators of PN columns

constexpr int kSmemLimit = 232448;  // dynamic shared memory a CTA may opt into

// Shared-memory layout of a CTA in a cluster of CL, for rows of KC chunks: the resident query
// tile, the ring of its shares of base chunks, and the survivor staging (SBUF 4-byte entries a
// row and warpgroup).
template <int KC, int CL>
struct HLayout {
  static constexpr int A_BYTES = KC * BM * H_CHUNK;  // query tile
  static constexpr int B_BYTES = HN / CL * H_CHUNK;  // one chunk of a base tile: 28 KB, or a pair's 14 KB
  static constexpr int STAGES = CL == 2 ? 7 : 4;
  static constexpr int SBUF = 24;
  static constexpr int A_OFF = 0;
  static constexpr int B_OFF = A_BYTES;
  static constexpr int S_OFF = B_OFF + STAGES * B_BYTES;  // [4][SBUF][BM] entries
  static constexpr int BAR_OFF = S_OFF + 4 * SBUF * BM * 4;
  static constexpr int SMEM = BAR_OFF + 256 + 1024;  // + barriers + alignment slack
  static_assert(SMEM <= kSmemLimit, "shared memory per CTA");
  static_assert(8 * (2 * STAGES + 7) + 8 <= 256, "barrier area");
};
static_assert(H_MAX_CH * HN <= 8192, "column offsets of a unit fit 13 bits");

struct HArgs {
  int nq;
  int64_t n;
  int QT;           // query tiles
  int QP;           // groups of CL of them
  int NP;           // base positions scanned (base tile = p * dstride)
  int dstride;
  int CH;           // positions a unit
  int NCH;          // chunks of positions
  int ksteps;       // MMA K steps (64 bits each) that cover a sketch
  float* gmax;      // MODE_GROUPMAX: [nq][M] group maxima
  int M;
  const float* tau; // MODE_FILTER: threshold a query (nullptr: keep every point)
  int* cnt;         // survivors a query
  uint64_t* cand;   // [nq][cap] survivor keys
  int cap;
  int* err;
  const uint4* xst;  // BITS: the packed sketches, [ceil(n/128)][wq][128] 16-byte words
  int wq;
};

// Survivor staging: a thread's entries lie BM words apart in its warpgroup's [SBUF][BM]
// array (lane = bank).  An entry is the score's float bits with the column's offset in the
// unit in the low 13 bits: scores are integers of magnitude at most 1024, whose mantissas
// leave the low 14 bits zero.  A push is a compare, an add and two predicated instructions,
// without a branch: at the one-bit MinHash rates (1.3% of the scores survive, about 25 a
// warp and tile) branches around each store had made the survivor path five times as long
// as everything else in the kernel.
__device__ __forceinline__ void h_push(uint32_t v, float tau, uint32_t& at, uint32_t off) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ge.f32 p, %1, %2;\n\t@p st.shared.u32 [%0], %3;\n\t@p add.u32 %0, %0, %4;\n\t}"
      : "+r"(at)
      : "f"(__uint_as_float(v)), "f"(tau), "r"(v + off), "n"(BM * 4)
      : "memory");
}

// Move this thread's `n` > 0 staged entries to its query's candidate array: one atomicAdd
// reserves the slots.  id0: the base id of offset 0.  Out of line: inlined copies would
// crowd the instruction cache.
__device__ __noinline__ void h_flush(int* cnt, uint64_t* dst, int cap, uint32_t at0, int n, int id0) {
  const int base = atomicAdd(cnt, n);
  for (int e = 0; e < n; ++e) {
    uint32_t w;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(at0 + e * (BM * 4)));
    if (base + e < cap) dst[base + e] = make_key(-__uint_as_float(w & ~0x3fffu), id0 + (int)(w & 0x1fffu));
  }
}

// A sketch word as the E2M1 values of its bits, sign bit = sketch bit: value j of word e is bit
// 4 j + 3 - e.  Any order does, as long as queries and points have the same.
__device__ __forceinline__ uint4 expand_word(uint32_t b) {
  constexpr uint32_t S = 0x88888888u, ONE = 0x22222222u;
  return make_uint4((b & S) | ONE, ((b << 1) & S) | ONE, ((b << 2) & S) | ONE, ((b << 3) & S) | ONE);
}

// BITS (CL = 1, batches of at most H_BITS_MAX_Q queries): the base tile is read as packed
// sketches, a quarter of the E2M1 rows' bytes, and expanded into the ring by the epilogue warps
// that have no query rows (TMEM lanes 64 and up): thread r takes row r, its next tile's words in
// flight while this one's are expanded, and its 16-byte stores of a chunk fall into distinct banks
// by the rows' swizzle.  Bounded by shared memory (114 KB written and 176 KB of operands read a
// tile) and by the expanding warps' chain of wait, store, fence and arrive; a quarter of the stores
// alone would take 27 us off the 82.
template <int MODE, int GW, int KC, int CL, bool BITS>
__global__ void __launch_bounds__(H_THREADS, 1)
    tc_hamming_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                      const HArgs a) {
  grid_ready();
  using LY = HLayout<KC, CL>;
  constexpr int STAGES = LY::STAGES, SBUF = LY::SBUF;
  static_assert(MODE != MODE_FILTER || GW == HW, "the filter reads whole pieces");
  static_assert(GW == HW || GW == 8, "group width");
  static_assert(!BITS || CL == 1, "one query tile");
  constexpr int EPI_WARPS = BITS ? H_EPI_WARPS / 2 : H_EPI_WARPS;  // those with query rows
  const int U = a.NCH * a.QP;
  const int cid = blockIdx.x / CL, ncl = gridDim.x / CL;  // cluster, clusters
  if (cid >= U) return;  // no unit for this cluster: leave before any barrier or TMEM use

  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t s0 = smem_u32(sm);
  const uint32_t bar0 = s0 + LY::BAR_OFF;
  auto FULL = [&](int s) { return bar0 + 8u * s; };
  auto EMPTY = [&](int s) { return bar0 + 8u * (STAGES + s); };
  const uint32_t A_FULL = bar0 + 8u * (2 * STAGES);
  const uint32_t A_EMPTY = bar0 + 8u * (2 * STAGES + 1);
  auto ACC_FULL = [&](int b) { return bar0 + 8u * (2 * STAGES + 2 + b); };
  auto ACC_EMPTY = [&](int b) { return bar0 + 8u * (2 * STAGES + 4 + b); };
  const uint32_t DONE = bar0 + 8u * (2 * STAGES + 6);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + LY::BAR_OFF + 8 * (2 * STAGES + 7));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform for the compiler too
  const int lane = threadIdx.x & 31;
  const int rank = CL > 1 ? (int)cluster_rank() : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(FULL(s), BITS ? HN / 32 : 1);
      mbar_init(EMPTY(s), 1);
    }
    mbar_init(A_FULL, 1);
    mbar_init(A_EMPTY, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(ACC_FULL(b), 1);
      mbar_init(ACC_EMPTY(b), CL * EPI_WARPS);  // a pair's even CTA waits for both
    }
    mbar_init(DONE, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) tmem_alloc<CL>(smem_u32(tmem_slot), H_TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (warp >= 4 && warp < 8) {  // scale factors: 1.0 in every byte of every lane
#pragma unroll
    for (int c = H_SF_COL; c < H_ACC_COL; c += 8)
      tmem_fill8(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, 0x7f7f7f7fu);
    tmem_wait_st();
  }
  tc_fence_before();
  if (CL > 1) cluster_sync();  // the peer's barriers are initialised before anything arrives on them
  else __syncthreads();
  tc_fence_after();

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      // a pair's bytes are counted on its even CTA's barriers, where the MMAs are issued
      auto load = [&](uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
        if (CL > 1) tma_load_2d_pair(dst, map, x, y, cluster_addr(bar, 0));
        else tma_load_2d(dst, map, x, y, bar);
      };
      int it = 0, na = 0;  // base chunks and query tiles issued
      int have = -1;       // query tile in shared memory
      bool ok = true;
      for (int u = cid; u < U && ok; u += ncl) {
        const int qp = u % a.QP, c = u / a.QP;
        const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
        // The unit's first STAGES base chunks are issued before its query tile: their
        // stages free up as the previous unit's MMAs consume the ring, so the copies run
        // while those MMAs finish.  The query tile is reloaded once the previous unit's MMAs
        // have completed, and kept when the next unit has the same one.  (A tile past the
        // last one, where the query tiles do not fill the cluster, reads as zeros.)
        const int total = BITS ? 0 : (p1 - p0) * KC, pre = min(STAGES, total);
        for (int ci = 0; ci <= total; ++ci) {
          if (ci == pre && qp != have) {
            if (!mbar_wait(A_EMPTY, (na & 1) ^ 1, abort_flag)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(A_FULL, CL * LY::A_BYTES);
#pragma unroll
            for (int kc = 0; kc < KC; ++kc)
              load(s0 + LY::A_OFF + kc * BM * H_CHUNK, &mapA, kc * H_CHUNK, (CL * qp + rank) * BM, A_FULL);
            ++na;
            have = qp;
          }
          if (ci == total) break;
          const int p = p0 + ci / KC, kc = ci % KC;
          const int st = it % STAGES, rd = it / STAGES;
          if (!mbar_wait(EMPTY(st), (rd & 1) ^ 1, abort_flag)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(FULL(st), CL * LY::B_BYTES);
          load(s0 + LY::B_OFF + st * LY::B_BYTES, &mapB, kc * H_CHUNK, p * a.dstride * HN + rank * (HN / CL), FULL(st));
          ++it;
        }
      }
      // drain: every copy has landed and every stage has been given back before the CTA may
      // exit (a pair's odd CTA sees its copies' end only by the stages that come back)
      for (int j = max(0, it - STAGES); j < it; ++j) {
        if (rank == 0) mbar_wait(FULL(j % STAGES), (j / STAGES) & 1, abort_flag, true);
        mbar_wait(EMPTY(j % STAGES), (j / STAGES) & 1, abort_flag, true);
      }
      if (rank == 0 && na > 0) mbar_wait(A_FULL, (na - 1) & 1, abort_flag, true);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (a pair's: its even CTA) ----------------
    if (rank == 0) {
      const uint32_t leader = elect_one();  // the warp stays converged (see elect_one)
      constexpr uint32_t idesc = idesc_mxf4(CL * BM, HN);
      auto commit = [&](uint32_t bar) {
        if (CL > 1) umma_commit_pair(bar, leader);
        else umma_commit(bar, leader);
      };
      // Running stage and parity, descriptors by 32-bit additions, steps cut off by the
      // predicate: a tile's MMAs take 448 cycles a chunk, and this warp's own time has to stay
      // below that.
      const uint32_t a_lo = smem_desc_lo(s0 + LY::A_OFF), b_lo0 = smem_desc_lo(s0 + LY::B_OFF);
      int st = 0, na = 0, b = 0;
      uint32_t ph = 0, acc_ph = 1;
      int have = -1;
      bool ok = true;
      for (int u = cid; u < U && ok; u += ncl) {
        const int qp = u % a.QP, c = u / a.QP;
        const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
        if (qp != have) {
          if (!mbar_wait_warp(A_FULL, na & 1, abort_flag)) break;
          tc_fence_after();
          ++na;
          have = qp;
        }
        for (int p = p0; p < p1; ++p) {
          if (!mbar_wait_warp(ACC_EMPTY(b), acc_ph, abort_flag)) { ok = false; break; }
          const uint32_t d_tmem = tmem + (uint32_t)(b * H_ACC_COL);
#pragma unroll
          for (int kc = 0; kc < KC; ++kc) {
            if (!mbar_wait_warp(FULL(st), ph, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t b_lo = b_lo0 + (uint32_t)st * (LY::B_BYTES >> 4);
#pragma unroll
            for (int kk = 0; kk < H_CHUNK / 32; ++kk)  // 32 bytes a step: K = 64
              if (4 * kc + kk < a.ksteps) umma_mxf4<CL>(d_tmem, smem_desc_of(a_lo + kc * (BM * H_CHUNK >> 4) + 2 * kk), smem_desc_of(b_lo + 2 * kk),
                            idesc, tmem + (uint32_t)H_SF_COL, (kc > 0 || kk > 0) ? 1u : 0u,
                            leader);
            commit(EMPTY(st));
            if (++st == STAGES) {
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
        if (u + ncl < U && (u + ncl) % a.QP != qp) commit(A_EMPTY);
      }
      commit(DONE);
    }
    // drain: all issued MMAs complete before TMEM is released
    mbar_wait(DONE, 0, abort_flag, true);
    __syncwarp();
  } else if (BITS && warp >= 4 && (warp & 2)) {
    // ---------------- expansion of the base tiles' words ----------------
    const int r = (((warp - 4) >> 2) * 2 + (warp & 1)) * 32 + lane;  // row of the tile
    if (r < HN) {  // warp-uniform: HN / 32 of the eight warps
      uint4 w[2 * KC];
      auto fetch = [&](int p, int i) {
        const int64_t row = (int64_t)p * a.dstride * HN + r;
        w[i] = row < a.n && i < a.wq ? __ldg(a.xst + ((row >> 7) * a.wq + i) * 128 + (row & 127)) : make_uint4(0, 0, 0, 0);
      };
      auto first = [&](int u) { return u / a.QP * a.CH; };
#pragma unroll
      for (int i = 0; i < 2 * KC; ++i) fetch(first(cid), i);
      int st = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int u = cid; u < U && ok; u += ncl) {
        const int p0 = first(u), p1 = min(a.NP, p0 + a.CH);
        for (int p = p0; p < p1 && ok; ++p) {
          const int next = p + 1 < p1 ? p + 1 : u + ncl < U ? first(u + ncl) : -1;
#pragma unroll
          for (int kc = 0; kc < KC; ++kc) {
            if (!mbar_wait_warp(EMPTY(st), ph, abort_flag)) { ok = false; break; }
            const uint32_t dst = s0 + LY::B_OFF + st * LY::B_BYTES + (uint32_t)r * H_CHUNK;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint4 c = w[2 * kc + i];
              if (next >= 0) fetch(next, 2 * kc + i);
              const uint32_t bits[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const uint4 o = expand_word(bits[e]);
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(
                                 dst + (uint32_t)(((4 * i + e) ^ (r & 7)) * 16)),
                             "r"(o.x), "r"(o.y), "r"(o.z), "r"(o.w)
                             : "memory");
              }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read what was stored
            __syncwarp();
            if (lane == 0) mbar_arrive(FULL(st));
            if (++st == STAGES) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    const int g = (warp - 4) >> 2;         // warpgroup: columns [56g, 56g + 56) of every accumulator
    const int r = (warp & 3) * 32 + lane;  // query row within the tile = TMEM lane
    const uint32_t tbase = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * HW);
    const uint32_t at0 = s0 + LY::S_OFF + (uint32_t)(g * SBUF * BM + r) * 4u;
    const uint32_t at_lim = at0 + (uint32_t)(SBUF - 8) * (BM * 4u);  // beyond: no room for a group of 8 more
    uint32_t at = at0;
    int ia = 0;
    bool ok = true;
    for (int u = cid; u < U && ok; u += ncl) {
      const int qp = u % a.QP, c = u / a.QP;
      const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
      const int q = (CL * qp + rank) * BM + r;
      const int id0 = p0 * HN;  // base id of offset 0 (MODE_FILTER scans every tile; n < 2^31)
      float tau = INFINITY;
      if (MODE == MODE_FILTER && q < a.nq) tau = a.tau ? a.tau[q] : -INFINITY;
      auto flush = [&] {
        if (at > at0)
          h_flush(a.cnt + q, a.cand + (int64_t)q * a.cap, a.cap, at0, (int)((at - at0) / (BM * 4u)), id0);
        at = at0;
        __syncwarp();
      };
      for (int p = p0; p < p1; ++p) {
        const int b = ia & 1, ub = ia >> 1;
        // warp-uniform, so that a warp which gives up leaves its votes together
        if (!mbar_wait_warp(ACC_FULL(b), ub & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        uint32_t v[HW];
        tmem_ld56(tbase + (uint32_t)(b * H_ACC_COL), v);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {  // scores are in registers: the MMA may reuse the buffer
          if (CL > 1) mbar_arrive_cluster(cluster_addr(ACC_EMPTY(b), 0));
          else mbar_arrive(ACC_EMPTY(b));
        }
        ++ia;
        const int64_t cbase = (int64_t)p * a.dstride * HN + g * HW;  // base id of v[0]
        if (cbase + HW > a.n) {  // last base tile: padding rows become NaN, which no maximum or compare takes
#pragma unroll
          for (int j = 0; j < HW; ++j)
            if (cbase + j >= a.n) v[j] = 0x7fc00000u;
        }
        float m[7];
#pragma unroll
        for (int gg = 0; gg < 7; ++gg) m[gg] = max8(v, gg);
        const float tm = max3f(max3f(m[0], m[1], m[2]), max3f(m[3], m[4], m[5]), m[6]);
        if (MODE == MODE_GROUPMAX) {
          const int piece = 4 * p + g;
          if (q < a.nq) {  // a group of padding only is NaN: stored as -inf, not a score
            if (GW == HW) {
              a.gmax[(int64_t)q * a.M + piece] = fmaxf(tm, -INFINITY);
            } else {  // 7 groups and an empty slot: rows of 16-byte stores
              float4* dst = reinterpret_cast<float4*>(a.gmax + (int64_t)q * a.M + 8 * piece);
              dst[0] = make_float4(fmaxf(m[0], -INFINITY), fmaxf(m[1], -INFINITY), fmaxf(m[2], -INFINITY),
                                   fmaxf(m[3], -INFINITY));
              dst[1] = make_float4(fmaxf(m[4], -INFINITY), fmaxf(m[5], -INFINITY), fmaxf(m[6], -INFINITY), -INFINITY);
            }
          }
        } else if (__any_sync(0xffffffffu, tm >= tau)) {
          const uint32_t off = (uint32_t)((p - p0) * HN + g * HW);
#pragma unroll
          for (int gg = 0; gg < 7; ++gg) {
            if (!__any_sync(0xffffffffu, m[gg] >= tau)) continue;
            if (__any_sync(0xffffffffu, at > at_lim)) flush();
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) h_push(v[8 * gg + jj], tau, at, off + (uint32_t)(8 * gg + jj));
          }
        }
      }
      if (MODE == MODE_FILTER) flush();  // the next unit counts its offsets from another tile, often for another query
    }
  }

  tc_fence_before();
  if (CL > 1) cluster_sync();  // both CTAs are done with TMEM and with each other's barriers
  else __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc<CL>(tmem, H_TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(a.err, 2);
  if (CL > 1) cluster_sync();  // a pair leaves together
}

// ---- projections kernel (tc_signs_kernel) -------------------------------------------------
// Shared-memory layout for split-BF16 rows of KC chunks.
template <int KC>
struct PLayout {
  static constexpr int A_BYTES = KC * BM * H_CHUNK;  // resident point tile
  static constexpr int B_BYTES = PN * H_CHUNK;       // one chunk of a plane tile: 32 KB
  static constexpr int STAGES = KC <= 4 ? 4 : 3;
  static constexpr int A_OFF = 0;
  static constexpr int B_OFF = A_BYTES;
  static constexpr int BAR_OFF = B_OFF + STAGES * B_BYTES;
  static constexpr int SMEM = BAR_OFF + 256 + 1024;  // + barriers + alignment slack
  static_assert(SMEM <= kSmemLimit, "shared memory per CTA");
  static_assert(8 * (2 * STAGES + 2 + 2 * P_NACC + 1) + 12 <= 256, "barrier area");
};

struct SignArgs {
  int n;            // points
  int QT;           // point tiles
  int NP;           // plane tiles
  int CH;           // plane tiles a unit
  int NCH;          // chunks of them
  const float* rown;   // point norms
  const float* pnorm;  // plane norms (padded to whole tiles with zeros)
  float band;          // a sign is certain when |score| > band * |x| * |r|
  uint32_t* out32;     // [n][words] sign bits
  int words, P;        // words a point, planes (32 * words)
  uint2* list;         // [grid][list_cap] (point, plane) of the uncertain signs, a segment a CTA
  int* list_cnt;       // [grid] entries a segment (may exceed list_cap: overflow)
  int list_cap;
  int* err;
};

// Operands are BF16 (kind::f16, 64 elements a 128-byte chunk).
template <int KC>
__global__ void __launch_bounds__(H_THREADS, 1)
    tc_signs_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                      const SignArgs a) {
  grid_ready();
  using LY = PLayout<KC>;
  constexpr int STAGES = LY::STAGES;
  const int U = a.NCH * a.QT;
  if ((int)blockIdx.x >= U) return;  // no unit for this CTA: leave before any barrier or TMEM use

  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t s0 = smem_u32(sm);
  const uint32_t bar0 = s0 + LY::BAR_OFF;
  auto FULL = [&](int s) { return bar0 + 8u * s; };
  auto EMPTY = [&](int s) { return bar0 + 8u * (STAGES + s); };
  const uint32_t A_FULL = bar0 + 8u * (2 * STAGES);
  const uint32_t A_EMPTY = bar0 + 8u * (2 * STAGES + 1);
  auto ACC_FULL = [&](int b) { return bar0 + 8u * (2 * STAGES + 2 + b); };
  auto ACC_EMPTY = [&](int b) { return bar0 + 8u * (2 * STAGES + 2 + P_NACC + b); };
  const uint32_t DONE = bar0 + 8u * (2 * STAGES + 2 + 2 * P_NACC);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + LY::BAR_OFF + 8 * (2 * STAGES + 3 + 2 * P_NACC));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform for the compiler too
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(FULL(s), 1);
      mbar_init(EMPTY(s), 1);
    }
    mbar_init(A_FULL, 1);
    mbar_init(A_EMPTY, 1);
    for (int b = 0; b < P_NACC; ++b) {
      mbar_init(ACC_FULL(b), 1);
      mbar_init(ACC_EMPTY(b), H_EPI_WARPS);
    }
    mbar_init(DONE, 1);
    *abort_flag = 0;
    *reinterpret_cast<int*>(tmem_slot + 2) = 0;  // list count
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) tmem_alloc(smem_u32(tmem_slot), H_TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int it = 0, na = 0;  // base chunks and query tiles issued
      bool ok = true;
      for (int u = blockIdx.x; u < U && ok; u += gridDim.x) {
        const int qt = u % a.QT, c = u / a.QT;
        const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
        // The unit's first STAGES base chunks are issued before its query tile: their
        // stages free up as the previous unit's MMAs consume the ring, so the copies run
        // while those MMAs finish.  There is one query-tile buffer: it is reloaded once
        // the previous unit's MMAs have completed.
        const int total = (p1 - p0) * KC, pre = min(STAGES, total);
        for (int ci = 0; ci <= total; ++ci) {
          if (ci == pre) {
            if (!mbar_wait(A_EMPTY, (na & 1) ^ 1, abort_flag)) { ok = false; break; }
            mbar_expect_tx(A_FULL, LY::A_BYTES);
#pragma unroll
            for (int kc = 0; kc < KC; ++kc)
              tma_load_2d(s0 + LY::A_OFF + kc * BM * H_CHUNK, &mapA, kc * H_CHUNK, qt * BM, A_FULL);
            ++na;
          }
          if (ci == total) break;
          const int p = p0 + ci / KC, kc = ci % KC;
          const int st = it % STAGES, rd = it / STAGES;
          if (!mbar_wait(EMPTY(st), (rd & 1) ^ 1, abort_flag)) { ok = false; break; }
          mbar_expect_tx(FULL(st), LY::B_BYTES);
          tma_load_2d(s0 + LY::B_OFF + st * LY::B_BYTES, &mapB, kc * H_CHUNK, p * PN, FULL(st));
          ++it;
        }
      }
      // drain: every issued copy has landed before the CTA may exit
      for (int j = max(0, it - STAGES); j < it; ++j) mbar_wait(FULL(j % STAGES), (j / STAGES) & 1, abort_flag, true);
      if (na > 0) mbar_wait(A_FULL, (na - 1) & 1, abort_flag, true);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    {
      const uint32_t leader = elect_one();  // the warp stays converged (see elect_one)
      constexpr uint32_t idesc = idesc_bf16(BM, PN);
      int it = 0, ia = 0, ua = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < U && ok; u += gridDim.x, ++ua) {
        const int c = u / a.QT;
        const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
        if (!mbar_wait_warp(A_FULL, ua & 1, abort_flag)) break;
        tc_fence_after();
        for (int p = p0; p < p1 && ok; ++p) {
          const int b = ia % P_NACC, ub = ia / P_NACC;
          if (!mbar_wait_warp(ACC_EMPTY(b), (ub & 1) ^ 1, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d_tmem = tmem + (uint32_t)(b * PN);
          for (int kc = 0; kc < KC; ++kc) {
            const int st = it % STAGES, rd = it / STAGES;
            if (!mbar_wait_warp(FULL(st), rd & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t a_base = s0 + LY::A_OFF + kc * BM * H_CHUNK;
            const uint32_t b_base = s0 + LY::B_OFF + st * LY::B_BYTES;
#pragma unroll
            for (int kk = 0; kk < H_CHUNK / 32; ++kk) {  // 32 bytes a step: K = 16
              umma_bf16(d_tmem, smem_desc(a_base + kk * 32), smem_desc(b_base + kk * 32), idesc,
                        (kc > 0 || kk > 0) ? 1u : 0u, leader);
            }
            umma_commit(EMPTY(st), leader);
            ++it;
          }
          if (!ok) break;
          umma_commit(ACC_FULL(b), leader);
          ++ia;
        }
        umma_commit(A_EMPTY, leader);  // the query tile is free once this unit's MMAs complete
      }
      // drain: all issued MMAs complete before TMEM is released
      umma_commit(DONE, leader);
      mbar_wait(DONE, 0, abort_flag, true);
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    const int g = (warp - 4) >> 2;         // warpgroup: columns [64g, 64g+64) of every accumulator
    const int r = (warp & 3) * 32 + lane;  // query row within the tile = TMEM lane
    const uint32_t tbase = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * 64);
    int ia = 0;
    bool ok = true;
    int* seg_cnt = reinterpret_cast<int*>(tmem_slot + 2);  // this CTA's list count
    uint2* seg = a.list + (int64_t)blockIdx.x * a.list_cap;
    for (int u = blockIdx.x; u < U && ok; u += gridDim.x) {
      const int qt = u % a.QT, c = u / a.QT;
      const int p0 = c * a.CH, p1 = min(a.NP, p0 + a.CH);
      const int q = qt * BM + r;
      for (int p = p0; p < p1; ++p) {
        const int b = ia % P_NACC, ub = ia / P_NACC;
        if (!mbar_wait(ACC_FULL(b), ub & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        uint32_t v[64];
        tmem_ld64(tbase + (uint32_t)(b * PN), v);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ACC_EMPTY(b));  // scores are in registers: the MMA may reuse the buffer
        ++ia;
        const int cbase = p * PN + g * 64;  // plane of v[0]
        {
          // bit = score >= 0, as the reference's sign test; a sign within the split-BF16
          // error bound of zero is listed for the exact recheck
          if (q < a.n && cbase < a.P) {
            const float bx = a.band * a.rown[q];
            const float4* pn4 = reinterpret_cast<const float4*>(a.pnorm + cbase);
            uint32_t w0 = 0, w1 = 0;
#pragma unroll
            for (int j4 = 0; j4 < 16; ++j4) {
              const float4 pn = __ldg(pn4 + j4);
              const float pv[4] = {pn.x, pn.y, pn.z, pn.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int j = 4 * j4 + e;
                const float sc = __uint_as_float(v[j]);
                const uint32_t bit = sc >= 0.0f ? 1u : 0u;
                if (j < 32) w0 |= bit << j;
                else w1 |= bit << (j - 32);
                if (fabsf(sc) <= bx * pv[e] && cbase + j < a.P) {
                  const int pos = atomicAdd(seg_cnt, 1);
                  if (pos < a.list_cap) seg[pos] = make_uint2((uint32_t)q, (uint32_t)(cbase + j));
                }
              }
            }
            uint32_t* row = a.out32 + (int64_t)q * a.words + (cbase >> 5);
            row[0] = w0;
            if (cbase + 32 < a.P) row[1] = w1;
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem, H_TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(a.err, 2);
  if (threadIdx.x == 0) a.list_cnt[blockIdx.x] = *reinterpret_cast<int*>(tmem_slot + 2);
}

// Sketch rows of wp words (the first `words` real) -> E2M1 rows of kp bytes: 16 bytes a word
// (expand_word), 0x2 (+1) for a 0 bit, 0xA (-1) for a 1 bit; nibbles past 32 * words and rows past n
// are 0x0.
__global__ void expand_bits_kernel(const uint32_t* __restrict__ xs, int64_t n, int wp, int words, int kp,
                                   int64_t rows_pad, uint4* __restrict__ out, int* counters, int ncounters) {
  grid_ready();
  zero_counters(counters, ncounters);
  const int per_row = kp / 16;
  const int64_t total = rows_pad * per_row;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / per_row;
    const int w = (int)(t - i * per_row);
    uint4 o = make_uint4(0, 0, 0, 0);
    if (i < n && w < words) o = expand_word(xs[i * wp + w]);
    out[t] = o;
  }
}

// Top-C (C <= 128) of each query's survivors, one warp a query; a query whose survivor count
// is below `need` or above `cap` is listed in ovf (ovf[0] = count, ovf[1..] = queries).
template <int E>
__global__ void __launch_bounds__(256) hsel_warp_kernel(const int* __restrict__ cnt, const uint64_t* __restrict__ cand,
                                                        int cap, int need, int nq, uint64_t* __restrict__ out,
                                                        int* __restrict__ ovf) {
  grid_ready();
  constexpr int CT = 32 * E;
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (q >= nq) return;  // warp-uniform
  const int c = cnt[q];
  uint64_t* dst = out + (int64_t)q * CT;
  if (c > cap || c < need) {
    if (lane == 0) ovf[1 + atomicAdd(ovf, 1)] = q;
    return;  // the rescan writes this row
  }
  const uint64_t* src = cand + (int64_t)q * cap;
  uint64_t best[E];
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
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint64_t rr = __shfl_sync(0xffffffffu, x[E - 1 - e], 31 - lane);
      best[e] = best[e] < rr ? best[e] : rr;
    }
    warp_bitonic<E>(best, lane, true);
  }
#pragma unroll
  for (int e = 0; e < E; ++e) dst[e * 32 + lane] = best[e];
}

// Top-C (C > 128) of each query's survivors as a set, one block a query, using the integer
// scores: t is the score of the C-th best survivor; every survivor above t is in, and of those
// at t the ones with the lowest ids.  The set goes out unordered -- the re-rank sorts it.  Up to
// kSelRegs keys a thread, t is found by bisection over the scores held in registers, and the
// id that ends the tied ones by bisection over their ids; longer lists (bases that keep every
// point) take t from a histogram of the scores (2 * bits + 1 bins).  A query whose survivors at
// t exceed H_TIE_MAX is listed for the exact rescan, as are those with fewer than `need` or
// more than `cap` survivors.
//
// Bisection costs a compare a key and a block sum a step, about 25 steps; the histogram's
// shared-memory atomics pile up on the few scores next to the threshold (10,000 queries, C =
// 4,096, 6,500 survivors of 256-bit sketches: 825 us, by bisection 371).
constexpr int H_TIE_MAX = 4096;
constexpr int H_BINS_MAX = 2049;
constexpr int kSelRegs = 16;

// Sum over the block of each thread's c (every thread; buf alternates between calls).
template <int T>
__device__ __forceinline__ int block_sum(int c, int (&part)[2][T / 32], int buf) {
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) part[buf][threadIdx.x >> 5] = c;
  __syncthreads();
  // every warp adds the warps' sums
  const int l = threadIdx.x & 31;
  return __reduce_add_sync(0xffffffffu, l < T / 32 ? part[buf][l] : 0);
}

// One slot a lane with `in` set, from a shared counter: one atomic a warp.
__device__ __forceinline__ int warp_slot(bool in, int* counter) {
  const unsigned mk = __ballot_sync(0xffffffffu, in);
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0 && mk) base = atomicAdd(counter, __popc(mk));
  return __shfl_sync(0xffffffffu, base, 0) + __popc(mk & ((1u << lane) - 1u));
}

// T threads: 256 for C <= 1024, whose survivors they hold, else 512.
template <int T>
__global__ void __launch_bounds__(T, 1536 / T)
    hsel_kernel(const int* __restrict__ cnt, const uint64_t* __restrict__ cand, int cap, int need, int C, int bits,
                uint64_t* __restrict__ out, int* __restrict__ ovf) {
  grid_ready();
  __shared__ int tie[H_TIE_MAX];  // ids at the C-th score
  __shared__ int hist[H_BINS_MAX];
  __shared__ int part[2][T / 32];
  __shared__ int s_t, s_below, s_nout, s_ntie;
  const int q = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const int c = cnt[q];
  if (c > cap || c < need) {
    if (tid == 0) ovf[1 + atomicAdd(ovf, 1)] = q;
    return;
  }
  const uint64_t* src = cand + (int64_t)q * cap;
  uint64_t* dst = out + (int64_t)q * C;
  if (c <= C) {  // a base of fewer than C points: all of them, then empty keys
    for (int i = tid; i < C; i += T) dst[i] = i < c ? src[i] : kEmptyKey;
    return;
  }
  if (tid == 0) {
    s_nout = 0;
    s_ntie = 0;
  }
  // a key holds -score: the smallest are the best
  int thr, below;  // -(C-th score); survivors above it
  if (c <= kSelRegs * T) {
    int v[kSelRegs];
    int mn = INT_MAX, mx = INT_MIN;
#pragma unroll
    for (int e = 0; e < kSelRegs; ++e) {
      const int i = e * T + tid;
      v[e] = INT_MAX;
      if (i < c) {
        v[e] = (int)key_dist(src[i]);
        mn = min(mn, v[e]);
        mx = max(mx, v[e]);
      }
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) {
      part[0][tid >> 5] = mn;
      part[1][tid >> 5] = mx;
    }
    __syncthreads();
    int lo = __reduce_min_sync(0xffffffffu, lane < T / 32 ? part[0][lane] : INT_MAX) - 1;
    int hi = __reduce_max_sync(0xffffffffu, lane < T / 32 ? part[1][lane] : INT_MIN);
    __syncthreads();
    below = 0;  // count(<= lo) = below < C <= count(<= hi)
    for (int it = 0; hi - lo > 1; ++it) {  // block-uniform
      const int mid = lo + ((hi - lo) >> 1);
      int n = 0;
#pragma unroll
      for (int e = 0; e < kSelRegs; ++e) n += v[e] <= mid ? 1 : 0;
      n = block_sum<T>(n, part, it & 1);
      if (n >= C) {
        hi = mid;
      } else {
        lo = mid;
        below = n;
      }
    }
    thr = hi;
  } else {
    const int nb = 2 * bits + 1;
    for (int i = tid; i < nb; i += T) hist[i] = 0;
    __syncthreads();
    for (int i = tid; i < c; i += T) atomicAdd(&hist[(int)key_dist(src[i]) + bits], 1);
    __syncthreads();
    if (tid < 32) {  // the bin where the running count reaches C
      const int per = (nb + 31) / 32, b0 = lane * per, b1 = min(nb, b0 + per);
      int own = 0;
      for (int b = b0; b < b1; ++b) own += hist[b];
      int incl = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, incl >= C);
      const int L = __ffs(hit) - 1;  // hit != 0: the bins hold c > C keys
      if (lane == L) {
        int acc = incl - own;
        for (int b = b0; b < b1; ++b) {
          if (acc + hist[b] >= C) {
            s_t = b - bits;
            s_below = acc;
            break;
          }
          acc += hist[b];
        }
      }
    }
    __syncthreads();
    thr = s_t;
    below = s_below;
  }
  __syncthreads();
  for (int i0 = 0; i0 < c; i0 += T) {  // whole warps: their slots are taken together
    const int i = i0 + tid;
    const uint64_t key = i < c ? src[i] : kEmptyKey;
    const int d = i < c ? (int)key_dist(key) : INT_MAX;
    const int at = warp_slot(d < thr, &s_nout);
    if (d < thr) dst[at] = key;
    const int tt = warp_slot(d == thr, &s_ntie);
    if (d == thr && tt < H_TIE_MAX) tie[tt] = key_id(key);
  }
  __syncthreads();
  const int nt = s_ntie, want = C - below;  // 1 <= want <= nt
  if (nt > H_TIE_MAX) {  // block-uniform
    if (tid == 0) ovf[1 + atomicAdd(ovf, 1)] = q;
    return;
  }
  // the want-th lowest id of the tied ones (ids are distinct)
  int lo = -1, hi = INT_MAX - 1;  // count(id <= lo) < want <= count(id <= hi)
  if (nt > want) {
    constexpr int R = H_TIE_MAX / T;
    int v[R];
    int mx = 0;
#pragma unroll
    for (int e = 0; e < R; ++e) {
      v[e] = e * T + tid < nt ? tie[e * T + tid] : INT_MAX;
      if (v[e] != INT_MAX) mx = max(mx, v[e]);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) part[0][tid >> 5] = mx;
    __syncthreads();
    hi = __reduce_max_sync(0xffffffffu, lane < T / 32 ? part[0][lane] : 0);
    __syncthreads();
    for (int it = 0; hi - lo > 1; ++it) {
      const int mid = lo + ((hi - lo) >> 1);
      int n = 0;
#pragma unroll
      for (int e = 0; e < R; ++e) n += v[e] <= mid ? 1 : 0;
      n = block_sum<T>(n, part, it & 1);
      if (n >= want) hi = mid;
      else lo = mid;
      if (n == want) break;  // exactly the ids up to mid
    }
  }
  const float dist = (float)thr;
  for (int i0 = 0; i0 < nt; i0 += T) {
    const int i = i0 + tid;
    const bool in = i < nt && tie[i] <= hi;
    const int at = warp_slot(in, &s_nout);  // s_nout == below
    if (in) dst[at] = make_key(dist, tie[i]);
  }
}

// Rows of kp bytes (a multiple of 128); boxes of 128 bytes x box_rows rows, 128-byte swizzle.
CUtensorMap map_sketch_rows(const void* base, int64_t rows, int kp, int box_rows) {
  LSHG_REQUIRE(((uintptr_t)base & 15) == 0 && kp % H_CHUNK == 0, "sketch rows: 16-byte base, 128-byte rows");
  return make_map_bytes(base, rows, kp, box_rows);
}

template <int MODE, int GW, int KC, int CL, bool BITS>
void run_hamming(const CUtensorMap& ma, const CUtensorMap& mb, HArgs a, const char* name, cudaStream_t s) {
  // units: long enough to amortise the query tile's reload, at least 8 a cluster
  const int G = std::max(1, num_sms() / CL);
  a.QP = ceil_div(a.QT, CL);
  const int64_t work = (int64_t)a.NP * a.QP;
  a.CH = (int)std::max<int64_t>(1, std::min<int64_t>(H_MAX_CH, (work + 8 * G - 1) / (8 * G)));
  a.NCH = ceil_div(a.NP, a.CH);
  const int grid = CL * std::min(G, a.NCH * a.QP);
  auto kern = tc_hamming_kernel<MODE, GW, KC, CL, BITS>;
  constexpr int smem = HLayout<KC, CL>::SMEM;
  raise_smem_limit(kern, smem);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(H_THREADS);
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
  LSHG_CUDA(cudaLaunchKernelEx(&cfg, kern, ma, mb, a));
  count_launch();
}

// cl: CTAs a cluster (1 when a.xst is set); mb's boxes hold a CTA's share of a base tile (HN / cl rows).
template <int MODE, int GW>
void run_hamming_kc(int kc, int cl, const CUtensorMap& ma, const CUtensorMap& mb, const HArgs& a, const char* name,
                    cudaStream_t s) {
  const int form = a.xst ? 2 : cl - 1;
  switch (kc * 3 + form) {
    case 3: run_hamming<MODE, GW, 1, 1, false>(ma, mb, a, name, s); break;
    case 4: run_hamming<MODE, GW, 1, 2, false>(ma, mb, a, name, s); break;
    case 5: run_hamming<MODE, GW, 1, 1, true>(ma, mb, a, name, s); break;
    case 6: run_hamming<MODE, GW, 2, 1, false>(ma, mb, a, name, s); break;
    case 7: run_hamming<MODE, GW, 2, 2, false>(ma, mb, a, name, s); break;
    case 8: run_hamming<MODE, GW, 2, 1, true>(ma, mb, a, name, s); break;
    case 9: run_hamming<MODE, GW, 3, 1, false>(ma, mb, a, name, s); break;
    case 10: run_hamming<MODE, GW, 3, 2, false>(ma, mb, a, name, s); break;
    case 11: run_hamming<MODE, GW, 3, 1, true>(ma, mb, a, name, s); break;
    case 12: run_hamming<MODE, GW, 4, 1, false>(ma, mb, a, name, s); break;
    case 13: run_hamming<MODE, GW, 4, 2, false>(ma, mb, a, name, s); break;
    case 14: run_hamming<MODE, GW, 4, 1, true>(ma, mb, a, name, s); break;
    default: throw Error(LSHG_ERR_INVALID_ARGUMENT, "tensor-core sketch scan: rows of 1..4 chunks of 256 bits");
  }
}

template <int KC>
void run_signs(const CUtensorMap& ma, const CUtensorMap& mb, SignArgs a, cudaStream_t s, int* grid_out) {
  const int G = num_sms();
  const int64_t work = (int64_t)a.NP * a.QT;
  a.CH = (int)std::max<int64_t>(1, std::min<int64_t>(32, (work + 8 * G - 1) / (8 * G)));
  a.NCH = ceil_div(a.NP, a.CH);
  const int grid = std::min(G, a.NCH * a.QT);
  *grid_out = grid;
  auto kern = tc_signs_kernel<KC>;
  constexpr int smem = PLayout<KC>::SMEM;
  raise_smem_limit(kern, smem);
  ProfScope _ps("tc_project_gemm", s);
  launch_next(kern, grid, H_THREADS, smem, s, ma, mb, a);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

// ---- SimHash projections on the tensor cores ---------------------------------------------
// A float v is split into two BF16 values hi = bf16(v), lo = bf16(v - hi) (the subtraction
// is exact), so v - hi - lo is within 2^-16 |v|.  Points become rows [hi | hi | lo] and
// planes [hi | lo | hi] (each part padded to kp columns), and one BF16 GEMM with K = 3 kp
// gives x_hi r_hi + x_hi r_lo + x_lo r_hi, within 3 * 2^-16 sum |x_j r_j| <= 3 * 2^-16 |x||r|
// of the exact x.r before the FP32 accumulation's own rounding.  norms: the rows' L2 norms.
__global__ void split_bf16_kernel(const float* __restrict__ x, int64_t n, int d, int kp, int64_t rows_pad, int order,
                                  __nv_bfloat16* __restrict__ out, float* __restrict__ norms) {
  grid_ready();
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = warp; i < rows_pad; i += nw) {
    __nv_bfloat16* row = out + i * 3 * kp;
    float ss = 0.0f;
    for (int j = lane; j < kp; j += 32) {
      const float v = (i < n && j < d) ? x[i * d + j] : 0.0f;
      const __nv_bfloat16 hi = __float2bfloat16_rn(v);
      const __nv_bfloat16 lo = __float2bfloat16_rn(v - __bfloat162float(hi));
      row[j] = hi;
      row[kp + j] = order == 0 ? hi : lo;
      row[2 * kp + j] = order == 0 ? lo : hi;
      ss = fmaf(v, v, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) norms[i] = sqrtf(ss);
  }
}

// Exact signs of the listed (point, plane) pairs: the reference's single-precision FMA chain
// over the dimensions in order (the same arithmetic as project_kernel), written into the
// sign bit.  A segment whose count exceeds its capacity raises *overflow.
__global__ void sign_recheck_kernel(const uint2* __restrict__ list, const int* __restrict__ cnt, int cap, int segs,
                                    const float* __restrict__ x, const float* __restrict__ planes, int d,
                                    uint32_t* __restrict__ out32, int words, int* __restrict__ overflow) {
  grid_ready();
  const int64_t total = (int64_t)segs * cap;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int seg = (int)(t / cap), i = (int)(t - (int64_t)seg * cap);
    const int c = cnt[seg];
    if (i == 0 && c > cap) atomicExch(overflow, 1);
    if (i >= c) continue;
    const uint2 e = list[t];
    const float* xr = x + (int64_t)e.x * d;
    const float* rr = planes + (int64_t)e.y * d;
    float acc = 0.0f;
    for (int j = 0; j < d; ++j) acc = __fmaf_rn(xr[j], rr[j], acc);
    uint32_t* w = out32 + (int64_t)e.x * words + (e.y >> 5);
    const uint32_t bit = 1u << (e.y & 31);
    if (acc >= 0.0f) atomicOr(w, bit);
    else atomicAnd(w, ~bit);
  }
}

}  // namespace

int signs_part_cols(int d) { return d <= 64 ? 64 : 128; }

void launch_split_bf16(const float* x, int64_t n, int d, int64_t rows_pad, int order, uint16_t* out, float* norms,
                       cudaStream_t s) {
  LSHG_REQUIRE(d >= 1 && d <= 128, "tensor-core projections: d must be <= 128");
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((rows_pad * 32 + 255) / 256, (int64_t)num_sms() * 16));
  launch_next(split_bf16_kernel, blocks, 256, 0, s, x, n, d, signs_part_cols(d), rows_pad, order,
                                           reinterpret_cast<__nv_bfloat16*>(out), norms);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

void launch_tc_signs(const float* x, int64_t n, int d, const uint16_t* planes_split, const float* pnorm,
                     const float* planes, int P, int words, uint32_t* out32, int* err, cudaStream_t s) {
  if (n <= 0) return;
  LSHG_REQUIRE(P == 32 * words && P >= 32, "tensor-core projections: whole 32-plane words");
  const int kp = signs_part_cols(d), kc = 3 * kp * 2 / H_CHUNK;
  const int64_t rows_pad = (int64_t)ceil_div(n, BM) * BM;
  const int64_t ppad = (int64_t)ceil_div(P, PN) * PN;
  LSHG_REQUIRE(rows_pad / BM * (ppad / PN) < (int64_t)INT_MAX, "tensor-core projections: problem too large");
  ProfScope _ps("tc_project", s);
  const int G = num_sms();
  DevBuf<int> cnt((size_t)G + 1, s);
  LSHG_CUDA(cudaMemsetAsync(cnt.ptr, 0, cnt.bytes(), s));
  DevBuf<uint16_t> xa((size_t)rows_pad * 3 * kp, s);
  DevBuf<float> xn((size_t)rows_pad, s);
  launch_split_bf16(x, n, d, rows_pad, 0, xa.ptr, xn.ptr, s);
  const CUtensorMap ma = map_sketch_rows(xa.ptr, rows_pad, 6 * kp, BM);
  const CUtensorMap mb = map_sketch_rows(planes_split, ppad, 6 * kp, PN);
  // about 0.1% of the signs of unit points and N(0, 1) planes fall inside the band; each
  // CTA's segment holds 4x its share, and the SIMT projection redoes everything if one
  // overflows
  const int64_t expect = (int64_t)n * P / 1000 / G + 1;
  const int cap = (int)std::min<int64_t>(1 << 22, std::max<int64_t>(4096, 4 * expect));
  DevBuf<uint2> list((size_t)G * cap, s);
  SignArgs a{};
  a.n = (int)n;
  a.QT = (int)(rows_pad / BM);
  a.NP = (int)(ppad / PN);
  a.err = err;
  a.rown = xn.ptr;
  a.pnorm = pnorm;
  a.band = 1.0f / 8192.0f;  // 2^-13: 2.7x the split's 3 * 2^-16, plus the accumulations' rounding
  a.out32 = out32;
  a.words = words;
  a.P = P;
  a.list = list.ptr;
  a.list_cnt = cnt.ptr;
  a.list_cap = cap;
  int grid = 0;
  if (kc == 3) run_signs<3>(ma, mb, a, s, &grid);
  else run_signs<6>(ma, mb, a, s, &grid);
  int* overflow = cnt.ptr + G;
  {
    const int64_t total = (int64_t)grid * cap;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, (int64_t)G * 16));
    launch_next(sign_recheck_kernel, blocks, 256, 0, s, list.ptr, cnt.ptr, cap, grid, x, planes, d, out32, words,
                overflow);
    count_launch();
    LSHG_CHECK_LAUNCH();
  }
  // an overflowing segment lost entries: the SIMT projection then redoes every sign (its
  // blocks leave at once when nothing overflowed)
  launch_project_gated(x, n, d, planes, P, words, out32, overflow, s);
}

HammingPlan plan_hamming(int64_t n, int C) {
  HammingPlan p{};
  p.ok = true;
  const int NT = ceil_div(n, HN);
  p.NT = NT;
  p.GW = 0;
  p.S = 1;
  p.NS = 0;
  p.M = 0;
  p.rank = C;
  // small base: every point survives (9 C covers what the 8-point maxima below cannot bound)
  if ((int64_t)NT * HN <= (C <= 128 ? 8192 : std::max(H_SEL_MAX, 9 * C))) {
    p.cap = NT * HN;
    return p;
  }
  for (int S : {16, 8, 4, 2, 1}) {
    const int NS = ceil_div(NT, S);
    const double m = (double)C / S;
    const int r = S == 1 ? C : std::min(C, (int)std::ceil(m + 4.0 * std::sqrt(m) + 8.0));
    for (int GW : {HW, 8}) {
      const int64_t M = (int64_t)NS * (HN / GW);  // maxima
      // about 4 r of them (28 short: a base keeps its plan when its tiles round differently)
      if (M + 28 >= 4 * (int64_t)r) {
        p.S = S;
        p.NS = NS;
        p.GW = GW;
        p.M = GW == HW ? (int)M : NS * 32;  // slots a row: 8-point groups are stored 8 a piece, 7 used
        p.rank = r;
        const int64_t want = 3 * (int64_t)r * S + 2048;
        int64_t cap = 1024;
        while (cap < want) cap <<= 1;
        if (C > 128) cap = std::min<int64_t>(cap, H_SEL_MAX);
        p.cap = (int)std::min<int64_t>(cap, (int64_t)NT * HN);
        return p;
      }
    }
  }
  // Fewer than 4 C group maxima without sampling: the C-th largest of 8-point maxima is a loose
  // bound, but while 1.1 C of them are there at most about a quarter of the points survive it
  // (60,000 points, C = 4,096: one query 185 us against 1,124 on the popcount scan, 500 414
  // against 1,538).  Below that the
  // popcount scan serves.
  if ((int64_t)NT * (HN / 8) * 10 >= 11 * (int64_t)C) {
    p.NS = NT;
    p.GW = 8;
    p.M = NT * 32;
    p.cap = (int)std::min<int64_t>(H_SEL_MAX, (int64_t)NT * HN);
    return p;
  }
  p.ok = false;
  return p;
}

int hamming_chunks(int words) { return (words + 7) / 8; }
int64_t hamming_rows(int64_t n) { return (int64_t)ceil_div(n, HN) * HN; }

void launch_expand_bits(const uint32_t* xs, int64_t n, int wp, int words, int64_t rows_pad, uint8_t* out,
                        int* counters, int ncounters, cudaStream_t s) {
  const int kp = hamming_chunks(words) * H_CHUNK;
  const int64_t total = rows_pad * (kp / 16);
  if (total <= 0) return;
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, (int64_t)num_sms() * 16);
  launch_next(expand_bits_kernel, blocks, 256, 0, s, xs, n, wp, words, kp, rows_pad, reinterpret_cast<uint4*>(out),
              counters, ncounters);
  count_launch();
  LSHG_CHECK_LAUNCH();
}

void launch_int_select(const int* cnt, const uint64_t* cand, int cap, int need, int C, int bits, int nq, uint64_t* out,
                       int* ovf, cudaStream_t s) {
  ProfScope _ps("tc_hamming_select", s);
  LSHG_REQUIRE(bits >= 1 && 2 * bits + 1 <= H_BINS_MAX, "integer select: scores of at most 1024 bits");
  // Short lists: a warp a query, or a block while every query's block is resident at once (6 an SM).  A
  // warp's chain of sorts is the longer one; blocks pay their barriers where the grid is full.  Batch
  // over 20,000 x 256 bits, C = 128, warps and blocks: 16 queries 79 and 70 us, 300 101 and 90, 1,000
  // 120 and 117, 5,000 262 and 261 (C = 32: 190 and 208).
  if (C <= 128 && nq > 6 * num_sms()) {
    if (C == 32) launch_next(hsel_warp_kernel<1>, ceil_div(nq, 8), 256, 0, s, cnt, cand, cap, need, nq, out, ovf);
    else if (C == 64) launch_next(hsel_warp_kernel<2>, ceil_div(nq, 8), 256, 0, s, cnt, cand, cap, need, nq, out, ovf);
    else launch_next(hsel_warp_kernel<4>, ceil_div(nq, 8), 256, 0, s, cnt, cand, cap, need, nq, out, ovf);
  } else {
    if (C <= 1024) launch_next(hsel_kernel<256>, nq, 256, 0, s, cnt, cand, cap, need, C, bits, out, ovf);
    else launch_next(hsel_kernel<512>, nq, 512, 0, s, cnt, cand, cap, need, C, bits, out, ovf);
  }
  count_launch();
  LSHG_CHECK_LAUNCH();
}

void launch_tc_hamming(const uint8_t* xse, int64_t n, const uint32_t* xst, int wp, int words, const uint32_t* qs,
                       int nq, int op, int C, uint64_t* out, int* err, cudaStream_t s) {
  if (nq <= 0) return;
  LSHG_REQUIRE(words >= 1 && words <= 32, "tensor-core sketch scan: 1..32 words a sketch");
  LSHG_REQUIRE(C >= 32 && C <= 4096 && (C & (C - 1)) == 0, "tensor-core sketch scan: C must be a power of two");
  const int kc = hamming_chunks(words), kp = kc * H_CHUNK;
  const int64_t qpad = (int64_t)ceil_div(nq, BM) * BM;
  const int QT = (int)(qpad / BM);
  const int64_t npad = hamming_rows(n);
  const HammingPlan plan = plan_hamming(n, C);
  LSHG_REQUIRE(plan.ok, "tensor-core sketch scan: C too large for this base");
  LSHG_REQUIRE((int64_t)QT * plan.NT < (int64_t)INT_MAX, "tensor-core sketch scan: problem too large");
  DevBuf<int> ctl((size_t)nq + 1 + nq, s);  // [0, nq): survivors; [nq]: listed queries; then their list
  int *cnt = ctl.ptr, *ovf = ctl.ptr + nq;
  DevBuf<uint8_t> qe((size_t)qpad * kp, s);
  {
    ProfScope _ps("tc_hamming_expand", s);
    launch_expand_bits(qs, nq, wp, words, qpad, qe.ptr, cnt, nq + 1, s);
  }
  const CUtensorMap ma = map_sketch_rows(qe.ptr, qpad, kp, BM);
  // clusters of two query tiles share each base tile's fetch; one tile alone would leave the
  // second CTA without work
  const int cl = QT > 1 ? 2 : 1;
  const CUtensorMap mb = map_sketch_rows(xse, npad, kp, HN / cl);
  HArgs a{};
  a.nq = nq;
  a.n = n;
  a.QT = QT;
  a.ksteps = (words + 1) / 2;
  a.err = err;
  if (nq <= H_BITS_MAX_Q) {
    a.xst = reinterpret_cast<const uint4*>(xst);
    a.wq = wp / 4;
  }
  DevBuf<float> tau(nq, s);
  if (plan.M > 0) {
    DevBuf<float> gmax((size_t)nq * plan.M, s);
    a.NP = plan.NS;
    a.dstride = plan.S;
    a.gmax = gmax.ptr;
    a.M = plan.M;
    if (plan.GW == HW) run_hamming_kc<MODE_GROUPMAX, HW>(kc, cl, ma, mb, a, "tc_hamming_prepass", s);
    else run_hamming_kc<MODE_GROUPMAX, 8>(kc, cl, ma, mb, a, "tc_hamming_prepass", s);
    // scores are integers, computed the same way in both passes: no margin
    launch_tau_select(gmax.ptr, nq, plan.M, plan.rank, 0.0f, tau.ptr, s);
  }
  const int room = survivor_room(nq, plan.cap, C);
  DevBuf<uint64_t> cand((size_t)nq * room, s);
  a.gmax = nullptr;
  a.M = 0;
  a.NP = plan.NT;
  a.dstride = 1;
  a.tau = plan.M > 0 ? tau.ptr : nullptr;
  a.cnt = cnt;
  a.cand = cand.ptr;
  a.cap = plan.cap;
  run_hamming_kc<MODE_FILTER, HW>(kc, cl, ma, mb, a, "tc_hamming", s);
  launch_int_select(cnt, cand.ptr, plan.cap, (int)std::min<int64_t>(C, n), C, 32 * words, nq, out, ovf, s);
  // listed queries: exact popcount rescan written straight into their rows of `out`
  launch_scan_bits_listed(xst, n, wp, words, 0, qs, nq, op, C, ovf, out, cand.ptr, room, s);
}

}  // namespace tc
}  // namespace lshg
