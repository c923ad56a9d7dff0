// Per-token quantisation and rank-32 down-projection of the same rows in one kernel:
//   s[m] = max(|x[m,:]|, 1e-8) / 127,  q[m,:] = round(x[m,:] / s[m]),  t[m, 0:32] = x[m,:] @ A     (deploy/int8_exec.py:382-393)
// Run as two kernels the pair reads x twice from HBM (5 bytes of traffic per element); here the second reading comes
// out of L2 and 3 bytes remain.
//
// What shapes it.  A row's scale is known only after the whole row has been seen, so a row block has to be read twice;
// for the second reading to hit L2 the rows in flight on the whole chip must stay well under its 126 MB, and for the
// tensor cores to amortise A (K x 32) a block should have at least 64 rows.  64 rows per SM would be 290 MB in flight
// at K = 15360.  So a cluster of CL CTAs shares one 64-row block, each CTA owning K / CL of the columns (CL = 8 at
// K = 15360: 36 MB in flight).  The slice of A that belongs to a CTA's columns (at most 128 KB) is loaded once and stays
// in shared memory for the whole launch: A is not re-read per block.  Row maxima (one value per row and CTA) and
// partial products t (64 x 32 per CTA) are exchanged through distributed shared memory.
//
// Roles of a CTA (704 threads):
//   warp 0       TMA producer: the A slice once, then the x tiles of its columns, 64 rows x 128 elements per stage
//   warp 1       one thread issues tcgen05.mma.kind::f16 64 x 32 x 16 into one of two 32-column accumulators
//   warps 2-5    first sweep: row maxima from the same shared-memory tiles; send them to every CTA of the cluster; then
//                send the drained partial t to its owner CTA (64 / CL rows each), and add up what the CTA owns
//   warps 6-21   second sweep: one row slice per warp and step, read back from L2, quantised, stored
// Measured, bf16, back to back over inputs rotating through HBM, against pq_lowrank_down + pq_quant_rows: 66048 x 15360
// 742 -> 665 us (4.6 TB/s of the 3 bytes per element), 66048 x 3072 160 -> 136 us, 16896 x 12288 166 -> 141 us,
// 4608 x 3072 16.0 -> 15.0 us, 512 x 12288 26.5 -> 13.2 us (the down-projection alone has eight 64-row tiles there).  The
// second sweep bounds it: its sixteen warps wait for L2, then quantise, four rows each per block; neither DRAM (48 % at K = 15360)
// nor L2 (32 %) is near its limit, a scheduler issues 0.6 instructions a cycle from its four warps, and clusters of eight leave
// 28 of the 148 SMs without a CTA.  Slower: eight
// quantising warps; the second sweep through a TMA ring of its own (two or three stages are all that fits beside A and
// cannot cover the L2 latency: 946 us at K = 15360); loading a row's registers ahead of the wait for the maxima (207 us
// at K = 3072 with clusters); reloading each chunk in place (208 us).
//
// The second sweep of block b runs while the first sweep of block b + 1 streams in.
//
// Exchange protocol.  Values travel by st.async, whose bytes complete a transaction barrier of the receiving CTA; there
// are two buffers of each kind.  A CTA sends its maxima (partial t) of block b only after it has itself read those of
// block b - 1, i.e. after every CTA has sent block b - 1, i.e. after every CTA has read block b - 2: the buffer of
// parity b is free everywhere.  Every wait is bounded (status word, abort flag); all CTAs of a cluster meet at a cluster
// barrier before any of them exits.
#include <type_traits>

#include "gemm_common.cuh"
#include "quant_common.cuh"

namespace pq {
namespace {

constexpr int QM = 64;                    // rows per block (tcgen05 M = 64)
constexpr int QKE = 64;                   // elements per TMA box row (128 bytes, one swizzle row)
constexpr int QKB = 128;                  // elements of K per stage (two boxes)
constexpr int QNC = 32;                   // columns of A
constexpr int kQBoxBytes = QM * QKE * 2;  // 8 KB
constexpr int kQABoxBytes = QNC * QKE * 2;   // 4 KB
constexpr int kQStageBytes = 2 * kQBoxBytes;
constexpr int kQMaxStages = 8;
constexpr int kMaxWarps = 4;              // row-maximum warps
constexpr int kQuantWarps = 16;
constexpr int kQDThreads = 32 * (2 + kMaxWarps + kQuantWarps);
constexpr int kRowsPerWarp = QM / kQuantWarps;
constexpr int kSliceKbMax = 16;           // K slices of a CTA: at most 2048 elements = 8 chunks of 16 bytes per lane
constexpr int kChunksPerLane = kSliceKbMax * QKB / 8 / 32;

struct QuantDownParams {
  const void* x0; const void* x1;
  int64_t ldx0, ldx1;
  int8_t* q; float* s; void* t;
  int64_t ldt;
  int32_t* status;
  int M, K, k0;                           // columns from k0 on come from the second tensor (k0 == K: one tensor)
  int kb_slice;                           // 128-element k-blocks per CTA of the cluster
  int stages;
};

__device__ __forceinline__ uint32_t cluster_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t num_clusters() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void st_async_b32(uint32_t addr, uint32_t v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];"
               ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar) : "memory");
}
// Shared memory: [A slice | x ring | t_in[2][CL][64 / CL][32] | amax_in[2][CL][64] | barriers]
template <int CL>
struct QDSmem {
  static constexpr int kTInBytes = QM * QNC * 4;               // 8 KB per buffer whatever CL is
  static constexpr int kMaxBytes = CL * QM * 4;                // per buffer
  __host__ __device__ static int a_bytes(int kb) { return kb * 2 * kQABoxBytes; }
  __host__ __device__ static int t_off(int kb, int stages) { return a_bytes(kb) + stages * kQStageBytes; }
  __host__ __device__ static int max_off(int kb, int stages) { return t_off(kb, stages) + 2 * kTInBytes; }
  __host__ __device__ static int bar_off(int kb, int stages) { return max_off(kb, stages) + 2 * kMaxBytes; }
  // full[S], empty[S], a_full, tfull[2], tempty[2], max_full[2], t_full[2], max_read, t_read
  static constexpr int kNumBars = 2 * kQMaxStages + 11;
  __host__ __device__ static int total(int kb, int stages) { return bar_off(kb, stages) + kNumBars * 8 + 24 + 1024; }
};

// TWO: the rows are the concatenation of two tensors along K.
template <typename T, int CL, bool TWO>
__global__ void __launch_bounds__(kQDThreads, 1)
pq_quant_down_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmX1,
                     const __grid_constant__ CUtensorMap tmA, const QuantDownParams p) {
  using L = QDSmem<CL>;
  constexpr int kOwnRows = QM / CL;                  // rows whose t (and scale) this CTA finishes
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* ring = smem + L::a_bytes(p.kb_slice);
  float* t_in = reinterpret_cast<float*>(smem + L::t_off(p.kb_slice, p.stages));
  float* max_in = reinterpret_cast<float*>(smem + L::max_off(p.kb_slice, p.stages));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::bar_off(p.kb_slice, p.stages));
  uint64_t* empty_bar = full_bar + kQMaxStages;
  uint64_t* a_full = empty_bar + kQMaxStages;
  uint64_t* tfull_bar = a_full + 1;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint64_t* max_full = tempty_bar + 2;
  uint64_t* t_full = max_full + 2;
  uint64_t* max_read = t_full + 2;
  uint64_t* t_read = max_read + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(full_bar + L::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const int blocks = (p.M + QM - 1) / QM;
  const int num_kb = (p.K + QKB - 1) / QKB;
  const int kb0 = static_cast<int>(rank) * p.kb_slice;
  const int kb1 = kb0 + p.kb_slice < num_kb ? kb0 + p.kb_slice : num_kb;
  const int my_kb = kb1 > kb0 ? kb1 - kb0 : 0;       // may be 0 in the last CTA of a short K
  const int stages = p.stages;
  const bool quant = p.q != nullptr;                 // without it: t only, one sweep (pq_lowrank_down)

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmX); tma_prefetch_desc(&tmX1); tma_prefetch_desc(&tmA);
    for (int s = 0; s < kQMaxStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], quant ? 1 + kMaxWarps : 1); }
    mbar_init(a_full, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], kMaxWarps);
      mbar_init(&max_full[b], 1); mbar_init(&t_full[b], 1);
    }
    mbar_init(max_read, kQuantWarps); mbar_init(t_read, kMaxWarps);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    // the receiving barriers of blocks 0 and 1
    for (int b = 0; b < 2; ++b) { mbar_arrive_expect_tx(&max_full[b], L::kMaxBytes); mbar_arrive_expect_tx(&t_full[b], L::kTInBytes); }
  }
  if (warp == 1) { tmem_alloc(tmem_holder, 64); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                 // every CTA's barriers exist before anyone sends to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const int first = static_cast<int>(cluster_id()), step = static_cast<int>(num_clusters());

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0; uint32_t phase = 0; long long issued = 0; bool ok = true;
      if (my_kb > 0) {
        mbar_arrive_expect_tx(a_full, static_cast<uint32_t>(L::a_bytes(my_kb)));
#pragma unroll 1
        for (int i = 0; i < 2 * my_kb; ++i) tma_load_2d(smem + i * kQABoxBytes, &tmA, a_full, kb0 * QKB + i * QKE, 0);
      }
#pragma unroll 1
      for (int blk = first; blk < blocks && ok; blk += step) {
#pragma unroll 1
        for (int kb = 0; kb < my_kb; ++kb) {
          if (!wait_or_abort(&empty_bar[stage], phase ^ 1u, abort_flag)) {
            report_timeout(p.status, 1, 1); *abort_flag = 1; ok = false; break;
          }
          uint8_t* xs = ring + stage * kQStageBytes;
          mbar_arrive_expect_tx(&full_bar[stage], kQStageBytes);
#pragma unroll
          for (int b = 0; b < 2; ++b) {              // boxes past the end of K are zero-filled
            const int col = (kb0 + kb) * QKB + b * QKE;
            if (col < p.k0) tma_load_2d(xs + b * kQBoxBytes, &tmX, &full_bar[stage], col, blk * QM);
            else tma_load_2d(xs + b * kQBoxBytes, &tmX1, &full_bar[stage], col - p.k0, blk * QM);
          }
          ++issued;
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      const int pending = issued < stages ? static_cast<int>(issued) : stages;
      for (int i = 0; i < pending; ++i) {            // copies in flight must land before the CTA may exit
        if (--stage < 0) { stage = stages - 1; phase ^= 1u; }
        if (!wait_or_abort(&full_bar[stage], phase, abort_flag)) {
          for (int k = 0; k < 64; ++k) __nanosleep(1000);
          break;
        }
      }
      if (my_kb > 0 && !wait_or_abort(a_full, 0u, abort_flag)) {
        for (int k = 0; k < 64; ++k) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (my_kb > 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_f16(QM, QNC, std::is_same<T, __nv_bfloat16>::value);
      int stage = 0; uint32_t phase = 0; int it = 0; bool ok = true;
      if (!wait_or_abort(a_full, 0u, abort_flag)) { report_timeout(p.status, 2, 3); *abort_flag = 1; ok = false; }
#pragma unroll 1
      for (int blk = first; blk < blocks && ok; blk += step, ++it) {
        const int buf = it & 1;
        if (!wait_or_abort(&tempty_bar[buf], (static_cast<uint32_t>(it >> 1) & 1u) ^ 1u, abort_flag)) {
          report_timeout(p.status, 2, 2); *abort_flag = 1; ok = false; break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * QNC);
#pragma unroll 1
        for (int kb = 0; kb < my_kb; ++kb) {
          if (!wait_or_abort(&full_bar[stage], phase, abort_flag)) {
            report_timeout(p.status, 2, 1); *abort_flag = 1; ok = false; break;
          }
          tc_fence_after();
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const uint64_t a_desc = make_kmajor_sw128_desc(smem_u32(ring + stage * kQStageBytes + b * kQBoxBytes));
            const uint64_t b_desc = make_kmajor_sw128_desc(smem_u32(smem + (2 * kb + b) * kQABoxBytes));
#pragma unroll
            for (int k = 0; k < QKE / 16; ++k)
              tc_mma_f16(d_tmem, a_desc + static_cast<uint64_t>(2 * k), b_desc + static_cast<uint64_t>(2 * k), idesc,
                         (kb > 0 || b > 0 || k > 0) ? 1u : 0u);
          }
          tc_commit(&empty_bar[stage]);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        tc_commit(&tfull_bar[buf]);
      }
    }
  } else if (warp < 2 + kMaxWarps) {
    // ------------------------------------------------------------------ row maxima, then partial t
    // Two threads per row: thread (row, half) reads the even or the odd 16-byte columns of the row's 128-byte box rows.
    // (A maximum does not care about the order the swizzle puts the columns in; eight neighbouring threads touch eight
    // different columns, so the reads are free of bank conflicts.)
    const int tid = threadIdx.x - 64;
    const int row = tid >> 1;
    const int quarter = warp & 3;
    const int own0 = static_cast<int>(rank) * kOwnRows;
    bool ok = true;
    int stage = 0; uint32_t phase = 0; int it = 0;
    // add up the partial t of the rows this CTA owns (fixed order: rank 0, 1, ..) and store them
    auto finish_t = [&](int blk, int iter) -> bool {
      const int buf = iter & 1;
      const bool landed = wait_or_abort(&t_full[buf], static_cast<uint32_t>(iter >> 1) & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, landed)) { report_timeout(p.status, 3, 4); *abort_flag = 1; return false; }
      const float* src = t_in + buf * (QM * QNC);
#pragma unroll 1
      for (int i = tid; i < kOwnRows * QNC / 2; i += kMaxWarps * 32) {
        const int r = i / (QNC / 2), c = (i % (QNC / 2)) * 2;
        float2 a = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < CL; ++k) {
          const float2 v = *reinterpret_cast<const float2*>(src + (k * kOwnRows + r) * QNC + c);
          a.x += v.x; a.y += v.y;
        }
        const int m = blk * QM + own0 + r;
        if (m < p.M) *reinterpret_cast<uint32_t*>(static_cast<T*>(p.t) + static_cast<int64_t>(m) * p.ldt + c) = pack2(a.x, a.y, T{});
      }
      return true;
    };
#pragma unroll 1
    for (int blk = first; blk < blocks && ok; blk += step, ++it) {
      const int buf = it & 1;
      uint32_t acc = 0u;
#pragma unroll 1
      for (int kb = 0; quant && kb < my_kb; ++kb) {
        const bool landed = wait_or_abort(&full_bar[stage], phase, abort_flag);
        if (!__all_sync(0xffffffffu, landed)) { report_timeout(p.status, 3, 1); *abort_flag = 1; ok = false; break; }
        const uint8_t* xs = ring + stage * kQStageBytes + row * 128;
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 v = *reinterpret_cast<const uint4*>(xs + b * kQBoxBytes + ((((tid & 7) + 2 * i) & 7) << 4));
            acc = absmax_chunk<T>(acc, v);
          }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[stage]);
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
      if (!ok) break;
      float amax = amax_of_packed<T>(acc);
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      if (quant && it > 0) {                         // this CTA has read the maxima of the previous block
        const bool seen = wait_or_abort(max_read, static_cast<uint32_t>(it - 1) & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, seen)) { report_timeout(p.status, 3, 5); *abort_flag = 1; ok = false; break; }
      }
      if (quant) {
        const uint32_t dst = smem_u32(max_in + (buf * CL + static_cast<int>(rank)) * QM + row), bar = smem_u32(&max_full[buf]);
#pragma unroll
        for (int k = tid & 1; k < CL; k += 2) st_async_b32(map_to_cta(dst, k), __float_as_uint(amax), map_to_cta(bar, k));
      }
      if (it > 0) {
        if (!finish_t(blk - step, it - 1)) { ok = false; break; }
        __syncwarp();
        if (lane == 0) {
          if (warp == 2) mbar_arrive_expect_tx(&t_full[(it - 1) & 1], L::kTInBytes);   // armed for block it + 1
          mbar_arrive(t_read);
        }
        const bool seen = wait_or_abort(t_read, static_cast<uint32_t>(it - 1) & 1u, abort_flag);   // all four warps have read it
        if (!__all_sync(0xffffffffu, seen)) { report_timeout(p.status, 3, 8); *abort_flag = 1; ok = false; break; }
      }
      uint32_t v[32];
      if (my_kb > 0) {
        const bool landed = wait_or_abort(&tfull_bar[buf], static_cast<uint32_t>(it >> 1) & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, landed)) { report_timeout(p.status, 3, 3); *abort_flag = 1; ok = false; break; }
        tc_fence_after();
        // a 64-row accumulator keeps rows 16 q .. 16 q + 15 in the first sixteen lanes of lane quarter q
        tmem_ld_32x32b_x32(tmem_base + static_cast<uint32_t>(buf * QNC) + (static_cast<uint32_t>(quarter * 32) << 16), v);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[buf]);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0u;
      }
      if (lane < 16) {
        const int r = quarter * 16 + lane;
        const uint32_t owner = static_cast<uint32_t>(r / kOwnRows);
        const uint32_t dst = map_to_cta(smem_u32(t_in + ((buf * CL + static_cast<int>(rank)) * kOwnRows + r % kOwnRows) * QNC), owner);
        const uint32_t bar = map_to_cta(smem_u32(&t_full[buf]), owner);
#pragma unroll
        for (int j = 0; j < 8; ++j) st_async_v4(dst + 16 * j, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3], bar);
      }
      __syncwarp();
    }
    if (ok && it > 0) finish_t(first + (it - 1) * step, it - 1);
  } else if (quant) {
    // ------------------------------------------------------------------ quantisation (second sweep)
    const int qw = warp - 2 - kMaxWarps;
    const int c_lo = kb0 * (QKB / 8) + lane;         // first 16-byte chunk of the row that this lane owns; then every 32nd
    const int c_hi = kb1 * (QKB / 8) < p.K / 8 ? kb1 * (QKB / 8) : p.K / 8;
    const int n_own = c_hi > c_lo ? (c_hi - c_lo + 31) / 32 : 0;
    const int n_first = TWO ? (p.k0 / 8 > c_lo ? (p.k0 / 8 - c_lo + 31) / 32 : 0) : kChunksPerLane;   // those before the seam
    const int n_warp = __shfl_sync(0xffffffffu, n_own, 0);
    const uint8_t* x0 = static_cast<const uint8_t*>(p.x0) + static_cast<int64_t>(c_lo) * 16;
    const uint8_t* x1 = static_cast<const uint8_t*>(p.x1) + (static_cast<int64_t>(c_lo) - p.k0 / 8) * 16;
    int it = 0;
#pragma unroll 1
    for (int blk = first; blk < blocks; blk += step, ++it) {
      const int buf = it & 1;
      {
        const bool landed = wait_or_abort(&max_full[buf], static_cast<uint32_t>(it >> 1) & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, landed)) { report_timeout(p.status, 3, 6); *abort_flag = 1; break; }
      }
      float amax = 0.0f;                             // of row qw + 16 (lane & 3) of the block
#pragma unroll
      for (int k = 0; k < CL; ++k) amax = fmaxf(amax, max_in[(buf * CL + k) * QM + qw + kQuantWarps * (lane & (kRowsPerWarp - 1))]);
      __syncwarp();
      if (lane == 0) {
        // this buffer's barrier, just seen complete, is armed for block it + 2 before this CTA can let anyone send it
        if (qw == 0) mbar_arrive_expect_tx(&max_full[buf], L::kMaxBytes);
        mbar_arrive(max_read);
      }
      // one copy of the row's code: unrolled over the rows the loop runs out of the instruction cache
#pragma unroll 1
      for (int i = 0; i < kRowsPerWarp; ++i) {
        const int r = qw + kQuantWarps * i;
        const int m = blk * QM + r;
        if (m >= p.M) break;
        const uint8_t* r0 = x0 + static_cast<int64_t>(m) * p.ldx0 * 2;
        const uint8_t* r1 = TWO ? x1 + static_cast<int64_t>(m) * p.ldx1 * 2 : r0;
        uint4 v[kChunksPerLane];
#pragma unroll
        for (int j = 0; j < kChunksPerLane; ++j) {
          if (j >= n_warp) break;                    // uniform: short slices skip the rest
          if (j < n_own) v[j] = ld_stream_v4((TWO && j >= n_first ? r1 : r0) + j * 512);
        }
        const QuantScale qs = make_quant_scale(__shfl_sync(0xffffffffu, amax, i));
        if (lane == 0 && r / kOwnRows == static_cast<int>(rank)) p.s[m] = qs.scale;
        int8_t* qrow = p.q + static_cast<int64_t>(m) * p.K + static_cast<int64_t>(c_lo) * 8;
#pragma unroll
        for (int j = 0; j < kChunksPerLane; ++j) {
          if (j >= n_warp) break;
          uint32_t lo, hi;
          quant_chunk<T>(v[j], qs, lo, hi);
          if (j < n_own) st_v2(qrow + j * 256, lo, hi);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    for (int k = 0; k < 64; ++k) __nanosleep(1000);
  }
  cluster_sync_all();                                 // nobody leaves while its peers may still send to it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 64);
  }
}

constexpr int kQDMaxSmem = 232448;

template <typename T, int CL, bool TWO>
int launch_qd(const CUtensorMap& tmX, const CUtensorMap& tmX1, const CUtensorMap& tmA, QuantDownParams p, cudaStream_t st) {
  using L = QDSmem<CL>;
  auto kern = pq_quant_down_kernel<T, CL, TWO>;
  static int max_clusters[64] = {0};
  int dev = 0;
  PQ_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return PQ_ERR_UNSUPPORTED;
  p.stages = kQMaxStages;
  while (p.stages > 3 && L::total(p.kb_slice, p.stages) > kQDMaxSmem) --p.stages;
  const int smem = L::total(p.kb_slice, p.stages);
  if (smem > kQDMaxSmem) return PQ_ERR_UNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kQDThreads, 1, 1);
  cfg.stream = st;
  cfg.attrs = attr; cfg.numAttrs = 1;
  if (max_clusters[dev] == 0) {
    PQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kQDMaxSmem));
    cfg.gridDim = dim3(static_cast<unsigned>(sm_count() / CL * CL), 1, 1);
    cfg.dynamicSmemBytes = kQDMaxSmem;
    int n = 0;
    PQ_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
    if (n <= 0) return PQ_ERR_UNSUPPORTED;
    max_clusters[dev] = n;
  }
  const int blocks = (p.M + QM - 1) / QM;
  const int clusters = blocks < max_clusters[dev] ? blocks : max_clusters[dev];
  cfg.gridDim = dim3(static_cast<unsigned>(clusters * CL), 1, 1);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  PQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmX, tmX1, tmA, p));
  return PQ_OK;
}

template <typename T, bool TWO>
int launch_qd_cl(int cl, const CUtensorMap& tmX, const CUtensorMap& tmX1, const CUtensorMap& tmA, const QuantDownParams& p,
                 cudaStream_t st) {
  switch (cl) {
    case 1: return launch_qd<T, 1, TWO>(tmX, tmX1, tmA, p, st);
    case 2: return launch_qd<T, 2, TWO>(tmX, tmX1, tmA, p, st);
    case 4: return launch_qd<T, 4, TWO>(tmX, tmX1, tmA, p, st);
    default: return launch_qd<T, 8, TWO>(tmX, tmX1, tmA, p, st);
  }
}

}  // namespace
}  // namespace pq

using namespace pq;

namespace pq {
namespace {
// Cluster size, a function of K alone so that a row's t does not depend on how many rows it is computed with: slices of
// at most twelve k-blocks (a 96 KB slice of A leaves the x ring six stages), sixteen with the largest cluster.  Slices of
// six: 512 x 3072 9.0 instead of 12.4 us, but 4608 x 3072 17.9 instead of 14.8 us and 65536 x 6144 273 instead of 255 us.
int cluster_size(int64_t K) {
  const int64_t num_kb = (K + QKB - 1) / QKB;
  int cl = 1;
  while (cl < 8 && (num_kb + cl - 1) / cl > 12) cl *= 2;
  return cl;
}
}  // namespace
// k-blocks of 128 elements that are summed in one accumulator, here and in the streaming kernel of lowrank.cu (whose rows may
// be longer than this kernel takes: those are one slice).
int lowrank_slice_blocks(int64_t K) {
  const int64_t num_kb = (K + QKB - 1) / QKB;
  if (K > 8 * kSliceKbMax * QKB) return static_cast<int>(num_kb);
  const int cl = cluster_size(K);
  return static_cast<int>((num_kb + cl - 1) / cl);
}
}  // namespace pq

namespace {
// Short rows in a launch of few: the two kernels one after the other run for less time than the one (whose set-up, exchange and
// second sweep are a chain that small blocks do not hide), but the extra launch costs the host more than that (4 us a call of the
// eager forward).  So they are taken where the launches are recorded and the host's time is not in the way: under stream capture.
// Device time of the whole forward, one launch / two, us: 154 x 640 -> 1280 14.7 / 12.3, 1024 x 1536 -> 1536 20.3 / 16.1, 8256 x 512
// -> 512 17.6 / 16.9; host time of the eager call 22.8 / 26.6.  From the row counts below on the one is ahead (16384 x 1024 -> 1024
// 47.4 / 47.3, 65536 x 640 -> 1280 132.7 / 133.0).  Codes, scales and t are the same bits either way.
bool two_launches(int64_t M, int64_t K, cudaStream_t st) {
  if (K > 1536 || M >= (K < 768 ? 65536 : 16384)) return false;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) { cudaGetLastError(); return false; }
  return capture == cudaStreamCaptureStatusActive;
}

// q == nullptr: t only
int quant_down_impl(const void* x0, int64_t K0, int64_t ldx0, const void* x1, int64_t K1, int64_t ldx1, int dtype, int64_t M,
                    const void* a_t, int64_t lda, int R, int8_t* q, float* s, void* t, int64_t ldt, void* workspace,
                    size_t ws_bytes, void* stream) {
  const int64_t K = K0 + K1;
  if (M < 0 || K0 <= 0 || K1 < 0 || M > 0x7fffff00LL || K > 0x7fffff00LL || ldx0 < K0 || lda < K || ldt < R) return PQ_ERR_SHAPE;
  if (K1 > 0 && ldx1 < K1) return PQ_ERR_SHAPE;
  if (dtype != PQ_DTYPE_BF16 && dtype != PQ_DTYPE_FP16) return PQ_ERR_DTYPE;
  if (R != QNC || K > 8 * kSliceKbMax * QKB) return PQ_ERR_UNSUPPORTED;
  if (M == 0) return PQ_OK;
  if (x0 == nullptr || a_t == nullptr || t == nullptr || (K1 > 0 && x1 == nullptr)) return PQ_ERR_NULL;
  if (K0 % 8 != 0 || ldx0 % 8 != 0 || lda % 8 != 0 || ldt % 8 != 0 || !aligned_to(x0, 16) || !aligned_to(a_t, 16) ||
      !aligned_to(t, 16) || !aligned_to(q, 8) || !aligned_to(s, 4))
    return PQ_ERR_ALIGN;
  if (K1 > 0 && (K1 % 8 != 0 || ldx1 % 8 != 0 || !aligned_to(x1, 16))) return PQ_ERR_ALIGN;
  if (K1 > 0 && K0 % QKE != 0) return PQ_ERR_UNSUPPORTED;       // the seam has to fall between two boxes
  if (workspace != nullptr && ws_bytes < PQ_GEMM_WORKSPACE_BYTES) return PQ_ERR_WORKSPACE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (q != nullptr && two_launches(M, K, st)) {
    const int rc = K1 > 0 ? pq_lowrank_down_cat(x0, K0, ldx0, x1, K1, ldx1, dtype, a_t, lda, R, t, ldt, M, workspace, ws_bytes, stream)
                          : pq_lowrank_down(x0, dtype, ldx0, a_t, lda, R, t, ldt, M, K, workspace, ws_bytes, stream);
    if (rc != PQ_OK) return rc;
    return K1 > 0 ? pq_quant_rows_cat(x0, K0, ldx0, x1, K1, ldx1, dtype, M, q, s, stream)
                  : pq_quant_rows(x0, dtype, M, K, ldx0, q, s, stream);
  }
  const bool bf16 = dtype == PQ_DTYPE_BF16;
  CUtensorMap tmX, tmX1, tmA;
  int rc = make_map16(&tmX, x0, M, K0, ldx0, QM, bf16);
  if (rc != PQ_OK) return rc;
  if (K1 > 0) {
    rc = make_map16(&tmX1, x1, M, K1, ldx1, QM, bf16);
    if (rc != PQ_OK) return rc;
  } else {
    tmX1 = tmX;
  }
  rc = make_map16(&tmA, a_t, R, K, lda, QNC, bf16);
  if (rc != PQ_OK) return rc;

  QuantDownParams p;
  p.x0 = x0; p.x1 = K1 > 0 ? x1 : x0;
  p.ldx0 = ldx0; p.ldx1 = K1 > 0 ? ldx1 : ldx0;
  p.q = q; p.s = s; p.t = t; p.ldt = ldt;
  p.status = static_cast<int32_t*>(workspace);
  p.M = static_cast<int>(M); p.K = static_cast<int>(K);
  p.k0 = static_cast<int>(K1 > 0 ? K0 : K + QKB);               // one source: nothing comes from the second
  const int cl = cluster_size(K);
  p.kb_slice = lowrank_slice_blocks(K);
  p.stages = 0;
  if (K1 > 0) {
    if (bf16) return launch_qd_cl<__nv_bfloat16, true>(cl, tmX, tmX1, tmA, p, st);
    return launch_qd_cl<__half, true>(cl, tmX, tmX1, tmA, p, st);
  }
  if (bf16) return launch_qd_cl<__nv_bfloat16, false>(cl, tmX, tmX1, tmA, p, st);
  return launch_qd_cl<__half, false>(cl, tmX, tmX1, tmA, p, st);
}
}  // namespace

namespace pq {
// Row lengths for which quantisation and down-projection are one launch (ops.QUANT_LOWRANK_K).
bool lowrank_sliced(int64_t K, int R) { return R == QNC && K >= 512 && K <= 8 * kSliceKbMax * QKB; }
// Where t alone is taken from this kernel: few and long rows, which leave most SMs without one of the streaming kernel's 64-row
// tiles.  With enough tiles that kernel is ahead (six stages of x on every SM, no exchange).  Streaming / this one, us:
// 512 x 3072 8.0 / 7.3, 2048 x 3072 8.8 / 8.6, 4608 x 3072 9.6 / 10.3, 2048 x 6144 13.8 / 9.9, 4608 x 6144 15.3 / 16.3,
// 512 x 12288 22.9 / 8.6, 4608 x 12288 27.2 / 23.4, 8256 x 12288 36.3 / 37.3, 66048 x 15360 301 / 325; 512 x 1024 4.9 / 6.7.
// The sums are the same bits either way.
bool lowrank_few_rows(int64_t M, int64_t K, int R) {
  return lowrank_sliced(K, R) && K >= 3072 && 2 * M <= K && M <= 32 * static_cast<int64_t>(sm_count());
}
int lowrank_down_sliced(const void* x0, int64_t K0, int64_t ldx0, const void* x1, int64_t K1, int64_t ldx1, int dtype,
                        const void* a_t, int64_t lda, int R, void* t, int64_t ldt, int64_t M, void* workspace, size_t ws_bytes,
                        void* stream) {
  return quant_down_impl(x0, K0, ldx0, x1, K1, ldx1, dtype, M, a_t, lda, R, nullptr, nullptr, t, ldt, workspace, ws_bytes, stream);
}
}  // namespace pq

extern "C" int pq_quant_rows_lowrank(const void* x0, int64_t K0, int64_t ldx0, const void* x1, int64_t K1, int64_t ldx1,
                                     int dtype, int64_t M, const void* a_t, int64_t lda, int R, int8_t* q, float* s, void* t,
                                     int64_t ldt, void* workspace, size_t ws_bytes, void* stream) {
  if (M > 0 && (q == nullptr || s == nullptr)) return PQ_ERR_NULL;
  return quant_down_impl(x0, K0, ldx0, x1, K1, ldx1, dtype, M, a_t, lda, R, q, s, t, ldt, workspace, ws_bytes, stream);
}
