// Mamba-2 chunk scan as a persistent, software-pipelined tcgen05 kernel (headdim 64): the codes in tensor memory, the decay on x.
//
//   out[t,p] = (C_q[t,:] . S_q[p,:]) s_C S_p exp(dA_t)  +  sum_{k<=t} cb_q[t,k] S_cb exp(dA_t - dA_k) dt_k x[k,p]  +  D x[t,p]
//                                                                                   (mamba2/chunk_scan_v2.py:120-250)
//
// The codes cb_q belong to a (batch, chunk, group) and are the same for all of its heads: a CTA walks heads of one chunk after
// another and keeps the masked lower triangle of the codes in tensor memory, as bf16 (exact), as the A operand of the causal
// product. The decay goes to the two sides of it. For a segment of rows (a chunk, or part of a row block) whose cumulative
// log-decay spans at most kSpan, with r its middle,
//   exp(dA_t - dA_k) dt_k x[k,p] = exp(dA_t - r) * ( exp(r - dA_k) dt_k x[k,p] ),
// both exponents within +-kSpan / 2 where t and k lie in the segment, the second one lower for earlier k. The bracket is
// the B operand: two bf16 pieces (16 bits, fp32's exponent range), one tile of 128 tokens at a time in a ring; the row factor
// is applied to the fp32 sum. An item therefore scales chunk x 64 values once or twice instead of building chunk^2 / 2 weights.
// Where 32 rows decay by more than the span (or dA or dt is not finite, or a step above 1024), they are summed in fp32 by the
// epilogue warps, over the k whose weight is not zero.
//
// One CTA per SM; a contiguous range of items each, so that the codes change once in a chunk's heads.
//   planner warp        span and segments of an item from dA; tiles to the scale warps, one command each
//   scale warps (8)     two teams of four, a tile of 128 tokens each in turn: x -> the two pieces, into the ring
//   MMA warp            state read (tcgen05.mma.kind::i8, M = 128, N = 64) once per 128 rows, then the tiles of a segment
//                       (kind::f16 on bf16, A in tensor memory, B = tile pieces, channel index contiguous)
//   epilogue warps (8)  when the chunk or the group changes: its codes -> tensor memory. Per segment: both accumulators, row
//                       factors, D x; the fp16 row is written over the x row
//   producer warp       TMA loads of item i + stages (x tile as it lies in memory, state, dA and dt rows), TMA store of the output
// Segments go from the last rows of the chunk to the first: the tiles of a segment read x rows up to its own end only,
// so its epilogue may overwrite its rows while earlier ones are still being scaled.
// Every wait is bounded. A role whose wait runs out raises the status word and leaves its loop; the roles that depend on
// it run into their own limits and leave too; the MMA warp waits for its products, the producer for its copies.
//
// Bound by the latency and the instruction issue of its roles (an item is handed on six times: plan, tile, products, segment,
// output, stage), not by memory or the tensor core. At 8 x 16384 tokens x 80 heads, d_state 128, chunk 256, bf16: 950 us, where the
// kernel that builds the weights (lq_ssd_scan_tc.cu) takes 1303; at 2 x 4096 x 80: 80 (93). Measured on the way there: all scale
// warps on one 64-token tile 1638, a warp pair per tile 1311, a leaner issuer 1193, 128-token tiles and sixteen epilogue warps 1073,
// eight of them 995 with two CTAs on the heads of a chunk (the codes change twice as often) and 950 with one.
#include <type_traits>

#include "lq_tc.cuh"

namespace lq {

namespace scancodes {

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ float lds_f(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];\n" ::"l"(reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
// plain (untiled) bulk copy global -> shared: both addresses 16-byte aligned, size a multiple of 16 bytes
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// the registers of two loads, from here on valid
__device__ __forceinline__ void tmem_wait(uint32_t (&a)[8], uint32_t (&b)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]), "+r"(b[0]), "+r"(b[1]),
                 "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7])::"memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// A in tensor memory (bf16, two consecutive k per column), B in shared memory, fp32 accumulator
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ float exp_decay(float x) {  // ex2.approx.ftz(x log2 e): decay factors, a denormal may be zero
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(__fmul_rn(x, 1.4426950408889634f)));
  return y;
}
// two fp32 values -> two bf16, an infinity to the largest finite value: with the remainder piece it is infinite again where its
// code is not zero, and rows above the diagonal (code 0) stay what they are
__device__ __forceinline__ uint32_t pack_bf16_sat(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;\n" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ uint32_t bmul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t bfma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;\n" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t bmax_abs2(uint32_t a, uint32_t b) {  // larger magnitudes (with some sign), NaN if either is
  uint32_t d;
  asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// a value all lanes hold alike, in a uniform register: tensor-core instructions take their operands from those
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __reduce_or_sync(0xffffffffu, v); }
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0u;
}
// Bounded wait on an mbarrier phase. Each probe may suspend the thread for up to the hinted time (so a waiting role does not
// spin through the issue slots of the working ones); 2^13 probes of at most 50 us bound the wait to well under a second.
__device__ __forceinline__ bool mbar_wait_suspending(uint32_t bar, uint32_t parity) {
  for (int it = 0; it < (1 << 13); ++it) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(bar), "r"(parity), "r"(50000u) : "memory");
    if (done) return true;
  }
  return false;
}
// by every lane (each needs its own acquire of the barrier's phase), warp-uniform result; one non-suspending probe first
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  if (__all_sync(0xffffffffu, done != 0u)) return true;
  return __all_sync(0xffffffffu, mbar_wait_suspending(bar, parity) ? 1 : 0) != 0;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}

constexpr int kEpi = 8, kProducerWarp = 8 + kEpi, kMmaWarp = 9 + kEpi, kPlanWarp = 10 + kEpi;
constexpr int kThreads = 32 * (11 + kEpi);  // 8 scale warps, epilogue warps, producer, MMA issuer, planner
constexpr int kFBufs = 3;        // fp32 accumulators of segments in flight
constexpr int kJobs = 16;        // segment descriptors: the scale warps run at most kRing tiles + kFBufs segments + 1 ahead
constexpr float kSpan = 120.f;   // exp(60) * dt * x * 127 * 256 stays below fp32's range for dt <= 1024, |x| < 1e5

template <int C_, int N_>
struct ScanCfg {
  static constexpr int C = C_, N = N_, MB = (C + 127) / 128, G32 = C / 32;
  static constexpr int kX = C * 128, kS = 64 * N;
  static constexpr int kOffS = kX, kOffDa = kX + kS, kOffDt = kOffDa + C * 4;  // and in the last KB the state scales and D of the head
  static constexpr int kOffSs = kOffDt + C * 4, kOffD = kOffSs + 256, kStage = (kOffD + 256 + 1023) / 1024 * 1024;
  static constexpr int kStages = 3;
  static constexpr int kTile = C < 128 ? C : 128;  // tokens of a tile; its low pieces, then its high pieces
  static constexpr int kRing = 2, kSlot = 256 * kTile;
  static constexpr int kQc = MB * 128 * N;
  static constexpr int oQc = kStages * kStage, oRing = oQc + kQc, oZero = oRing + kRing * kSlot;
  static constexpr int oCmd = oZero + 128, oDesc = oCmd + 32 * kRing, oJobs = oDesc + 16, oBars = oJobs + 16 * kJobs;
  enum {
    FULL = 0, OUT_READY = FULL + kStages, RING_FULL = OUT_READY + kStages, CMD_EMPTY = RING_FULL + kRing, CMD_FULL = CMD_EMPTY + kRing,
    RING_EMPTY = CMD_FULL + kRing, ACC_FULL = RING_EMPTY + kRing, ACC_EMPTY = ACC_FULL + kFBufs, I_EMPTY = ACC_EMPTY + kFBufs,
    QC_FULL = I_EMPTY + 2, QC_FREE, A_READY, E_SYNC, DRAIN, kBars
  };
  static constexpr int oTbase = oBars + 8 * kBars;
  static constexpr int kBytes = oTbase + 16 + 1024;  // + alignment slack
  static_assert(kRing <= 4 && kStage % 1024 == 0 && oQc % 1024 == 0 && oRing % 1024 == 0 && oZero % 16 == 0 && oCmd % 16 == 0 &&
                oJobs % 16 == 0 && oBars % 8 == 0 && kBytes <= 232448, "shared memory layout");
  // tensor memory: codes of row block 0 (64 columns), of row block 1 (128), accumulators
  static constexpr int tA = 0, tF = 64 + (MB == 2 ? 128 : 0), tI = tF + 64 * kFBufs;
  static constexpr int kTmem = 512;
};

// the items of a CTA: a contiguous range, head fastest
struct ItemWalk {
  int b, c, h, H, NC, left;
  __device__ __forceinline__ void init(int n_items, int H_, int NC_) {
    H = H_; NC = NC_;
    const int i0 = (int)((long long)n_items * blockIdx.x / gridDim.x), i1 = (int)((long long)n_items * (blockIdx.x + 1) / gridDim.x);
    left = i1 - i0;
    h = i0 % H;
    const int q = i0 / H;
    c = q % NC;
    b = q / NC;
  }
  __device__ __forceinline__ void next() {
    if (++h == H) {
      h = 0;
      if (++c == NC) { c = 0; ++b; }
    }
  }
};

// What the MMA warp does with a tile of the ring. Bits 0 - 7: column of the codes in tensor memory; accumulators, and the phase
// in which they are free (the planner counts their uses); a second accumulator when both row blocks share the tile
enum : uint32_t {
  D_FB = 8, D_IB = 10, D_FPAR = 11, D_IPAR = 12, D_FB2 = 13,  // shifts; the second accumulator's fields lie like the first's
  D_FIRST = 1u << 18, D_LAST = 1u << 19, D_IREAD = 1u << 20, D_END = 1u << 22, D_MB = 1u << 23, D_TWO = 1u << 24, D_FIRST2 = 1u << 25,
  D_LAST2 = 1u << 26, D_UP = 1u << 27, D_LOW = 1u << 28 /* halves of the tile that count */, D_QUIT = 1u << 31
};
// segment flags for the epilogue, and above them the number of the segment
enum : int { J_MB = 1, J_IBUF = 2, J_DIRECT = 4, J_IDONE = 8, J_END = 16, J_NUM = 8 };

}  // namespace scancodes

template <typename T, int C, int N>
__global__ void __launch_bounds__(scancodes::kThreads, 1) ssd_chunk_scan_codes_kernel(const __grid_constant__ CUtensorMap tm_qc,
                                                                                      const __grid_constant__ CUtensorMap tm_s,
                                                                                      const __grid_constant__ CUtensorMap tm_x,
                                                                                      const __grid_constant__ CUtensorMap tm_out, lq_ssd_problem p,
                                                                                      int* status, int n_items) {
  pdl_enter();
  using namespace scancodes;
  typedef ScanCfg<C, N> S;
  constexpr int P = 64, MB = S::MB;
  const int NC = p.L / C, hpg = p.H / p.G;
  extern __shared__ uint8_t smem_dyn[];
  const uint32_t s_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  const uint32_t s_ring = s_base + S::oRing;
  auto bar = [&](int which, int idx = 0) { return s_base + S::oBars + 8u * (which + idx); };
  auto stage = [&](int s) { return s_base + s * S::kStage; };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dmode = p.D == nullptr ? 0 : (p.D_has_hdim ? 2 : 1);
  ItemWalk w;
  w.init(n_items, p.H, NC);

  if (tid == 0) {
    for (int i = 0; i < S::kBars; ++i) {
      uint32_t n = 1;
      if (i >= S::OUT_READY && i < S::RING_FULL) n = kEpi;               // one arrival per epilogue warp
      if (i >= S::RING_FULL && i < S::CMD_FULL) n = 4;                   // the four warps of a tile
      if (i >= S::ACC_FULL && i < S::ACC_EMPTY) n = 2;                   // the products, and the issuer (segment descriptor)
      if ((i >= S::ACC_EMPTY && i < S::QC_FULL) || i == S::A_READY || i == S::E_SYNC) n = kEpi;
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar(i)), "r"(n));
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (tid >= 32 && tid < 40) sts128(s_base + S::oZero + 16 * (tid - 32), make_uint4(0u, 0u, 0u, 0u));
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(s_base + S::oTbase), "r"((uint32_t)S::kTmem) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tbase = lds_u32(s_base + S::oTbase);
  bool failed = false;
  const int n_mine = w.left;

  // Whole warps stay inside their role's loop: every lane waits, one issues.
  if (warp == kProducerWarp) {
    // ============================================================ producer: TMA loads, TMA stores
    ItemWalk st = w;
    int key = -1, n_qc = 0, issued = 0;
    for (int j = 0, s = 0; j < n_mine + S::kStages; ++j, s = s + 1 == S::kStages ? 0 : s + 1) {
      if (j >= S::kStages) {  // the stage holds item j - kStages: its output tile stands in the place of the x tile
        if (!warp_wait(bar(S::OUT_READY, s), (uint32_t)(((j / S::kStages) - 1) & 1))) { failed = true; break; }
        if (lane == 0) {
          tma_store_4d(&tm_out, stage(s), 0, st.h, st.c * C, st.b);
          asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
          asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");  // the tile has been read: the stage is free
        }
        st.next();
        __syncwarp();
      }
      if (j >= n_mine) continue;
      const int grp = p.G == 1 ? 0 : w.h / hpg;
      if (lane == 0) {
        const uint32_t sb = stage(s), fb = bar(S::FULL, s);
        mbar_expect(fb, (uint32_t)(S::kX + S::kS + 2 * C * 4 + 256 + (dmode == 2 ? 256 : 0)));
        const size_t cbase = (((size_t)w.b * p.H + w.h) * NC + w.c) * C;
        bulk_load(sb + S::kOffDa, p.dA + cbase, (uint32_t)(C * 4), fb);
        bulk_load(sb + S::kOffDt, p.dt + cbase, (uint32_t)(C * 4), fb);
        tma_load_4d(sb, &tm_x, 0, w.h, w.c * C, w.b, fb);
        bulk_load(sb + S::kOffSs, p.state_scale + w.h * P, 256u, fb);
        if (dmode == 2) bulk_load(sb + S::kOffD, p.D + w.h * P, 256u, fb);
        tma_load_2d(sb + S::kOffS, &tm_s, 0, (int)((((size_t)w.b * NC + w.c) * p.H + w.h) * P), fb);
      }
      __syncwarp();
      ++issued;
      const int k2 = (w.b * NC + w.c) * p.G + grp;
      if (k2 != key) {  // the q_C tile of the next chunk, once the state reads of the last one are complete
        if (key >= 0 && !warp_wait(bar(S::QC_FREE), (uint32_t)((n_qc - 1) & 1))) { failed = true; break; }
        if (lane == 0) {
          mbar_expect(bar(S::QC_FULL), (uint32_t)(C * N));
#pragma unroll
          for (int r0 = 0; r0 < C; r0 += 64)
            tma_load_2d(s_base + S::oQc + r0 * N, &tm_qc, grp * N, w.b * p.L + w.c * C + r0, bar(S::QC_FULL));
        }
        __syncwarp();
        ++n_qc;
        key = k2;
      }
      w.next();
    }
    if (failed) {
      if (lane == 0 && status != nullptr) atomicExch(status, 1);
      // copies still in flight must land before the CTA may exit: wait (bounded) on what was requested last
      for (int j = max(0, issued - S::kStages); j < issued; ++j) warp_wait(bar(S::FULL, j % S::kStages), (uint32_t)((j / S::kStages) & 1));
      if (n_qc > 0) warp_wait(bar(S::QC_FULL), (uint32_t)((n_qc - 1) & 1));
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");  // every store complete
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // ============================================================ MMA issuer
    const uint32_t idesc_s = idesc_i8(128, P);
    // bf16 x bf16 -> fp32, B MN-major (rows of 128 bytes are tokens)
    const uint32_t idesc_c = idesc_f16(128, P) | (1u << 7) | (1u << 10) | (1u << 16);
    const uint32_t tb = uniform(tbase);
    const uint64_t dq0 = desc_kmajor<N>(s_base + S::oQc), db0 = desc_kmajor<128>(s_ring), dst0 = desc_kmajor<N>(s_base + S::kOffS);
    int key = -1, n_qc = 0;
    uint32_t slot = 0u, rph = 0u;
    // the products of 64 tokens into one accumulator: 16 (two 8-row groups) per step, low pieces first
    auto products = [&](uint32_t tf, uint32_t ta, uint64_t db, uint32_t acc) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) umma_ts(tf, ta + 8 * ks, db + (uint64_t)(ks * (2048 >> 4)), idesc_c, ks > 0 ? 1u : acc);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) umma_ts(tf, ta + 8 * ks, db + (uint64_t)((S::kSlot / 2 + ks * 2048) >> 4), idesc_c, 1u);
    };
    auto state_read = [&](uint32_t ti, uint64_t dq, uint64_t ds) {
#pragma unroll
      for (int ks = 0; ks < N / 32; ++ks) umma_i8(ti, dq + 2 * ks, ds + 2 * ks, idesc_s, ks > 0);
    };
    for (int j = 0, s = 0; j < n_mine && !failed; ++j, s = s + 1 == S::kStages ? 0 : s + 1, w.next()) {
      if (!warp_wait(bar(S::FULL, s), (uint32_t)((j / S::kStages) & 1))) { failed = true; break; }
      const int k2 = (w.b * NC + w.c) * p.G + (p.G == 1 ? 0 : w.h / hpg);
      if (k2 != key) {
        if (key >= 0 && elect_one()) umma_commit(bar(S::QC_FREE));
        __syncwarp();
        if (!warp_wait(bar(S::QC_FULL), (uint32_t)(n_qc & 1)) || !warp_wait(bar(S::A_READY), (uint32_t)(n_qc & 1))) { failed = true; break; }
        ++n_qc;
        key = k2;
      }
      const uint64_t ds = dst0 + (uint64_t)(s * (S::kStage >> 4));
      // One warp issues everything, a few hundred cycles of tensor work per tile: what is not a product is kept short, and the
      // code small (several roles share the instruction cache)
      for (;;) {
        if (!warp_wait(bar(S::RING_FULL) + 8u * slot, rph)) { failed = true; break; }
        uint32_t d = uniform(lds_u32(s_base + S::oDesc + 4u * slot));
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint64_t db = db0 + (uint64_t)(slot * (S::kSlot >> 4));
        const bool end = (d & D_END) != 0u;
        for (;;) {
          const uint32_t fb = (d >> D_FB) & 3u, ta = tb + (d & 255u), tf = tb + S::tF + 64u * fb;
          if (d & (D_FIRST | D_IREAD)) {
            const uint32_t ib = (d >> D_IB) & 1u;
            if (!warp_wait(bar(S::ACC_EMPTY) + 8u * fb, (d >> D_FPAR) & 1u)) { failed = true; break; }
            if ((d & D_IREAD) && !warp_wait(bar(S::I_EMPTY) + 8u * ib, (d >> D_IPAR) & 1u)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if ((d & D_IREAD) && elect_one()) state_read(tb + S::tI + 64u * ib, dq0 + (uint64_t)(d & D_MB ? (128 * N) >> 4 : 0), ds);
          }
          if (elect_one()) {
            uint32_t acc = d & D_FIRST ? 0u : 1u;
            if (d & D_UP) {
              products(tf, ta + 32u, db + (uint64_t)(8192 >> 4), acc);
              acc = 1u;
            }
            if (d & D_LOW) products(tf, ta, db, acc);
            if (d & D_LAST) {
              umma_commit(bar(S::ACC_FULL) + 8u * fb);
              mbar_arrive(bar(S::ACC_FULL) + 8u * fb);  // passes on the segment descriptor
            }
            if (!(d & D_TWO)) umma_commit(bar(S::RING_EMPTY) + 8u * slot);
          }
          if (!(d & D_TWO)) break;
          // the second accumulator (row block 0): its fields take the places of the first one's
          d = ((d & 255u) - 64u) | (((d >> D_FB2) & 31u) << D_FB) | (d & D_FIRST2 ? D_FIRST | D_IREAD : 0u) | (d & D_LAST2 ? D_LAST : 0u) |
              (d & (D_UP | D_LOW));
        }
        if (failed) break;
        slot = (slot + 1u) & (S::kRing - 1);
        rph ^= slot == 0u ? 1u : 0u;
        if (end) break;
      }
    }
    if (failed && lane == 0 && status != nullptr) atomicExch(status, 1);
    if (elect_one()) umma_commit(bar(S::DRAIN));  // no product in flight when tensor memory is freed
    __syncwarp();
    warp_wait(bar(S::DRAIN), 0u);
  } else if (warp == kPlanWarp) {
    // ============================================================ planner: segments and tiles of every item, from dA
    int n = 0, fbuf = 0, icnt = 0, jobs = 0;
    uint32_t fpar = 1u;  // phase in which the next fp32 accumulator is free
    auto send = [&](uint4 c0, uint4 c1) -> bool {  // to the team of warps whose turn it is
      const int slot = n & (S::kRing - 1);
      if (!warp_wait(bar(S::CMD_EMPTY, slot), (uint32_t)(((n / S::kRing) & 1) ^ 1))) return false;
      if (lane == 0) {
        sts128(s_base + S::oCmd + 32 * slot, c0);
        sts128(s_base + S::oCmd + 32 * slot + 16, c1);
        mbar_arrive(bar(S::CMD_FULL, slot));
      }
      ++n;
      return true;
    };
    // accumulators of the next segment and of the next row block: number and phase
    auto next_f = [&]() -> uint32_t {
      const uint32_t f = (uint32_t)fbuf | (fpar << 3);
      if (++fbuf == kFBufs) { fbuf = 0; fpar ^= 1u; }
      return f;
    };
    auto state_buf = [&](int c) -> uint32_t { return ((uint32_t)(c & 1) << 2) | ((((uint32_t)c >> 1 & 1u) ^ 1u) << 4); };
    for (int j = 0, s = 0; j < n_mine && !failed; ++j, s = s + 1 == S::kStages ? 0 : s + 1) {
      if (!warp_wait(bar(S::FULL, s), (uint32_t)((j / S::kStages) & 1))) { failed = true; break; }
      const uint32_t sb = stage(s);
      // ---- lowest and highest log-decay of every 32 tokens (lanes 4 g .. hold group g) and the lowest so far
      float mn = INFINITY, mx = -INFINITY;
      if (8 * lane < C) {
        const float4 a = lds_f4(sb + S::kOffDa + 32 * lane), b = lds_f4(sb + S::kOffDa + 32 * lane + 16);
        const float4 u = lds_f4(sb + S::kOffDt + 32 * lane), v = lds_f4(sb + S::kOffDt + 32 * lane + 16);
        mn = fminf(fminf(fminf(a.x, a.y), fminf(a.z, a.w)), fminf(fminf(b.x, b.y), fminf(b.z, b.w)));
        mx = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
        const float sum = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
        const float mag = ((fabsf(u.x) + fabsf(u.y)) + (fabsf(u.z) + fabsf(u.w))) + ((fabsf(v.x) + fabsf(v.y)) + (fabsf(v.z) + fabsf(v.w)));
        if (!(fabsf(sum) < 1e30f) || !(mag <= 1024.f)) mn = -INFINITY;  // not finite, or a huge step: no segment from here on
      }
#pragma unroll
      for (int d = 1; d < 4; d <<= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, d));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
      }
      float low = mn, top = mx;  // of groups 0 .. own; of all groups
#pragma unroll
      for (int d = 4; d < 32; d <<= 1) {
        const float o = __shfl_up_sync(0xffffffffu, low, d);
        if (lane >= d) low = fminf(low, o);
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
      }
      auto at = [&](float v, int g) { return __shfl_sync(0xffffffffu, v, 4 * g); };
      const float mn64 = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, 4));      // of 64 tokens
      const float mn128 = fminf(mn64, __shfl_xor_sync(0xffffffffu, mn64, 8));  // of 128
      constexpr int G = S::G32;
      const float lo_all = at(low, G - 1);
      const bool whole = MB == 2 && top - lo_all <= kSpan;  // one segment over both row blocks: every tile is scaled once
      int g1 = G;
      bool fresh = true;  // first segment of its row block
      while (g1 > 0 && !failed) {
        const int gb = MB == 2 && !whole ? (g1 - 1) & ~3 : 0;  // first group of the row block
        const float lo = at(low, g1 - 1);
        float hi = whole ? top : at(mx, g1 - 1);
        const bool direct = !(hi - lo <= kSpan);
        int g0 = whole ? 0 : g1 - 1;
        while (!direct && g0 > gb) {
          const float h2 = fmaxf(hi, at(mx, g0 - 1));
          if (!(h2 - lo <= kSpan)) break;
          hi = h2;
          --g0;
        }
        const float r = 0.5f * (hi + lo);
        const bool done = g0 == gb;
        const int mb = whole ? 1 : gb >> 2, ktl = (32 * g1 - 1) >> 7;
        const uint32_t d = (next_f() << D_FB) | (state_buf(icnt) << D_FB) | (mb ? D_MB | 64u : 0u) | D_FIRST | (fresh ? D_IREAD : 0u);
        uint4 c1 = make_uint4(0u, 0u, 0u, 0u);
        c1.x = (uint32_t)((whole ? 128 : 32 * g0) | (32 * g1 << 16));
        c1.y = (uint32_t)(mb * J_MB | (icnt & 1) * J_IBUF | (direct ? J_DIRECT : 0) | (done ? J_IDONE : 0) | (g0 == 0 && !whole ? J_END : 0) | (jobs << J_NUM));
        ++jobs;
        uint32_t d2 = 0u;
        if (whole) {
          d2 = (next_f() << D_FB2) | (state_buf(icnt + 1) << D_FB2) | D_TWO;
          c1.z = (uint32_t)(128 << 16);
          c1.w = (uint32_t)(((icnt + 1) & 1) * J_IBUF | J_IDONE | J_END | (jobs << J_NUM));
          ++jobs;
          ++icnt;
        }
        // last tile first: row block 0 joins at the last one (its accumulators are needed late). Halves and tiles whose weights
        // are all zero in fp32 are left out.
        uint32_t once = D_FIRST | D_IREAD;
#pragma unroll 1
        for (int kt = direct ? 0 : ktl; kt >= 0 && !failed; --kt) {
          const int live = 32 * g1 - 128 * kt;  // rows of the tile that count
          const bool last = kt == 0 || (!whole && r - at(mn128, 4 * kt - 4) < -88.f);
          uint32_t e = (d + 64u * kt) & (once | ~(D_FIRST | D_IREAD));
          if (last) e |= D_LAST | (g0 == 0 ? D_END : 0u);
          if (whole && kt == 0) e |= d2 | D_FIRST2 | D_LAST2;
          const bool up = live > 64 && (kt == ktl || !(r - at(mn64, 4 * kt + 2) < -88.f));
          const bool lowh = !up || 4 * kt + 2 > g0 || !(r - at(mn64, 4 * kt) < -88.f);
          if (!direct) e |= (up ? D_UP : 0u) | (lowh ? D_LOW : 0u);
          if (!send(make_uint4(e, sb + 16384u * kt, __float_as_uint(r), (uint32_t)live), c1)) failed = true;
          once = 0u;
          if (last) break;
        }
        fresh = done;
        if (done) ++icnt;
        g1 = g0;
      }
    }
    for (int i = 0; i < S::kRing && !failed; ++i)
      if (!send(make_uint4(D_QUIT, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u))) failed = true;
    if (failed && lane == 0 && status != nullptr) atomicExch(status, 1);
  } else if (warp < 8) {
    // ============================================================ scale warps: two teams of four, a ring slot and every second tile each
    const int slot = warp >> 2, row = 32 * (warp & 3) + lane;  // a token of the tile per thread
    const uint32_t xo = row * 128, dst = s_ring + slot * S::kSlot + xo, sw = (row & 7) << 4;
    uint32_t ph = 0u;
    for (;;) {
      if (!warp_wait(bar(S::CMD_FULL, slot), ph)) { failed = true; break; }
      const uint4 c0 = lds128(s_base + S::oCmd + 32 * slot), c1 = lds128(s_base + S::oCmd + 32 * slot + 16);
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(S::CMD_EMPTY, slot));
      if (c0.x & D_QUIT) break;
      // tokens of x (128 rows at c0.y) times dt_k exp(r - dA_k) (zero from row c0.w on: those may hold outputs already) as two
      // pieces. Eight rows of a tile hold a 16-byte piece in eight different places: a thread walks its row without conflicts.
      const bool dead = row >= (int)c0.w;
      const uint32_t tile = c0.y, kb8 = (tile - s_base) % S::kStage;  // bytes into the stage: 128 per token
      const uint32_t da = tile - kb8 + S::kOffDa + (kb8 >> 5) + 4 * row;
      float wk = __fmul_rn(exp_decay(__fsub_rn(__uint_as_float(c0.z), lds_f(da))), lds_f(da + (S::kOffDt - S::kOffDa)));
      if (dead) wk = 0.f;
      const uint32_t xr = dead ? s_base + S::oZero : tile + xo;
      if (!warp_wait(bar(S::RING_EMPTY, slot), ph ^ 1u)) { failed = true; break; }
      ph ^= 1u;
      if (c0.x & (row < 64 ? D_LOW : D_UP)) {
        auto piece32 = [&](const uint4& raw, uint32_t (&hi)[4], uint32_t (&lo)[4]) {  // in fp32
          float x[8];
          Act<T>::unpack8(raw, x);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const F2 y = mul2(F2(x[2 * i], x[2 * i + 1]), F2(wk, wk));
            float y0, y1;
            y.get(y0, y1);
            hi[i] = pack_bf16_sat(y0, y1);
            sub2(y, F2(__uint_as_float(hi[i] << 16), __uint_as_float(hi[i] & 0xffff0000u))).get(y0, y1);
            lo[i] = pack_bf16_sat(y0, y1);
          }
        };
        auto put = [&](uint32_t o, const uint32_t (&hi)[4], const uint32_t (&lo)[4]) {
          sts128(dst + o, make_uint4(lo[0], lo[1], lo[2], lo[3]));
          sts128(dst + S::kSlot / 2 + o, make_uint4(hi[0], hi[1], hi[2], hi[3]));
        };
        bool in32 = !std::is_same<T, __nv_bfloat16>::value;
        if (!in32) {
          // bf16 x: the weight as two bf16 pieces; x * high piece has 16 bits, so its rounding and the remainder are exact, and the
          // remainder takes x * low piece in. Three packed operations a pair instead of eight; not with infinities (inf - inf).
          const uint32_t wh = Act<__nv_bfloat16>::pack2(wk, wk);
          const float wr = __fsub_rn(wk, __uint_as_float(wh << 16));
          const uint32_t wl = Act<__nv_bfloat16>::pack2(wr, wr);
          uint32_t big = 0u;
#pragma unroll 2
          for (uint32_t q = 0; q < 128; q += 16) {
            const uint4 raw = lds128(xr + (q ^ sw));
            const uint32_t x[4] = {raw.x, raw.y, raw.z, raw.w};
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              hi[i] = bmul2(x[i], wh);
              lo[i] = bfma2(x[i], wl, bfma2(x[i], wh, hi[i] ^ 0x80008000u));
              big = bmax_abs2(big, hi[i]);
            }
            put(q ^ sw, hi, lo);
          }
          in32 = __any_sync(0xffffffffu, (((big & 0x7fff7fffu) + 0x00800080u) & 0x80008000u) != 0u);
        }
        if (in32) {
#pragma unroll 2
          for (uint32_t q = 0; q < 128; q += 16) {
            uint32_t hi[4], lo[4];
            piece32(lds128(xr + (q ^ sw)), hi, lo);
            put(q ^ sw, hi, lo);
          }
        }
      }
      if (row == 0) {  // what the MMA warp does with the tile, and the segments that end with it
        sts_u32(s_base + S::oDesc + 4 * slot, c0.x);
        if (c0.x & D_LAST) sts128(s_base + S::oJobs + 16 * ((c1.y >> J_NUM) & (kJobs - 1)), make_uint4(c1.x & 0xffffu, c1.x >> 16, c0.z, c1.y));
        if (c0.x & D_LAST2) sts128(s_base + S::oJobs + 16 * ((c1.w >> J_NUM) & (kJobs - 1)), make_uint4(c1.z & 0xffffu, c1.z >> 16, c0.z, c1.w));
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(S::RING_FULL, slot));
    }
    if (failed && lane == 0 && status != nullptr) atomicExch(status, 1);
  } else {
    // ============================================================ epilogue warps
    const int ew = warp - 8, q4 = warp & 3, c0 = (256 / kEpi) * (ew >> 2);  // lane quadrant of tensor memory, first of its channels
    const uint32_t lane_addr = (uint32_t)(32 * q4) << 16;
    int fb = 0, jobs = 0, key = -1;
    uint32_t fph = 0u, sync_ph = 0u;
    float sC = 0.f, Scb = 0.f, D_n = 0.f;
    if (dmode == 1 && n_mine > 0) D_n = p.D[w.h];  // of the next item: requested one item ahead
    for (int j = 0, s = 0; j < n_mine && !failed; ++j, s = s + 1 == S::kStages ? 0 : s + 1) {
      if (!warp_wait(bar(S::FULL, s), (uint32_t)((j / S::kStages) & 1))) { failed = true; break; }
      const int grp = p.G == 1 ? 0 : w.h / hpg, cbi = (w.b * NC + w.c) * p.G + grp;
      if (cbi != key) {
        // ---- the codes of this chunk -> tensor memory (every product with the old ones is complete: the last item's segments
        // have been seen): the warps of a lane quadrant in turn, 64 codes of a row at a time
        key = cbi;
        sC = p.C_scale[grp];
        Scb = p.cb_scale[grp];
        const int8_t* cb = p.cb + (size_t)cbi * C * C;
#pragma unroll 1
        for (int u = ew >> 2; u < (MB == 2 ? 6 : 2); u += kEpi / 4) {
          const int mb = u < 2 ? 0 : 1, kb = u < 2 ? u : u - 2;
          const int t = 128 * mb + 32 * q4 + lane;
          if (64 * kb >= C) continue;
          uint4 raw[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            raw[i] = t < C && 64 * kb + 16 * i <= t ? __ldg(reinterpret_cast<const uint4*>(cb + (size_t)t * C + 64 * kb + 16 * i)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t wd[4] = {raw[i].x ^ 0x80808080u, raw[i].y ^ 0x80808080u, raw[i].z ^ 0x80808080u, raw[i].w ^ 0x80808080u};
            uint32_t v[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int k = 64 * kb + 16 * i + 4 * e;
              const float f0 = s8_to_float<0>(wd[e]), f1 = s8_to_float<1>(wd[e]), f2 = s8_to_float<2>(wd[e]), f3 = s8_to_float<3>(wd[e]);
              v[2 * e] = Act<__nv_bfloat16>::pack2(k <= t ? f0 : 0.f, k + 1 <= t ? f1 : 0.f);
              v[2 * e + 1] = Act<__nv_bfloat16>::pack2(k + 2 <= t ? f2 : 0.f, k + 3 <= t ? f3 : 0.f);
            }
            tmem_st8(tbase + lane_addr + S::tA + (mb ? 64 : 0) + 32 * kb + 8 * i, v);
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(S::A_READY));
      }
      const F2 D2(D_n, D_n);
      w.next();
      if (dmode == 1 && j + 1 < n_mine) D_n = p.D[w.h];
      const uint32_t sb = stage(s);
      bool end = false;
      while (!end) {
        if (!warp_wait(bar(S::ACC_FULL, fb), fph)) { failed = true; break; }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint4 job = lds128(s_base + S::oJobs + 16 * (jobs & (kJobs - 1)));
        const int flags = (int)job.w, tw = 128 * (flags & J_MB ? 1 : 0) + 32 * q4;
        const uint32_t ib = flags & J_IBUF ? 1u : 0u;
        end = (flags & J_END) != 0;
        if (tw >= (int)job.x && tw < (int)job.y) {
          const int t = tw + lane;
          const uint32_t xrow = sb + t * 128;
          const float r = __uint_as_float(job.z), dAt = lds_f(sb + S::kOffDa + 4 * t);
          const float ga = __fmul_rn(sC, exp_decay(dAt)), rf = __fmul_rn(Scb, exp_decay(__fsub_rn(dAt, r)));
          const F2 ga2(ga, ga), rf2(rf, rf);
          const uint32_t ti = tbase + lane_addr + S::tI + 64 * ib + c0, tf = tbase + lane_addr + S::tF + 64 * fb + c0;
          // 8 channels (a 16-byte piece of the row): state sums, causal sums times rf
          auto finish = [&](int q, const uint32_t (&ri)[8], const F2 (&f)[4]) {
            const uint32_t px = xrow + (((c0 / 8 + q) ^ (t & 7)) << 4);
            float x[8];
            if (dmode != 0) Act<T>::unpack8(lds128(px), x);
            uint32_t o[4];
#pragma unroll
            for (int v4 = 0; v4 < 2; ++v4) {
              const float4 cs = lds_f4(sb + S::kOffSs + 4 * c0 + 32 * q + 16 * v4);
              float4 dv;
              if (dmode == 2) dv = lds_f4(sb + S::kOffD + 4 * c0 + 32 * q + 16 * v4);
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int e = 4 * v4 + 2 * u;
                F2 v = fma2(mul2(F2((float)(int)ri[e], (float)(int)ri[e + 1]), u ? F2(cs.z, cs.w) : F2(cs.x, cs.y)), ga2, f[2 * v4 + u]);
                if (dmode != 0) v = fma2(F2(x[e], x[e + 1]), dmode == 1 ? D2 : u ? F2(dv.z, dv.w) : F2(dv.x, dv.y), v);
                float v0, v1;
                v.get(v0, v1);
                o[2 * v4 + u] = Act<__half>::pack2(v0, v1);
              }
            }
            sts128(px, make_uint4(o[0], o[1], o[2], o[3]));
          };
          if (!(flags & J_DIRECT)) {
#pragma unroll 1
            for (int q = 0; q < 32 / kEpi; ++q) {
              uint32_t ri[8], rr[8];
              tmem_ld8(ti + 8 * q, ri);
              tmem_ld8(tf + 8 * q, rr);
              tmem_wait(ri, rr);
              F2 f[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) f[i] = mul2(F2(__uint_as_float(rr[2 * i]), __uint_as_float(rr[2 * i + 1])), rf2);
              finish(q, ri, f);
            }
          } else {
            // fp32 sums over the k whose weight is not zero for every row of the warp
            float top = dAt;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
            const int8_t* cbr = p.cb + (size_t)cbi * C * C + (size_t)t * C;
#pragma unroll 1
            for (int q = 0; q < 32 / kEpi; ++q) {
              uint32_t ri[8], none[8] = {};
              tmem_ld8(ti + 8 * q, ri);
              tmem_wait(ri, none);
              F2 f[4] = {F2(0.f, 0.f), F2(0.f, 0.f), F2(0.f, 0.f), F2(0.f, 0.f)};
#pragma unroll 1
              for (int k0 = 0; k0 <= tw; k0 += 32) {
                if (k0 < tw && __all_sync(0xffffffffu, top - lds_f(sb + S::kOffDa + 4 * (k0 + lane)) < -104.f)) continue;
#pragma unroll 1
                for (int k = k0; k < k0 + 32; ++k) {
                  if (k > t) continue;
                  const float wk = __fmul_rn(__fmul_rn((float)cbr[k], exp_decay(__fsub_rn(dAt, lds_f(sb + S::kOffDa + 4 * k)))),
                                             __fmul_rn(Scb, lds_f(sb + S::kOffDt + 4 * k)));
                  float x[8];
                  Act<T>::unpack8(lds128(sb + k * 128 + (((c0 / 8 + q) ^ (k & 7)) << 4)), x);
#pragma unroll
                  for (int i = 0; i < 4; ++i) f[i] = fma2(F2(x[2 * i], x[2 * i + 1]), F2(wk, wk), f[i]);
                }
              }
              __syncwarp();
              finish(q, ri, f);
              __syncwarp();
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        if (end) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the output rows -> visible to the TMA store
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar(S::ACC_EMPTY, fb));
          if (flags & J_IDONE) mbar_arrive(bar(S::I_EMPTY, ib));
          if (end) mbar_arrive(bar(S::OUT_READY, s));
          if ((flags & J_DIRECT) && !end) mbar_arrive(bar(S::E_SYNC));
        }
        __syncwarp();
        // earlier rows, which this segment has read directly, may be overwritten when all warps are through
        if ((flags & J_DIRECT) && !end) {
          if (!warp_wait(bar(S::E_SYNC), sync_ph)) { failed = true; break; }
          sync_ph ^= 1u;
        }
        ++jobs;
        if (++fb == kFBufs) { fb = 0; fph ^= 1u; }
      }
    }
    if (failed && lane == 0 && status != nullptr) atomicExch(status, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tbase), "r"((uint32_t)S::kTmem) : "memory");
}

// ------------------------------------------------------------------------------------------------ host side
static int encode_codes_map(CUtensorMap* m, CUtensorMapDataType dt, int rank, const void* base, const cuuint64_t* gdim,
                            const cuuint64_t* gstride_bytes, const cuuint32_t* box, CUtensorMapSwizzle swizzle, const char* what) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (enc == nullptr) return fail(LQ_ERR_LAUNCH, "%s: the driver does not export cuTensorMapEncodeTiled", what);
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = enc(m, dt, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstride_bytes, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(LQ_ERR_LAUNCH, "%s: cuTensorMapEncodeTiled failed with CUresult %d", what, (int)r);
  return LQ_OK;
}

template <typename T, int C, int N>
static int launch_scan_codes(const lq_ssd_problem* p, int* status, cudaStream_t st, const CUtensorMap& tq, const CUtensorMap& ts, const CUtensorMap& tx,
                             const CUtensorMap& to, int items) {
  const int sms = sm_count();
  const cudaError_t e = launch_opt_in(ssd_chunk_scan_codes_kernel<T, C, N>, items < sms ? items : sms, scancodes::kThreads,
                                      (size_t)scancodes::ScanCfg<C, N>::kBytes, st, tq, ts, tx, to, *p, status, items);
  if (e != cudaSuccess) return fail(LQ_ERR_LAUNCH, "ssd_chunk_scan_codes_kernel: %s", cudaGetErrorString(e));
  return check_launch("ssd_chunk_scan_codes_kernel");
}
template <typename T>
static int launch_scan_codes_T(const lq_ssd_problem* p, int* status, cudaStream_t st, const CUtensorMap& tq, const CUtensorMap& ts, const CUtensorMap& tx,
                               const CUtensorMap& to, int items) {
#define LQ_SCAN(C_)                                                                                        \
  case C_: return p->N == 128 ? launch_scan_codes<T, C_, 128>(p, status, st, tq, ts, tx, to, items)        \
                              : launch_scan_codes<T, C_, 64>(p, status, st, tq, ts, tx, to, items)
  switch (p->chunk) {
    LQ_SCAN(64);
    LQ_SCAN(128);
    LQ_SCAN(192);
    default:
    LQ_SCAN(256);
  }
#undef LQ_SCAN
}

// operands that TMA and the bulk copies can address: aligned, x strides positive and below 2^40 bytes
bool chunk_scan_codes_applies(const lq_ssd_problem* p) {
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  auto stride = [](long long s) { return s > 0 && s < (1LL << 38); };
  return aligned(p->state_scale) && (p->D == nullptr || !p->D_has_hdim || aligned(p->D)) && aligned(p->out) && aligned(p->q_C) && aligned(p->passed) &&
         aligned(p->dA) && aligned(p->dt) && aligned(p->cb) && stride(p->x_stride_h) && stride(p->x_stride_t) &&
         (p->B == 1 ? stride(p->x_stride_t * p->L) : stride(p->x_stride_b));
}
// headdim 64; every tensor map covers memory of the launching GPU only
int run_chunk_scan_codes(const lq_ssd_problem* p, int* status, cudaStream_t st) {
  const int C = p->chunk, NC = p->L / C, N = p->N;
  const long long items = (long long)p->B * NC * p->H;
  if (items > 0x7fffffffLL) return fail(LQ_ERR_SHAPE, "chunk_scan: too many (batch, chunk, head) items");
  const CUtensorMapSwizzle rows = N == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  CUtensorMap tq, ts, tx, to;
  {
    const cuuint64_t gdim[2] = {(cuuint64_t)p->G * N, (cuuint64_t)p->B * p->L};
    const cuuint64_t gstr[1] = {(cuuint64_t)p->G * N};
    const cuuint32_t box[2] = {(cuuint32_t)N, 64};
    if (int e = encode_codes_map(&tq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, p->q_C, gdim, gstr, box, rows, "chunk_scan (q_C)")) return e;
  }
  {
    const cuuint64_t gdim[2] = {(cuuint64_t)N, (cuuint64_t)p->B * NC * p->H * 64};
    const cuuint64_t gstr[1] = {(cuuint64_t)N};
    const cuuint32_t box[2] = {(cuuint32_t)N, 64};
    if (int e = encode_codes_map(&ts, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, p->passed, gdim, gstr, box, rows, "chunk_scan (states)")) return e;
  }
  {
    // x [B, L, H, 64] with element strides (a view into xBC is fine: strides are multiples of 16 bytes); a batch of one
    // gets a dummy batch stride
    const cuuint64_t gdim[4] = {64, (cuuint64_t)p->H, (cuuint64_t)p->L, (cuuint64_t)p->B};
    const cuuint64_t sb = p->B > 1 ? (cuuint64_t)p->x_stride_b * 2 : (cuuint64_t)p->x_stride_t * 2 * p->L;
    const cuuint64_t gstr[3] = {(cuuint64_t)p->x_stride_h * 2, (cuuint64_t)p->x_stride_t * 2, sb};
    const cuuint32_t box[4] = {64, 1, (cuuint32_t)C, 1};
    const CUtensorMapDataType dt = p->x_dtype == LQ_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    if (int e = encode_codes_map(&tx, dt, 4, p->x, gdim, gstr, box, CU_TENSOR_MAP_SWIZZLE_128B, "chunk_scan (x)")) return e;
  }
  {
    const cuuint64_t gdim[4] = {64, (cuuint64_t)p->H, (cuuint64_t)p->L, (cuuint64_t)p->B};
    const cuuint64_t gstr[3] = {128, (cuuint64_t)p->H * 128, (cuuint64_t)p->L * p->H * 128};
    const cuuint32_t box[4] = {64, 1, (cuuint32_t)C, 1};
    if (int e = encode_codes_map(&to, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, p->out, gdim, gstr, box, CU_TENSOR_MAP_SWIZZLE_128B, "chunk_scan (out)")) return e;
  }
  if (p->x_dtype == LQ_F16) return launch_scan_codes_T<__half>(p, status, st, tq, ts, tx, to, (int)items);
  return launch_scan_codes_T<__nv_bfloat16>(p, status, st, tq, ts, tx, to, (int)items);
}

}  // namespace lq
