// Inter-chunk state pass of the linear family (none / scalar decay) on INT8 tiles.
//
// Every (k, v) element of the state is an independent scalar recurrence over the chunks,
//     carry <- carry * exp(gc_last) + dequant( sum_t kw[t,k] * vw[t,v] ),
// so the grid tiles the state: one CTA owns a 32(v) x 16 NTW(k) tile of one (batch, head) and walks the chunks,
// four warps each holding a 16 x 8 NTW sub-tile of the fp32 carry in registers. Per chunk it stores the INT8 copy
// of the carry *entering* the chunk (what the output kernel and the next chunk read), runs the INT8 write
// product on the tensor cores straight from the prologue's transposed code tiles (both operands have the token
// index contiguous, fragments are fetched with one 128-bit load per row), and folds it into the carry.
// The fragments of the next DEPTH chunks are in flight (a register ring) while the current one is being multiplied: with few
// CTAs per SM a step of the walk costs one trip to memory divided by DEPTH. Measured: 16.9 -> 7.7 us at 15 (b, h) x 37
// chunks, K = V = 64 (NTW 4, DEPTH 1 -> NTW 1, DEPTH 4); 46.6 -> 32.0 us at 32 x 64 chunks, K = V = 128, diagonal decay
// (DEPTH 1 -> 3).
//
// Reference arithmetic: zoo/simple_gla.py:46-72 (_state_body), reference.py:77-103 (fp32 carry, INT8 stored
// copy, no error feedback).  Stored-state layout: hT [BH, NT, V, K] (k contiguous) = B operand of q.S.
#include "lq_common.cuh"

namespace lq {

struct StateArgs {
  const int8_t *kwT, *vwT;
  const float *gc, *skw, *svw, *ss;
  const float* gcl;  // diagonal decay: [BH,NT,K] decay factor of the chunk, per key channel
  int8_t* hT;
  float* final_state;  // [B,H,K,V] or null
  const float* initial_state;  // [B,H,K,V] or null
  int H, NT, use_g;
};

template <int NC>
__device__ __forceinline__ void store_codes(int8_t* dst, const float (&x)[NC], float inv) {
  if constexpr (NC == 8) {
    *reinterpret_cast<uint2*>(dst) = make_uint2(q8x4_127(x[0], x[1], x[2], x[3], inv), q8x4_127(x[4], x[5], x[6], x[7], inv));
  } else {
    static_assert(NC == 2, "key channels per thread");
    *reinterpret_cast<uint16_t*>(dst) = (uint16_t)pack_sat_s8x2(q8_lower127(x[1], inv), q8_lower127(x[0], inv), 0u);
  }
}

template <int K, int V, bool DIAG, int NTW, int DEPTH>
__global__ void __launch_bounds__(128, DEPTH == 3 ? 2 : 4) zoo_state_linear_kernel(StateArgs a) {
  pdl_enter();
  constexpr int C = 64;
  constexpr int TK = K / (16 * NTW), NC = 2 * NTW;  // key tiles per head; consecutive key channels per thread
  const int vt = blockIdx.x / TK, kt = blockIdx.x % TK;
  const int bh = blockIdx.y, h = bh % a.H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, j = lane & 3;
  const int v0 = vt * 32 + (warp & 1) * 16;
  const int k0 = kt * 16 * NTW + (warp >> 1) * 8 * NTW;
  const int va = v0 + g, vb = v0 + g + 8;

  // MMA column (nt, cn) carries the physical key channel k0 + NC*(cn/2) + 2*nt + (cn%2): a thread then owns
  // NC consecutive channels k0 + NC*j .. k0 + NC*j + NC-1 of its two value rows.
  int krow[NTW];
#pragma unroll
  for (int nt = 0; nt < NTW; ++nt) krow[nt] = k0 + NC * (g >> 1) + 2 * nt + (g & 1);

  const float svw_a = a.svw[h * V + va], svw_b = a.svw[h * V + vb];
  const float iss_a = 1.0f / a.ss[h * V + va], iss_b = 1.0f / a.ss[h * V + vb];
  float skw[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) skw[i] = a.skw[h * K + k0 + NC * j + i];

  const int8_t* vw = a.vwT + (size_t)bh * a.NT * V * C;
  const int8_t* kw = a.kwT + (size_t)bh * a.NT * K * C;
  int8_t* hT = a.hT + (size_t)bh * a.NT * V * K;
  const float* gc = a.gc + (size_t)bh * a.NT * C;

  float carry_a[NC], carry_b[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) carry_a[i] = carry_b[i] = 0.f;
  if (a.initial_state != nullptr) {
    const float* is = a.initial_state + (size_t)bh * K * V;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      carry_a[i] = is[(size_t)(k0 + NC * j + i) * V + va];
      carry_b[i] = is[(size_t)(k0 + NC * j + i) * V + vb];
    }
  }

  struct Tile {
    uint4 lo, hi, b[NTW];
    float gl;
    float gk[DIAG ? NC : 1];
  } ring[DEPTH];
  const float* gcl = DIAG ? a.gcl + (size_t)bh * a.NT * K + k0 + NC * j : nullptr;
  auto fetch = [&](int c, Tile& t) {
    const int8_t* vwc = vw + (size_t)c * V * C;
    const int8_t* kwc = kw + (size_t)c * K * C;
    t.lo = __ldg(reinterpret_cast<const uint4*>(vwc + va * C + 16 * j));
    t.hi = __ldg(reinterpret_cast<const uint4*>(vwc + vb * C + 16 * j));
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt) t.b[nt] = __ldg(reinterpret_cast<const uint4*>(kwc + krow[nt] * C + 16 * j));
    if constexpr (DIAG) {
#pragma unroll
      for (int i = 0; i < NC; i += 2) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(gcl + (size_t)c * K + i));
        t.gk[i] = v.x;
        t.gk[i + 1] = v.y;
      }
    } else {
      t.gl = a.use_g ? __ldg(gc + (size_t)c * C + (C - 1)) : 0.f;
    }
  };
  auto step = [&](int c, const Tile& t) {
    // INT8 copy of the carry entering chunk c
    int8_t* hc = hT + (size_t)c * V * K;
    store_codes<NC>(hc + state_row_of_channel(va) * K + k0 + NC * j, carry_a, iss_a);
    store_codes<NC>(hc + state_row_of_channel(vb) * K + k0 + NC * j, carry_b, iss_b);
    int acc[NTW][4];
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt) {
      mma_s8_first(acc[nt], t.lo.x, t.hi.x, t.lo.y, t.hi.y, t.b[nt].x, t.b[nt].y);
      mma_s8(acc[nt], t.lo.z, t.hi.z, t.lo.w, t.hi.w, t.b[nt].z, t.b[nt].w);
    }
    float gamv[NC];
    if constexpr (DIAG) {
#pragma unroll
      for (int i = 0; i < NC; ++i) gamv[i] = t.gk[i];
    } else {
      const float gs = a.use_g ? expf(t.gl) : 1.0f;
#pragma unroll
      for (int i = 0; i < NC; ++i) gamv[i] = gs;
    }
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = 2 * nt + e;
        const float gam = gamv[i];
        const float ta = __fmul_rn(__fmul_rn((float)acc[nt][e], skw[i]), svw_a);
        const float tb = __fmul_rn(__fmul_rn((float)acc[nt][2 + e], skw[i]), svw_b);
        carry_a[i] = fmaf(carry_a[i], gam, ta);
        carry_b[i] = fmaf(carry_b[i], gam, tb);
      }
    }
  };
#pragma unroll
  for (int u = 0; u < DEPTH; ++u)
    if (u < a.NT) fetch(u, ring[u]);
  int c = 0;
  for (; c + DEPTH <= a.NT; c += DEPTH) {
#pragma unroll
    for (int u = 0; u < DEPTH; ++u) {
      const Tile cur = ring[u];
      fetch(min(c + u + DEPTH, a.NT - 1), ring[u]);
      step(c + u, cur);
    }
  }
#pragma unroll
  for (int u = 0; u < DEPTH - 1; ++u)
    if (c + u < a.NT) step(c + u, ring[u]);

  if (a.final_state != nullptr) {
    float* fs = a.final_state + (size_t)bh * K * V;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      fs[(size_t)(k0 + NC * j + i) * V + va] = carry_a[i];
      fs[(size_t)(k0 + NC * j + i) * V + vb] = carry_b[i];
    }
  }
}

int validate_zoo_problem(const lq_zoo_problem* p, bool delta, bool diagonal);

int run_state_linear_unrot(const lq_zoo_problem* p, const lq_zoo_workspace* ws, cudaStream_t st);

int run_state_linear(const lq_zoo_problem* p, const lq_zoo_workspace* ws, cudaStream_t st) {
  if (p->unrot_t != nullptr) return run_state_linear_unrot(p, ws, st);  // canonical storage: CTA spans all value channels
  StateArgs a;
  a.kwT = ws->kwT; a.vwT = ws->vwT; a.gc = ws->gc; a.skw = p->skw; a.svw = p->svw; a.ss = p->sstate;
  a.hT = ws->hT; a.final_state = p->final_state; a.initial_state = p->initial_state; a.H = p->H; a.NT = p->T / p->chunk;
  a.use_g = p->g != nullptr;
  a.gcl = ws->gcl;
  const bool diag = p->decay == LQ_DECAY_DIAGONAL;
  // Tile and prefetch depth follow from how many CTAs of 64 key channels there are, since all of them should be resident at
  // once: up to one per SM, quarter tiles (16 key channels: four times the warps, a quarter of the work in each step) with
  // four chunks in flight; up to two per SM, three chunks in flight (up to 219 registers); beyond that one in flight, which
  // keeps five CTAs per SM (at 512 CTAs two in flight in 128 registers took 59 us instead of 52).
  const long long n64 = (long long)(p->V / 32) * (p->K / 64) * p->B * p->H;
  const int sms = sm_count();
  const bool quarter = n64 <= sms, deep = n64 <= 2 * sms;
  dim3 grid((p->V / 32) * (p->K / (quarter ? 16 : 64)), p->B * p->H), block(128);
#define LQ_LAUNCH_STATE_N(KK_, VV_, DD_)                                                                \
  if (quarter) launch(zoo_state_linear_kernel<KK_, VV_, DD_, 1, 4>, grid, block, 0, st, a);             \
  else if (deep) launch(zoo_state_linear_kernel<KK_, VV_, DD_, 4, 3>, grid, block, 0, st, a);           \
  else launch(zoo_state_linear_kernel<KK_, VV_, DD_, 4, 1>, grid, block, 0, st, a)
#define LQ_LAUNCH_STATE(KK_, VV_)                                                                       \
  if (diag) { LQ_LAUNCH_STATE_N(KK_, VV_, true); }                                                      \
  else { LQ_LAUNCH_STATE_N(KK_, VV_, false); }
  if (p->K == 64 && p->V == 64) { LQ_LAUNCH_STATE(64, 64); }
  else if (p->K == 64 && p->V == 128) { LQ_LAUNCH_STATE(64, 128); }
  else if (p->K == 128 && p->V == 64) { LQ_LAUNCH_STATE(128, 64); }
  else if (p->K == 128 && p->V == 128) { LQ_LAUNCH_STATE(128, 128); }
  else return fail(LQ_ERR_UNSUPPORTED, "state: K and V must be 64 or 128");
#undef LQ_LAUNCH_STATE
#undef LQ_LAUNCH_STATE_N
  return check_launch("zoo_state_linear_kernel");
}

}  // namespace lq

extern "C" int lq_zoo_state_linear(const lq_zoo_problem* p, const lq_zoo_workspace* ws, lq_stream stream) {
  if (int e = lq::validate_zoo_problem(p, false, p && p->decay == LQ_DECAY_DIAGONAL)) return e;
  if (!ws) return lq::fail(LQ_ERR_NULL, "state: workspace descriptor is null");
  return lq::run_state_linear(p, ws, (cudaStream_t)stream);
}
