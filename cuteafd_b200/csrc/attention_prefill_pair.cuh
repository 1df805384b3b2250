// Prompt attention with two query tiles per CTA, or one where there are too few of them (rules: `pf_tiles_paged`, `pf_tiles_latent`).
//
// Of one 128-row tile, scores, softmax and P V are a chain: the tensor pipe idles under the softmax and the exponential units under the products
// (attention_mla_prefill.cu: tensor pipe active 20 to 40 %).  Here a CTA owns two neighbouring tiles A and B of one head; while A's softmax runs,
// the pipe computes B's products, over the same K and V in shared memory.  A 128 x 128 tile costs 1,024 cycles of exponentials (16 per cycle and SM)
// and, at widths 128 + 128, 1,024 of the tensor pipe, which are the two floors.
//   tensor memory   S_A, S_B [128 x 128] fp32, O_A, O_B [128 x VC 64] fp32.  A row's thread reads its whole S row into registers and writes P over
//                   it (bf16, 64 columns), the A operand of P V: no trip through shared memory, whose reads the score product already fills.
//                   P leaves in two parts, 96 and 32 keys: most of the product runs under the last exponentials.
//   shared memory   both query tiles (the A operands of the score products) and a ring of 16 KB chunks (64 columns x 128 keys), in the order K(0) V(0)
//                   K(1) V(1) .. in which they are first used and freed
//   threads         warp 0 loads, warp 1 issues, warps 4-7 and 8-11 are A's and B's softmax, one thread per query row
// Key tiles, the reference maximum's rule and every sum are those of the one-tile kernels: all of a row's values are added key after key, so
// both give the same bits.
// Measured, one-tile kernel / this one: 4096 rows of 64 heads over 4: 643 / 285 us; 2048 rows over 8192 keys of 128 latent heads: 1432 / 1127
// (a pair takes 3,650 and 4,250 cycles a key tile, 2,048 and 2,560 of them of the tensor pipe: each softmax 1,830, 440 of them the maximum, and its wait for the next scores
// 1,700 and 2,400.  One tile alone takes 3,210, of which 1,375 are that wait: the chain from the last part of P through P V and the scores, which nothing hides within a tile).
#pragma once
#include "tc_issue.cuh"

#define PP_THREADS 384
#define PP_MAX_CHUNKS 12

template <int KC, int VC>
struct PairCfg {
  static constexpr int Q_BYTES = 2 * KC * 16384, PER_TILE = KC + VC;
  static constexpr int FIT = (226 * 1024 - Q_BYTES) / 16384;
  static constexpr int NCH = FIT < PP_MAX_CHUNKS ? FIT : PP_MAX_CHUNKS;
  static constexpr int SMEM = Q_BYTES + NCH * 16384 + 512;
  static constexpr int O_COL = 256;
  static_assert(256 + 2 * VC * 64 <= 512, "scores and outputs of two tiles exceed tensor memory");
  static_assert(NCH >= PER_TILE + KC, "the next score product's keys must fit beside the tile in use");
};

// What differs between the paged and the expanded form: where a tile's rows, keys and values lie.
struct GqaPairSrc {
  using Args = GqaPrefillArgs;
  template <int KC, int VC> static constexpr bool alone() { return KC <= 2; }           // whether the rules below give such steps one tile per CTA
  static __device__ __forceinline__ int group(const Args& a) { return a.Hq / a.Hkv; }
  static __device__ __forceinline__ bool bidir(const Args& a) { return a.window < 0; }
  template <int KC>
  static __device__ __forceinline__ const bf16* q_chunk(const Args& a, int kvh, int t, int g, int c) {
    return a.q + (size_t)t * a.q_stride + (size_t)(kvh * (a.Hq / a.Hkv) + g) * (KC * 64) + c * 64;
  }
  // chunk c of key tile i (keys below KC, then values)
  template <int KC, int VC>
  static __device__ __forceinline__ void load(const Args& a, int kvh, int seq, int i, int c, uint8_t* dst, uint64_t* bar) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int pi = i * 2 + p;                            // pages past the sequence's table are read as page 0 (finite rows, masked keys)
      const int slot0 = (pi < a.max_pages ? a.page_table[(size_t)seq * a.max_pages + pi] : 0) * 64;
      if (c < KC) tma_load_3d(dst + p * 8192, a.k_map, bar, c * 64, kvh, slot0);
      else tma_load_3d(dst + p * 8192, a.v_map, bar, (c - KC) * 64, a.v_head0 + kvh, slot0);
    }
  }
  static __device__ __forceinline__ const float* sink(const Args& a) { return a.x.sink; }
  static __device__ __forceinline__ float head_factor(const Args& a, int t, int h) { return a.x.head_factor(t, h); }
  static __device__ __forceinline__ bool gated(const Args& a) { return a.x.gate && a.x.gate_values; }
  static __device__ __forceinline__ float value_factor(const Args& a, int t, int col) { return a.x.value_factor(t, col); }
};

template <int KN>
struct MlaPairSrc {
  using Args = MlaPrefillArgs;
  template <int KC, int VC> static constexpr bool alone() { return KC == KN && KN + VC <= 3; }
  static __device__ __forceinline__ int group(const Args&) { return 1; }
  static __device__ __forceinline__ bool bidir(const Args&) { return false; }
  template <int KC>
  static __device__ __forceinline__ const bf16* q_chunk(const Args& a, int head, int t, int, int c) {
    return c < KN ? a.q_nope + ((size_t)head * a.ldt + t) * (KN * 64) + c * 64 : a.q_rope + (size_t)t * a.qr_t + (size_t)head * a.qr_h + (c - KN) * 64;
  }
  template <int KC, int VC>
  static __device__ __forceinline__ void load(const Args& a, int head, int seq, int i, int c, uint8_t* dst, uint64_t* bar) {
    const int row = a.ctx_start[seq] + i * PF_KT;
    if (c < KN) tma_load_3d(dst, &a.kvb_map, bar, head * (KN + VC) * 64 + c * 64, row, 0);
    else if (c < KC) tma_load_3d(dst, &a.lat_map, bar, a.rope_col + (c - KN) * 64, row, 0);
    else tma_load_3d(dst, &a.kvb_map, bar, head * (KN + VC) * 64 + (KN + c - KC) * 64, row, 0);
  }
  static __device__ __forceinline__ const float* sink(const Args& a) { return a.sink; }
  static __device__ __forceinline__ float head_factor(const Args& a, int t, int h) { return a.gate ? a.gate[(size_t)t * a.Hl + h] : 1.f; }
  static __device__ __forceinline__ bool gated(const Args&) { return false; }
  static __device__ __forceinline__ float value_factor(const Args&, int, int) { return 1.f; }
};

__device__ __forceinline__ void pp_tmem_ld_x32(uint32_t addr, float* r) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
               : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]),
                 "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]),
                 "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31]) : "r"(addr));
}
// both halves rounded as fmaf rounds one value
__device__ __forceinline__ float2 pp_fma2(float2 x, float2 y, float2 z) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\tfma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(z.x), "f"(z.y));
  return d;
}
__device__ __forceinline__ uint32_t pp_desc_mn(uint32_t saddr) { return (uint32_t)pf_desc_mn_sw128(saddr, 16384, 1024); }
// d (+)= a b with a in tensor memory and b MN-major (16 of K: 2,048 bytes), issued as in tc_issue.cuh: keys 0 .. 95 of a tile, or the rest
template <bool MOST>
__device__ __forceinline__ void pp_mma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
#define PP_TS(K_, P_) "add.u32 al, %1, 8 * " #K_ ";\n\tadd.u32 bl, %2, 128 * " #K_ ";\n\tmov.b64 b, {bl, " TI_DESC_HI "};\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], b, %4, " P_ ";\n\t"
  if (MOST)
    asm volatile(TI_BEGIN PP_TS(0, "z") PP_TS(1, "t") PP_TS(2, "t") PP_TS(3, "t") PP_TS(4, "t") PP_TS(5, "t") "}" ::"r"(d), "r"(a), "r"(b_lo), "r"(accumulate), "r"(idesc) : "memory");
  else
    asm volatile(TI_BEGIN PP_TS(6, "t") PP_TS(7, "t") "}" ::"r"(d), "r"(a), "r"(b_lo), "r"(1), "r"(idesc) : "memory");
#undef PP_TS
}

template <class Src, int KC, int VC, int PER_CTA>
__global__ void __launch_bounds__(PP_THREADS, 1) prefill_pair_kernel(const __grid_constant__ typename Src::Args a) {
  using C = PairCfg<KC, VC>;
  pdl_launch(); pdl_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* ring = smem + C::Q_BYTES;
  uint64_t* bars = (uint64_t*)(ring + C::NCH * 16384);
  uint64_t* ch_full = bars; uint64_t* ch_empty = bars + PP_MAX_CHUNKS;
  uint64_t* q_full = bars + 2 * PP_MAX_CHUNKS;      // [2] from here on: one per tile
  uint64_t* s_full = q_full + 2;
  uint64_t* p_most = q_full + 4;                    // keys 0 .. 95 of P written (and O rescaled)
  uint64_t* p_full = q_full + 6;
  uint64_t* o_done = q_full + 8;
  uint32_t& tmem_slot = *(uint32_t*)(q_full + 10);
  int& abort_flag = *(int*)(q_full + 11);
  if (smem_u32(smem) & 1023) { if (threadIdx.x == 0) ca_dev_fail(a.status, CA_DEV_BAD_INDEX, 0xA15); return; }
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, tid = threadIdx.x;

  // the heaviest query tiles (most visible keys) are scheduled first
  const int G = Src::group(a), tok_per_tile = 128 / G;
  const int head = blockIdx.x, units = (a.max_q_tiles + PER_CTA - 1) / PER_CTA;
  const int seq = blockIdx.y / units, unit = units - 1 - blockIdx.y % units;
  const int qlen = a.q_len[seq], kvlen = a.kv_len[seq];
  const int tok0 = unit * PER_CTA * tok_per_tile;
  if (tok0 >= qlen) return;
  const bool bidir = Src::bidir(a);
  // tile x: its tokens, and the key tiles that its rows see (0 where there is no such tile)
  auto tokens_of = [&](int x) { return x >= PER_CTA ? 0 : max(0, min(tok_per_tile, qlen - tok0 - x * tok_per_tile)); };
  auto first_pos_of = [&](int x) { return bidir ? kvlen - 1 : kvlen - qlen + tok0 + x * tok_per_tile; };
  auto tiles_of = [&](int x) {
    const int nt = tokens_of(x);
    return nt == 0 ? 0 : max(0, ((bidir ? kvlen : first_pos_of(x) + nt) + PF_KT - 1) / PF_KT);
  };
  const int n_a = tiles_of(0), n_b = tiles_of(1), n = max(n_a, n_b);

  if (tid == 0) {
    for (int s = 0; s < C::NCH; ++s) { mbar_init(&ch_full[s], 1); mbar_init(&ch_empty[s], 1); }
    for (int x = 0; x < 2; ++x) { mbar_init(&q_full[x], 4); mbar_init(&s_full[x], 1); mbar_init(&p_most[x], 4); mbar_init(&p_full[x], 4); mbar_init(&o_done[x], 1); }
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* abortp = &abort_flag;

  // Registers: 64,512 at launch (384 x 168); 128 x 104 + 256 x 200 = 64,512 of them after the split.
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
    if (warp == 0 && lane == 0) {
      // ---------------------------------------------------------------- K / V producer
      bool ok = true;
      int idx = 0;
      for (int i = 0; ok && i < n; ++i) {
#pragma unroll 1
        for (int c = 0; c < KC + VC; ++c, ++idx) {
          const int s = idx % C::NCH;
          if (!mbar_wait_bounded(&ch_empty[s], ((idx / C::NCH) & 1) ^ 1, abortp)) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_PRODUCER, idx); ok = false; break; }
          mbar_expect_tx(&ch_full[s], 16384);
          Src::template load<KC, VC>(a, head, seq, i, c, ring + s * 16384, &ch_full[s]);
        }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer (products execute in the order of issue)
      // One warp for both tiles: two of them fall into step, both tiles' exponentials at once and then both tiles' products (381 us for the
      // 4096 rows above, 320 with one, both with P in two halves).
      const uint32_t id_s = pf_idesc(PF_KT, 0), id_o = pf_idesc(VC * 64, 1), id_o1 = pf_idesc(64, 1);
      const uint32_t qd = ti_desc(smem_u32(sQ)), kd = ti_desc(smem_u32(ring)), vd = pp_desc_mn(smem_u32(ring));
      bool ok = true;
      auto wait = [&](uint64_t* bar, int ph, int what) {
        if (ok && !mbar_wait_warp(bar, ph & 1, abortp)) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_MMA, what); ok = false; }
        return ok;
      };
      // a place in the ring: slot, and the parity of its round
      struct Place { int s, ph; };
      auto plus = [](Place p, int d) { p.s += d; if (p.s >= C::NCH) { p.s -= C::NCH; p.ph ^= 1; } return p; };
      // S_x = Q_x K(i)^T.  P_x(i - 1) stands in the same columns: its product was issued before, and S_x(i - 1) was read before P was written.
      auto scores = [&](int x, Place k0, bool last_use) {
#pragma unroll
        for (int c = 0; c < KC; ++c) {
          const Place p = plus(k0, c);
          if (!wait(&ch_full[p.s], p.ph, 0x1000 + p.s)) return;
          if (c == 0) tc_fence_after();
          ti_mma4<TI_F16>(tmem + x * 128, qd + (x * KC + c) * 1024, kd + p.s * 1024, id_s, c);
        }
        ti_commit(&s_full[x]);
        if (last_use)
#pragma unroll
          for (int c = 0; c < KC; ++c) ti_commit(&ch_empty[plus(k0, c).s]);
      };
      // O_x += P_x(i) V(i)
      auto values = [&](int x, int i, Place v0, bool last_use, bool last) {
#pragma unroll
        for (int c = 0; c < VC; ++c) { const Place p = plus(v0, c); if (!wait(&ch_full[p.s], p.ph, 0x2000 + i)) return; }
        const uint32_t o = tmem + C::O_COL + x * VC * 64, p = tmem + x * 128, lo = vd + v0.s * 1024;
        const bool whole = VC == 1 || v0.s + VC <= C::NCH;                      // the value chunks lie behind each other
        if (!wait(&p_most[x], i, 0x3000 + i)) return;
        tc_fence_after();
        if (whole) pp_mma_ts<true>(o, p, lo, id_o, i);
        else
#pragma unroll
          for (int c = 0; c < VC; ++c) pp_mma_ts<true>(o + c * 64, p, vd + plus(v0, c).s * 1024, id_o1, i);
        if (!wait(&p_full[x], i, 0x3000 + i)) return;
        tc_fence_after();
        if (whole) pp_mma_ts<false>(o, p, lo, id_o, 1);
        else
#pragma unroll
          for (int c = 0; c < VC; ++c) pp_mma_ts<false>(o + c * 64, p, vd + plus(v0, c).s * 1024, id_o1, 1);
        if (last_use)
#pragma unroll
          for (int c = 0; c < VC; ++c) ti_commit(&ch_empty[plus(v0, c).s]);
        if (last) ti_commit(&o_done[x]);
      };
      Place at = {0, 0};                              // K(i); V(i) lies KC behind
      if (n_a > 0 && wait(&q_full[0], 0, 0x4000)) scores(0, at, n_b == 0);
      if (n_b > 0 && wait(&q_full[1], 0, 0x4001)) scores(1, at, true);
      for (int i = 0; ok && i < n; ++i) {
        const Place v = plus(at, KC), next = plus(v, VC);
        if (i < n_a) {
          values(0, i, v, i >= n_b, i + 1 == n_a);
          if (ok && i + 1 < n_a) scores(0, next, i + 1 >= n_b);
        }
        if (ok && i < n_b) {
          values(1, i, v, true, i + 1 == n_b);
          if (ok && i + 1 < n_b) scores(1, next, true);
        }
        at = next;
      }
    }
    __syncwarp();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    // ------------------------------------------------------------------ softmax + epilogue: a thread per query row
    const int x = (warp >> 2) - 1, q4 = warp & 3, r = q4 * 32 + lane;
    const int ntok = tokens_of(x), nt = x ? n_b : n_a, R = ntok * G;
    const int first_pos = first_pos_of(x), row_base = a.q_start[seq] + tok0 + x * tok_per_tile;
    if (nt > 0) {
      // query rows -> shared memory: eight threads per 128-byte row
      const int w = tid & 127, u = w & 7;
      uint4 v[KC][8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int rr = (w >> 3) + 16 * j;
#pragma unroll
        for (int c = 0; c < KC; ++c) v[c][j] = rr < R ? *(const uint4*)(Src::template q_chunk<KC>(a, head, row_base + rr / G, rr % G, c) + u * 8) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int rr = (w >> 3) + 16 * j;
#pragma unroll
        for (int c = 0; c < KC; ++c) *(uint4*)(sQ + (x * KC + c) * 16384 + rr * 128 + ((u ^ (rr & 7)) << 4)) = v[c][j];
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_full[x]);
    }
    const uint32_t lane_addr = tmem + ((uint32_t)(q4 * 32) << 16);
    const uint32_t s_addr = lane_addr + x * 128, o_addr = lane_addr + C::O_COL + x * VC * 64;
    const bool live = r < R;
    const int qpos = live ? (bidir ? first_pos : first_pos + r / G) : -1;
    const float sc2 = a.scale * 1.4426950408889634f;
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    for (int i = 0; i < nt; ++i) {
      // (the score product is issued behind P V of tile i - 1: that one is done too)
      if (!mbar_wait_warp(&s_full[x], i & 1, abortp)) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_EPILOGUE, i); ok = false; break; }
      tc_fence_after();
      float s[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) pp_tmem_ld_x32(s_addr + c * 32, s + c * 32);
      tc_wait_ld();
      const int key0 = i * PF_KT;
      if (key0 + PF_KT - 1 > first_pos) {            // warp-uniform: some row does not see all keys of the tile
        const int last = qpos - key0;
#pragma unroll
        for (int j = 0; j < 128; ++j) s[j] = j <= last ? s[j] : -INFINITY;
      }
      float m4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) m4[j] = fmaxf(fmaxf(s[j], s[j + 4]), s[j + 8]);
#pragma unroll
      for (int j = 12; j < 124; j += 8)
#pragma unroll
        for (int q = 0; q < 4; ++q) m4[q] = fmaxf(m4[q], fmaxf(s[j + q], s[j + 4 + q]));
#pragma unroll
      for (int q = 0; q < 4; ++q) m4[q] = fmaxf(m4[q], s[124 + q]);
      const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sc2;        // sc2 > 0: scaling commutes with the maximum
      float alpha = 1.f;
      if (mx > m_ref + 8.f) {
        if (m_ref != -INFINITY) alpha = exp2f(m_ref - mx);
        m_ref = mx;
      }
      if (i > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {      // warp-uniform: tcgen05.ld/st are warp collectives
#pragma unroll 1
        for (int c = 0; c < VC * 4; ++c) {
          uint32_t o[16];
          tmem_ld_x16(o_addr + c * 16, o);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          pf_tmem_st_x16(o_addr + c * 16, o);
        }
      }
      const float m_sub = m_ref == -INFINITY ? 0.f : -m_ref;     // a row that has seen no key yet: exponentials of -inf
      const float2 sc = make_float2(sc2, sc2), ms = make_float2(m_sub, m_sub);
      float run = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int k = c * 32 + 2 * j;
          const float2 t = pp_fma2(make_float2(s[k], s[k + 1]), sc, ms);
          const float e0 = pf_exp2(t.x), e1 = pf_exp2(t.y);
          run += e0 + e1;
          bf162 h = __floats2bfloat162_rn(e0, e1);
          pk[j] = *(uint32_t*)&h;
        }
        pf_tmem_st_x16(s_addr + c * 16, pk);
        if (c >= 2) {
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(c == 3 ? &p_full[x] : &p_most[x]);
        }
      }
      l = __fadd_rn(__fmul_rn(l, alpha), run);
    }
    if (ok && nt > 0 && !mbar_wait_warp(&o_done[x], 0, abortp)) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_EPILOGUE, 999); ok = false; }
    tc_fence_after();
    if (__all_sync(0xffffffffu, ok) && R > 0) {
      const int rr = live ? r : 0;
      const int t = row_base + rr / G, h = head * G + rr % G;
      float scale_o = 1.f, lt = l;
      if (Src::sink(a)) {                               // learned sink logit: one more softmax term with a zero value
        const float m_nat = (m_ref == -INFINITY) ? -INFINITY : m_ref * 0.6931471805599453f;
        const float sk = Src::sink(a)[h], m2 = fmaxf(m_nat, sk);
        const float e1 = (m_nat == -INFINITY) ? 0.f : __expf(m_nat - m2);
        lt = l * e1 + __expf(sk - m2); scale_o = e1;
      }
      float inv = (lt > 0.f ? scale_o / lt : 0.f) * (live ? Src::head_factor(a, t, h) : 1.f);
      if (l == 0.f && qpos >= 0 && !Src::sink(a)) inv = NAN;          // keys seen, and all of them scored -inf: no weights (a row without keys is 0)
      const bool gated = Src::gated(a);
      bf16* dst = a.out + (size_t)t * a.ldo + (size_t)h * a.dv;
      const bool vec = ((a.dv | a.ldo) & 7) == 0;
#pragma unroll 1
      for (int c = 0; c < VC * 2; ++c) {
        float o[32];
        if (nt > 0) { pp_tmem_ld_x32(o_addr + c * 32, o); tc_wait_ld(); }
        else {
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = 0.f;
        }
        if (!live) continue;
        if (gated) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c * 32 + j < a.dv) o[j] *= Src::value_factor(a, t, h * a.dv + c * 32 + j);
        }
        uint32_t w[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) { bf162 hh = __floats2bfloat162_rn(o[2 * j] * inv, o[2 * j + 1] * inv); w[j] = *(uint32_t*)&hh; }
        if (vec) {                            // value widths that do not fill their last 64-wide chunk stop at column dv
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (c * 32 + j * 8 < a.dv) *(uint4*)(dst + c * 32 + j * 8) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c * 32 + j < a.dv) dst[c * 32 + j] = ((const bf16*)w)[j];
        }
      }
    }
  }
  if (*abortp && warp == 0) { const uint64_t t0 = globaltimer_ns(); while (globaltimer_ns() - t0 < 200000) __nanosleep(1000); }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

template <class Src, int KC, int VC, int PER_CTA>
static int launch_prefill_tiles(const typename Src::Args& a, int heads, int n_seq, cudaStream_t s) {
  auto kern = prefill_pair_kernel<Src, KC, VC, PER_CTA>;
  constexpr int SMEM = PairCfg<KC, VC>::SMEM;
  static bool attr_set[64] = {false};
  int dev = 0; cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return ca_cuda(e, "cudaFuncSetAttribute(prefill_pair)");
    attr_set[dev & 63] = true;
  }
  CA_LAUNCH_PDL(kern, dim3(heads, n_seq * ((a.max_q_tiles + PER_CTA - 1) / PER_CTA)), PP_THREADS, SMEM, s, a);
  return CA_OK;
}
// Hidden scores are -inf here before they are scaled, which hides them only if the scale is positive (0 x -inf is NaN): any other takes the one-tile kernels,
// which clear the probabilities.
static bool pf_pair_takes(float scale) { return scale > 0.f; }
// Query tiles per CTA here, or 0: the one-tile kernels.
//
// A pair takes 1.3 to 1.6 of a tile's time, so pairs have to save whole waves; less than a wave of them pays only with few tiles, which see about as many keys each
// (2,048 rows of 16 latent heads, 1 to 16 key tiles, one-tile kernel / pairs: 59 / 70 us).
static bool pf_pairs_save_waves(long long tiles, long long pairs, int max_q_tiles) {
  const long long sms = ca_sm_count();
  return (pairs >= sms || max_q_tiles <= 4) && 4 * ((pairs + sms - 1) / sms) < 3 * ((tiles + sms - 1) / sms);
}
// Paged: with keys of up to 128 columns one tile per CTA while that is one wave, else pairs.  us, one-tile kernel / one tile per CTA here / pairs, 64 heads over 4:
// 296 rows (148 tiles) 24.6 / 16.4 / 20.5; 300 behind 6,000 227 / 178 / 115; 512 40 / 27 / 24; 17 behind 4,000 84 / 66 / 76.
// In 400 random steps (1 to 49 sequences, 1 to 32 key heads, keys of 64 to 192 and values of 64 and 128 columns) no choice of this rule is slower than the one-tile kernel.
static int pf_tiles_paged(int kc, int heads, int n_seq, int max_q_tiles) {
  const long long tiles = (long long)heads * n_seq * max_q_tiles, pairs = (long long)heads * n_seq * ((max_q_tiles + 1) / 2);
  if (kc <= 2) return tiles <= ca_sm_count() ? 1 : 2;
  return pf_pairs_save_waves(tiles, pairs, max_q_tiles) ? 2 : 0;
}
// Latent: the one-tile kernel takes less per tile than the paged one, so a lone tile here gains little or loses.  One-tile kernel / one tile per CTA here / pairs, us
// (columns of keys, rotated ones behind the +, and of values; rows, behind as many): 64 and 64, 2,048 rows of 12 heads 36 / 34 / 40; 128 and 128, 64 behind 4,000 of 48 heads
// 58 / 67 / 65; 64 + 64 and 128, 2,048 of 12 heads 38 / 44 / 50; 128 + 64 and 128, 128 heads, 200 behind 4,000 125 / - / 101, 257 behind 4,000 183 / - / 177, 2,048 behind
// 6,144 1473 / - / 1178.  On average over random steps of lone tiles, one tile per CTA here takes 0.88 to 1.02 of the one-tile kernel's time with up to 192 columns of keys and
// values and no rotated ones, 0.95 to 1.09 with 128 and 128, 1.08 to 1.18 with 64 + 64, and pairs' lone tiles 0.9 to 1.2 with 192.
// Of sequences of different lengths the grid's rectangle says little; `T` bounds how many tiles and pairs there are.  What pairs win is won by second tiles, what they
// lose is lost by lone ones: 128 + 64 and 128, 16 heads, 1,024 rows beside 15 of one behind 4,000 142 / - / 155; 64 heads, 2,048 behind 4,000 beside 20 of one behind 500
// 824 / - / 647.  Contexts are on the device, so lone tiles that read far more keys than the prompts do lose all the same (128 heads, the first of these: 890 / - / 1011).
// Where the lines lie: of 5,000 random steps (1 to 49 sequences, 2 to 128 heads, all widths) 2.4 % are over 4 % slower than in the one-tile kernel, with the rule of the paged form 19 %.
static int pf_tiles_latent(int kn, int kr, int vc, int heads, int n_seq, int T, int max_q_len) {
  const long long max_q_tiles = (max_q_len + 127) / 128;
  long long tiles = n_seq * max_q_tiles, pairs = n_seq * ((max_q_tiles + 1) / 2);
  bool two;
  if (T >= (long long)n_seq * max_q_len) two = pf_pairs_save_waves(heads * tiles, heads * pairs, (int)max_q_tiles);
  else {
    tiles = heads * min(tiles, (T + n_seq * 127LL) / 128); pairs = heads * min(pairs, (T + n_seq * 255LL) / 256);
    const long long second = tiles - pairs, lone = pairs - second;
    two = 20 * second > 15 * ca_sm_count() + lone;
  }
  return two ? 2 : kr == 0 && kn + vc <= 3 ? 1 : 0;
}
template <class Src, int KC, int VC>
static int launch_prefill_pair(const typename Src::Args& a, int heads, int n_seq, int per_cta, cudaStream_t s) {
  if constexpr (Src::template alone<KC, VC>())
    if (per_cta == 1) return launch_prefill_tiles<Src, KC, VC, 1>(a, heads, n_seq, s);
  return launch_prefill_tiles<Src, KC, VC, 2>(a, heads, n_seq, s);
}
// The latent rule's answer, for tests; widths in chunks of 64 columns.
extern "C" int cuteafd_latent_prefill_tiles(int key_chunks, int rotated_chunks, int value_chunks, int heads, int n_seq, int T, int max_q_len) {
  return pf_tiles_latent(key_chunks, rotated_chunks, value_chunks, heads, n_seq, T, max_q_len);
}
