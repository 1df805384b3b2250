// Gated delta-rule linear attention (the recurrent layers of the GDN / KDA hybrid families): decode, verify and prompt runs.
//
// Per (sequence, head) a state S [dk x dv] in fp32 is carried from token to token:
//     S   <- diag(g_t) S                       g_t: decay, one scalar per head (GDN) or one value per key channel (KDA), in (0, 1]
//     u   =  S^T k_t                           what the state currently returns for this key          [dv]
//     S   <- S + k_t (beta_t (v_t - u))^T      delta rule: move the stored value towards v_t
//     o_t =  S^T q_t                                                                                   [dv]
// q and k arrive L2-normalised (q also scaled by dk^-1/2) from the projection side.  The state crosses HBM once in and once out per call, and
// columns of S (value channels) do not meet.  Two forms:
//   short runs of many sequences (decoding, verifying): one block per (sequence, head), a thread per column with all 128 rows in registers; all
//     blocks run at once and the time is that of the states' bytes and a few tokens' latencies.
//   everything else: a (sequence, head) is spread over four blocks of 32 columns, and a pair of columns over eight lanes with 16 rows each (two
//     fp32 values per FMA).  Keys and queries come from shared memory, 128 bytes per lane and token whatever the layout: with one column per lane
//     these reads alone took 256 cycles a token (1,330 us for the run below), so a lane has two.  What then bounds a run is the chain from token to
//     token, a dot product and its reduction over lanes.  It is taken off the path of every second token: with P_t the decayed state before token t's update,
//         P_t = g_t P_(t-1) + g_t k_(t-1) d_(t-1),     u_t = k_t . (g_t P_(t-1)) + (k_t . g_t k_(t-1)) d_(t-1),     o_t = q_t . P_t + (q_t . k_t) d_t
//     so the reduction of k_t . (g_t P_(t-1)) does not wait for d_(t-1), and the products of keys and queries among themselves belong to no
//     column and are computed once per block.  Operands of eight tokens at a time go through shared memory as fp32, the next eight on
//     their way meanwhile; the eight outputs are reduced together.  4,096 tokens of 32 heads: 735 us (the short form: 6,680 us).
//
// Reference: the `gdn*` / `kda*` programs of the Qwen 3.8 and GLM 5.3 Flash families (AOT-exported, sources absent:
// python/tools/aot/) and their per-slot recurrent state, rust/crates/cuteafd-daemon/src/families/qwen4/ (state slots per
// sequence, draft rows rolled back by restoring the state snapshot).
#include "common.cuh"

#define LA_DK 128
#define LA_DV 128

struct LinAttnArgs {
  const bf16* q; const bf16* k; const bf16* v;   // [T, H, 128]
  const float* g;                                 // [T, H] (per_channel = 0) or [T, H, 128]
  const float* beta;                              // [T, H]
  float* state;                                   // [slots, H, dk, dv]
  const int* slot_of_seq; const int* q_start; const int* q_len;
  bf16* out;                                      // [T, H, 128]
  float* snapshots;                               // optional [T, H, dk, dv]: the state AFTER each token (verify rollback), or null
  int H, per_channel, n_slots;             // per_channel: bit 0 = one decay per key channel, bit 1 = do not write the state back
  int* status;
};

// two fp32 values per register pair
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float sum2(f32x2 v) { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return a + b; }
__device__ __forceinline__ float2 unpack2(f32x2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

#define LA_COLS 32          // value channels of a block
#define LA_THREADS 128      // two columns x 16 rows each
#define LA_TOK 8            // tokens staged at a time

__device__ __forceinline__ float4 floats4(uint2 r) {
  const bf16* e = (const bf16*)&r;
  return make_float4(__bfloat162float(e[0]), __bfloat162float(e[1]), __bfloat162float(e[2]), __bfloat162float(e[3]));
}

template <bool PER_CHANNEL, bool SNAPSHOTS>
__global__ void __launch_bounds__(LA_THREADS) gated_delta_kernel(const LinAttnArgs a) {
  pdl_launch(); pdl_wait();
  __shared__ __align__(16) float sq[2][LA_TOK][LA_DK], sk[2][LA_TOK][LA_DK], sg[2][PER_CHANNEL ? LA_TOK : 1][LA_DK], sv[2][LA_TOK][LA_COLS];
  __shared__ float4 ss[2][LA_TOK];                                             // beta; decay (one per head); k_t . g_t k_(t-1); q_t . k_t
  const int seq = blockIdx.y, h = blockIdx.x >> 2, col0 = (blockIdx.x & 3) * LA_COLS, tid = threadIdx.x;
  const int slot = a.slot_of_seq[seq];
  if (slot < 0 || slot >= a.n_slots) { if (tid == 0) ca_dev_fail(a.status, CA_DEV_BAD_INDEX, 0x6D1); return; }
  const int t0 = a.q_start[seq], n = a.q_len[seq];
  if (n <= 0) return;
  const int r = tid & 7, col = (tid >> 3) * 2;                                 // this lane's rows: 32 i + 4 r + {0..3}; its two columns of the block
  float* S = a.state + ((size_t)slot * a.H + h) * LA_DK * LA_DV + col0 + col;
  f32x2 st[2][8];                                                              // [column][pair of rows]
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float* p = S + (size_t)((i >> 1) * 32 + r * 4 + (i & 1) * 2) * LA_DV;
    const float x0 = p[0], x1 = p[1], y0 = p[LA_DV], y1 = p[LA_DV + 1];
    st[0][i] = pack2(x0, y0); st[1][i] = pack2(x1, y1);
  }
  // Staging: a warp takes tokens w and w + 4, four channels per lane; the values by the first two warps.  The loads are unconditional (tokens past
  // the run's end repeat its last one, and are not used) and stay unconverted until they are staged: a branch or a conversion behind them
  // would wait for them, 320 of 790 cycles per token.
  const int wtok = tid >> 5, lch = (tid & 31) * 4, vtok = (tid >> 3) & (LA_TOK - 1), vch = (tid & 7) * 4;
  uint2 fq[2], fk[2], fp[2], fv;
  float4 fg[2];
  float fb[2];
  auto fetch = [&](int at) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int tok = min(at + wtok + 4 * e, n - 1);
      const size_t th = (size_t)(t0 + tok) * a.H + h, o = th * LA_DK + lch, before = ((size_t)(t0 + max(tok - 1, 0)) * a.H + h) * LA_DK + lch;
      fq[e] = __ldg((const uint2*)(a.q + o)); fk[e] = __ldg((const uint2*)(a.k + o)); fp[e] = __ldg((const uint2*)(a.k + before));
      if (PER_CHANNEL) fg[e] = __ldg((const float4*)(a.g + o));
      else fg[e].x = __ldg(a.g + th);
      fb[e] = __ldg(a.beta + th);
    }
    fv = __ldg((const uint2*)(a.v + ((size_t)(t0 + min(at + vtok, n - 1)) * a.H + h) * LA_DV + col0 + vch));
  };
  auto stage = [&](int b) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int tok = wtok + 4 * e;
      const float4 q = floats4(fq[e]), k = floats4(fk[e]), kb = floats4(fp[e]), g = PER_CHANNEL ? fg[e] : make_float4(fg[e].x, fg[e].x, fg[e].x, fg[e].x);
      *(float4*)&sq[b][tok][lch] = q; *(float4*)&sk[b][tok][lch] = k;
      if (PER_CHANNEL) *(float4*)&sg[b][PER_CHANNEL ? tok : 0][lch] = g;
      float qk = q.x * k.x + q.y * k.y + q.z * k.z + q.w * k.w, kk = k.x * (g.x * kb.x) + k.y * (g.y * kb.y) + k.z * (g.z * kb.z) + k.w * (g.w * kb.w);
#pragma unroll
      for (int w = 16; w; w >>= 1) { qk += __shfl_xor_sync(0xffffffffu, qk, w); kk += __shfl_xor_sync(0xffffffffu, kk, w); }
      if ((tid & 31) == 0) ss[b][tok] = make_float4(fb[e], g.x, kk, qk);
    }
    if (tid < LA_TOK * 8) *(float4*)&sv[b][vtok][vch] = floats4(fv);
  };
  fetch(0);
  stage(0);
  __syncthreads();
  // `cnt` tokens of buffer b (all eight: a constant, so that the loop is straight-line code)
  auto block = [&](int b, int at, int cnt) {
    float op[2][LA_TOK], mine[2] = {}, dp[2] = {};
    ulonglong2 kp[4] = {}, kn[4], qn[4], gn[4];                                // keys of the token before; the next token's operands
    float4 sn; float2 vn;
    auto read = [&](int t) {
      sn = ss[b][t]; vn = *(const float2*)&sv[b][t][col];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        kn[i] = *(const ulonglong2*)&sk[b][t][i * 32 + r * 4]; qn[i] = *(const ulonglong2*)&sq[b][t][i * 32 + r * 4];
        if (PER_CHANNEL) gn[i] = *(const ulonglong2*)&sg[b][PER_CHANNEL ? t : 0][i * 32 + r * 4];
      }
    };
    read(0);
#pragma unroll
    for (int t = 0; t < LA_TOK; ++t) {
      op[0][t] = op[1][t] = 0.f;
      if (t >= cnt) continue;
      const float4 sc = sn;
      const float2 v2 = vn;
      const f32x2 g1 = pack2(sc.y, sc.y);
      ulonglong2 k4[4], g4[4], q4[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { k4[i] = kn[i]; q4[i] = qn[i]; g4[i] = PER_CHANNEL ? gn[i] : make_ulonglong2(g1, g1); }
      if (t + 1 < LA_TOK) read(t + 1);
      // st: P_(t-1) (in front of a block's first token: the whole state) -> g_t P_(t-1), and its product with k_t
      f32x2 u2[2][2] = {};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          st[c][2 * i] = mul2(st[c][2 * i], g4[i].x); st[c][2 * i + 1] = mul2(st[c][2 * i + 1], g4[i].y);
          u2[c][0] = fma2(st[c][2 * i], k4[i].x, u2[c][0]); u2[c][1] = fma2(st[c][2 * i + 1], k4[i].y, u2[c][1]);
        }
      }
      float u[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) u[c] = sum2(u2[c][0]) + sum2(u2[c][1]);
#pragma unroll
      for (int w = 1; w < 8; w <<= 1) {
        const float x = __shfl_xor_sync(0xffffffffu, u[0], w), y = __shfl_xor_sync(0xffffffffu, u[1], w);
        u[0] += x; u[1] += y;
      }
      // P_t, once d_(t-1) is known, and what the output takes from it
      f32x2 o2[2][2] = {};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const f32x2 x = PER_CHANNEL ? mul2(kp[i].x, g4[i].x) : kp[i].x, y = PER_CHANNEL ? mul2(kp[i].y, g4[i].y) : kp[i].y;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (t > 0) {
            const float e = PER_CHANNEL ? dp[c] : sc.y * dp[c];
            st[c][2 * i] = fma2(x, pack2(e, e), st[c][2 * i]); st[c][2 * i + 1] = fma2(y, pack2(e, e), st[c][2 * i + 1]);
          }
          o2[c][0] = fma2(st[c][2 * i], q4[i].x, o2[c][0]); o2[c][1] = fma2(st[c][2 * i + 1], q4[i].y, o2[c][1]);
        }
        kp[i] = k4[i];
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        op[c][t] = sum2(o2[c][0]) + sum2(o2[c][1]);
        const float d = sc.x * ((c ? v2.y : v2.x) - (t > 0 ? fmaf(sc.z, dp[c], u[c]) : u[c]));
        if (r == t) mine[c] = sc.w * d;
        dp[c] = d;
      }
      if (SNAPSHOTS) {
        float* snap = a.snapshots + ((size_t)(t0 + at + t) * a.H + h) * LA_DK * LA_DV + col0 + col;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float* p = snap + (size_t)((i >> 1) * 32 + r * 4 + (i & 1) * 2) * LA_DV;
          const f32x2 kk = i & 1 ? k4[i >> 1].y : k4[i >> 1].x;
#pragma unroll
          for (int c = 0; c < 2; ++c) { const float2 v = unpack2(fma2(kk, pack2(dp[c], dp[c]), st[c][i])); p[c] = v.x; p[LA_DV + c] = v.y; }
        }
      }
    }
    // the state behind the block's last token
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        st[c][2 * i] = fma2(kp[i].x, pack2(dp[c], dp[c]), st[c][2 * i]); st[c][2 * i + 1] = fma2(kp[i].y, pack2(dp[c], dp[c]), st[c][2 * i + 1]);
      }
    // eight outputs over eight lanes: lane r is left with token r's
#pragma unroll
    for (int w = 4; w; w >>= 1)
#pragma unroll
      for (int j = 0; j < w; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float keep = (r & w) ? op[c][j + w] : op[c][j], send = (r & w) ? op[c][j] : op[c][j + w];
          op[c][j] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
    if (r < cnt) {
      bf16* o = a.out + ((size_t)(t0 + at + r) * a.H + h) * LA_DV + col0 + col;
      o[0] = __float2bfloat16(op[0][0] + mine[0]); o[1] = __float2bfloat16(op[1][0] + mine[1]);
    }
  };
  for (int at = 0, b = 0; at < n; at += LA_TOK, b ^= 1) {
    fetch(at + LA_TOK);
    if (at + LA_TOK <= n) block(b, at, LA_TOK);
    else block(b, at, n - at);
    stage(b ^ 1);
    __syncthreads();
  }
  if (a.per_channel & 2) return;          // verify rows of a speculative step: outputs only, the state is committed later by a replay
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float* p = S + (size_t)((i >> 1) * 32 + r * 4 + (i & 1) * 2) * LA_DV;
#pragma unroll
    for (int c = 0; c < 2; ++c) { const float2 v = unpack2(st[c][i]); p[c] = v.x; p[LA_DV + c] = v.y; }
  }
}

__global__ void __launch_bounds__(LA_DV) gated_delta_short_kernel(const LinAttnArgs a) {
  pdl_launch(); pdl_wait();
  __shared__ float sq[LA_DK], sk[LA_DK], sg[LA_DK];
  const int seq = blockIdx.y, h = blockIdx.x, j = threadIdx.x;
  const int slot = a.slot_of_seq[seq];
  if (slot < 0 || slot >= a.n_slots) { if (j == 0) ca_dev_fail(a.status, CA_DEV_BAD_INDEX, 0x6D1); return; }
  float* S = a.state + ((size_t)slot * a.H + h) * LA_DK * LA_DV;
  float col[LA_DK];
#pragma unroll
  for (int i = 0; i < LA_DK; ++i) col[i] = S[(size_t)i * LA_DV + j];
  const int t0 = a.q_start[seq], n = a.q_len[seq];
  for (int t = t0; t < t0 + n; ++t) {
    const size_t th = (size_t)t * a.H + h;
    __syncthreads();                                   // the previous token's readers are done with sq / sk / sg
    sq[j] = __bfloat162float(a.q[th * LA_DK + j]);
    sk[j] = __bfloat162float(a.k[th * LA_DK + j]);
    sg[j] = (a.per_channel & 1) ? a.g[th * LA_DK + j] : a.g[th];
    __syncthreads();
    const float vj = __bfloat162float(a.v[th * LA_DV + j]), bt = a.beta[th];
    float u = 0.f;
#pragma unroll
    for (int i = 0; i < LA_DK; ++i) { col[i] *= sg[i]; u = fmaf(col[i], sk[i], u); }
    const float d = bt * (vj - u);
    float o = 0.f;
#pragma unroll
    for (int i = 0; i < LA_DK; ++i) { col[i] = fmaf(sk[i], d, col[i]); o = fmaf(col[i], sq[i], o); }
    a.out[th * LA_DV + j] = __float2bfloat16(o);
    if (a.snapshots) {
      float* snap = a.snapshots + th * LA_DK * LA_DV;
#pragma unroll
      for (int i = 0; i < LA_DK; ++i) snap[(size_t)i * LA_DV + j] = col[i];
    }
  }
  if (a.per_channel & 2) return;          // verify rows of a speculative step: outputs only, the state is committed later by a replay
#pragma unroll
  for (int i = 0; i < LA_DK; ++i) S[(size_t)i * LA_DV + j] = col[i];
}

// `max_len`: the longest run (0: not known).  Short runs take the short form when the four-block form would need more than one wave, and the longer
// the more waves it needs: it has four times the blocks, and a shorter chain per token.  Measured, short / four-block form in us, 32 heads:
//     sequences     2 tokens       3            4            5            6            7            8
//       3          12.4 / 14.3  14.5 / 14.5  16.4 / 14.5  18.4 / 16.3  19.5 / 16.4  20.5 / 16.5  22.6 / 14.4        (1.3 waves)
//       5          14.3 / 16.4  16.4 / 18.3  18.4 / 18.5  18.5 / 18.5  20.7 / 18.8  22.6 / 20.4                     (2.2)
//       8          14.4 / 20.6  16.4 / 22.5  18.5 / 22.6  20.5 / 24.6  22.6 / 24.6  24.6 / 26.6  26.7 / 24.6        (3.5)
//      48          51.3 / 79.9  63.5 / 84.0  73.7 / 90.1  84.0 / 94.1  96.3 / 98.3   107 / 103    119 / 94          (21)
// Not told apart: where the short form itself is just over a wave (5 sequences of 64 heads) its line is at 4 tokens (6 tokens: 34.8 / 28.8).
extern "C" int cuteafd_gated_delta_run(const void* q, const void* k, const void* v, const float* g, const float* beta, float* state,
                                       const int* slot_of_seq, const int* q_start, const int* q_len, void* out, float* snapshots, int n_seq,
                                       int H, int per_channel, int n_slots, int max_len, int* status, cudaStream_t s) {
  CA_REQUIRE(q && k && v && g && beta && state && slot_of_seq && q_start && q_len && out, "gated_delta_step: null argument");
  CA_REQUIRE(H >= 1 && n_slots >= 1, "gated_delta_step: bad geometry");
  if (n_seq <= 0) return CA_OK;
  LinAttnArgs a;
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.g = g; a.beta = beta; a.state = state; a.slot_of_seq = slot_of_seq;
  a.q_start = q_start; a.q_len = q_len; a.out = (bf16*)out; a.snapshots = snapshots; a.H = H; a.per_channel = per_channel; a.n_slots = n_slots;
  a.status = status;
  const dim3 grid(H * (LA_DV / LA_COLS), n_seq);
  // the four-block form loads four channels at a time, and every block all of a head's q and k: no output may take their place
  const bool in_place = out == q || out == k;
  const float waves = (float)((long long)H * n_seq * (LA_DV / LA_COLS)) / (float)(2 * ca_sm_count());
  const bool aligned = (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 7) == 0 && (!(per_channel & 1) || ((uintptr_t)g & 15) == 0);
  if (!aligned || in_place || (max_len > 0 && waves > 1.f && max_len <= (waves < 3.f ? 2 + (int)waves : 6))) CA_LAUNCH_PDL(gated_delta_short_kernel, dim3(H, n_seq), LA_DV, 0, s, a);
  else if (per_channel & 1) { if (snapshots) CA_LAUNCH_PDL((gated_delta_kernel<true, true>), grid, LA_THREADS, 0, s, a); else CA_LAUNCH_PDL((gated_delta_kernel<true, false>), grid, LA_THREADS, 0, s, a); }
  else { if (snapshots) CA_LAUNCH_PDL((gated_delta_kernel<false, true>), grid, LA_THREADS, 0, s, a); else CA_LAUNCH_PDL((gated_delta_kernel<false, false>), grid, LA_THREADS, 0, s, a); }
  CA_CHECK_LAUNCH("gated_delta_step");
  return CA_OK;
}

extern "C" int cuteafd_gated_delta_step(const void* q, const void* k, const void* v, const float* g, const float* beta, float* state,
                                        const int* slot_of_seq, const int* q_start, const int* q_len, void* out, float* snapshots, int n_seq,
                                        int H, int per_channel, int n_slots, int* status, cudaStream_t s) {
  return cuteafd_gated_delta_run(q, k, v, g, beta, state, slot_of_seq, q_start, q_len, out, snapshots, n_seq, H, per_channel, n_slots, 0, status, s);
}

// Causal depthwise convolution of width 4 over the token axis with a per-sequence carry of the last three inputs (the short
// convolution in front of q / k / v in these layers), SiLU on the output.  x: [T, C] bf16 with row pitch ldx, y: [T, C]; w: [C, 4] fp32; carry: [slots, 3, C]
// bf16, updated in place to the last three inputs of each sequence.
// A thread takes V neighbouring channels of CONV_TOK tokens and re-reads the three inputs in front of them; blocks beyond the first of a sequence
// never look at the carry, and the first one replaces it after reading it, so no block reads what another writes.  Bound by its bytes:
// 4,096 tokens x 8,192 channels take 57 us (one thread per channel walking the whole sequence: 2,040 us, a chain of dependent loads on 32 SMs).
#define CONV_TOK 16
template <bool UPDATE, int V>
__global__ void __launch_bounds__(128) short_conv4_kernel(const bf16* __restrict__ x, const float* __restrict__ w, bf16* __restrict__ carry, const int* __restrict__ slot_of_seq,
                                   const int* __restrict__ q_start, const int* __restrict__ q_len, bf16* __restrict__ y, int C, int ldx, int n_slots, int* status) {
  pdl_launch(); pdl_wait();
  struct __align__(2 * V) Vec { bf16 e[V]; };
  const int seq = blockIdx.y, c = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (c >= C) return;
  const int slot = slot_of_seq[seq];
  if (slot < 0 || slot >= n_slots) { if (c == 0 && blockIdx.z == 0) ca_dev_fail(status, CA_DEV_BAD_INDEX, 0x6D2); return; }
  const int t0 = q_start[seq], n = q_len[seq];
  bf16* cr = carry + (size_t)slot * 3 * C + c;
  const bf16* xs = x + (size_t)t0 * ldx + c;
  bf16* ys = y + (size_t)t0 * C + c;
  float wt[V][4];
  const bool wvec = ((uintptr_t)w & 15) == 0;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (wvec) { const float4 f = *(const float4*)(w + (size_t)(c + v) * 4); wt[v][0] = f.x; wt[v][1] = f.y; wt[v][2] = f.z; wt[v][3] = f.w; }
    else {
#pragma unroll
      for (int i = 0; i < 4; ++i) wt[v][i] = w[(c + v) * 4 + i];
    }
  }
  auto input = [&](int t) { return t >= 0 ? *(const Vec*)(xs + (size_t)t * ldx) : *(const Vec*)(cr + (size_t)(3 + t) * C); };
  // the launch may have fewer token blocks than the longest sequence needs: each takes every gridDim.z-th chunk
  Vec h0, h1, h2;
  for (int c0 = blockIdx.z * CONV_TOK; c0 < n; c0 += gridDim.z * CONV_TOK) {
    // (a block that walks the whole sequence has the three inputs in front already, and does not look at rows that it may have written: x == y)
    if (c0 == 0 || gridDim.z > 1) { h0 = input(c0 - 3); h1 = input(c0 - 2); h2 = input(c0 - 1); }
    Vec in[CONV_TOK];
    const int m = min(CONV_TOK, n - c0);
#pragma unroll
    for (int i = 0; i < CONV_TOK; ++i) if (i < m) in[i] = *(const Vec*)(xs + (size_t)(c0 + i) * ldx);
    if (UPDATE && c0 == 0) {
      const Vec l0 = input(n - 3), l1 = input(n - 2), l2 = input(n - 1);
      *(Vec*)cr = l0; *(Vec*)(cr + C) = l1; *(Vec*)(cr + 2 * (size_t)C) = l2;
    }
#pragma unroll
    for (int i = 0; i < CONV_TOK; ++i) {
      if (i >= m) break;
      Vec out;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const float acc = wt[v][0] * __bfloat162float(h0.e[v]) + wt[v][1] * __bfloat162float(h1.e[v]) + wt[v][2] * __bfloat162float(h2.e[v]) + wt[v][3] * __bfloat162float(in[i].e[v]);
        out.e[v] = __float2bfloat16(acc / (1.f + __expf(-acc)));
      }
      *(Vec*)(ys + (size_t)(c0 + i) * C) = out;
      h0 = h1; h1 = h2; h2 = in[i];
    }
  }
}

template <bool UPDATE>
static int short_conv4(const void* x, const float* w, void* carry, const int* slot_of_seq, const int* q_start, const int* q_len, void* y, int n_seq, int C, int ldx, int n_slots,
                       int max_len, int* status, cudaStream_t s) {
  CA_REQUIRE(x && w && carry && slot_of_seq && q_start && q_len && y && C >= 1 && ldx >= C, "short_conv4: bad arguments");
  if (n_seq <= 0) return CA_OK;
  // a step of few tokens is a chain of latencies: more threads with one channel each
  const bool vec = (max_len <= 0 || max_len > 8) && C % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)y | (uintptr_t)carry) & 7) == 0;
  const int V = vec ? 4 : 1, chunks = max_len > 0 && x != y ? (max_len + CONV_TOK - 1) / CONV_TOK : 1;      // in place: no block reads what another writes
  const dim3 grid((C + 128 * V - 1) / (128 * V), n_seq, chunks < 1024 ? chunks : 1024);
  if (vec) CA_LAUNCH_PDL((short_conv4_kernel<UPDATE, 4>), grid, 128, 0, s, (const bf16*)x, w, (bf16*)carry, slot_of_seq, q_start, q_len, (bf16*)y, C, ldx, n_slots, status);
  else CA_LAUNCH_PDL((short_conv4_kernel<UPDATE, 1>), grid, 128, 0, s, (const bf16*)x, w, (bf16*)carry, slot_of_seq, q_start, q_len, (bf16*)y, C, ldx, n_slots, status);
  CA_CHECK_LAUNCH("short_conv4");
  return CA_OK;
}

// `max_len`: the longest run of the step, which sizes the launch (0: not known, one block walks each sequence).  `update` 0: the carry stays as it is
// (the verify rows of a speculative step; the accepted ones are replayed with `update` 1, which then moves it).
extern "C" int cuteafd_short_conv4_run(const void* x, const float* w, void* carry, const int* slot_of_seq, const int* q_start, const int* q_len, void* y, int n_seq, int C, int ldx,
                                       int n_slots, int max_len, int update, int* status, cudaStream_t s) {
  return update ? short_conv4<true>(x, w, carry, slot_of_seq, q_start, q_len, y, n_seq, C, ldx, n_slots, max_len, status, s)
                : short_conv4<false>(x, w, carry, slot_of_seq, q_start, q_len, y, n_seq, C, ldx, n_slots, max_len, status, s);
}

extern "C" int cuteafd_short_conv4(const void* x, const float* w, void* carry, const int* slot_of_seq, const int* q_start, const int* q_len, void* y,
                                   int n_seq, int C, int ldx, int n_slots, int* status, cudaStream_t s) {
  return short_conv4<true>(x, w, carry, slot_of_seq, q_start, q_len, y, n_seq, C, ldx, n_slots, 0, status, s);
}

// ---------------------------------------------------------------- glue of a gated delta-rule layer
// After the convolution: conv [T, (2 Hk + Hv) * 128] bf16 holds q (Hk heads), k (Hk heads), v (Hv heads); ba [T, ldb] fp32 holds
// b [Hv] then a [Hv] (or a per key channel [Hv * 128]).  One warp per (token, value head) writes what the recurrence consumes:
// q_e / k_e [T, Hv, 128] = the L2-normalised q (scaled by 128^-1/2) and k of key head hv / (Hv / Hk), v_e [T, Hv, 128] (contiguous
// copy), beta = sigmoid(b), g = exp(-exp(a_log[hv]) * softplus(a + dt_bias)) per head or per channel.
__global__ void linear_prepare_kernel(const bf16* __restrict__ conv, const float* __restrict__ ba, const float* __restrict__ a_log,
                                      const float* __restrict__ dt_bias, bf16* __restrict__ q_e, bf16* __restrict__ k_e, bf16* __restrict__ v_e,
                                      float* __restrict__ g, float* __restrict__ beta, int T, int Hk, int Hv, int ldb, int per_channel) {
  pdl_launch(); pdl_wait();
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= T * Hv) return;
  const int t = w / Hv, hv = w % Hv, hk = hv / (Hv / Hk);
  const int C = (2 * Hk + Hv) * 128;
  const bf16* row = conv + (size_t)t * C;
  const uint2 qr = *(const uint2*)(row + hk * 128 + lane * 4), kr = *(const uint2*)(row + (Hk + hk) * 128 + lane * 4);
  const uint2 vr = *(const uint2*)(row + (2 * Hk + hv) * 128 + lane * 4);
  const bf16* qe = (const bf16*)&qr; const bf16* ke = (const bf16*)&kr;
  float q[4], k[4], sq = 0.f, sk = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) { q[j] = __bfloat162float(qe[j]); k[j] = __bfloat162float(ke[j]); sq += q[j] * q[j]; sk += k[j] * k[j]; }
  sq = warp_sum(sq); sk = warp_sum(sk);
  const float iq = 0.08838834764831845f / fmaxf(sqrtf(sq), 1e-6f), ik = 1.f / fmaxf(sqrtf(sk), 1e-6f);     // 128^-1/2 folded into q
  bf16 qo[4], ko[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) { qo[j] = __float2bfloat16(q[j] * iq); ko[j] = __float2bfloat16(k[j] * ik); }
  const size_t o = ((size_t)t * Hv + hv) * 128 + lane * 4;
  *(uint2*)(q_e + o) = *(uint2*)qo; *(uint2*)(k_e + o) = *(uint2*)ko; *(uint2*)(v_e + o) = vr;
  const float* bar = ba + (size_t)t * ldb;
  const float al = __expf(a_log[hv]);
  if (per_channel) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = hv * 128 + lane * 4 + j;
      const float x = bar[Hv + c] + dt_bias[c];
      g[(size_t)t * Hv * 128 + c] = __expf(-al * (x > 20.f ? x : log1pf(__expf(x))));
    }
  } else if (lane == 0) {
    const float x = bar[Hv + hv] + dt_bias[hv];
    g[(size_t)t * Hv + hv] = __expf(-al * (x > 20.f ? x : log1pf(__expf(x))));
  }
  if (lane == 0) beta[(size_t)t * Hv + hv] = 1.f / (1.f + __expf(-bar[hv]));
}

extern "C" int cuteafd_linear_prepare(const void* conv, const float* ba, const float* a_log, const float* dt_bias, void* q_e, void* k_e, void* v_e,
                                      float* g, float* beta, int T, int Hk, int Hv, int ldb, int per_channel, cudaStream_t s) {
  CA_REQUIRE(conv && ba && a_log && dt_bias && q_e && k_e && v_e && g && beta && Hk >= 1 && Hv % Hk == 0, "linear_prepare: bad arguments");
  if (T <= 0) return CA_OK;
  const long long threads = (long long)T * Hv * 32;
  CA_LAUNCH_PDL(linear_prepare_kernel, (int)((threads + 255) / 256), 256, 0, s, (const bf16*)conv, ba, a_log, dt_bias, (bf16*)q_e, (bf16*)k_e, (bf16*)v_e, g,
                beta, T, Hk, Hv, ldb, per_channel);
  CA_CHECK_LAUNCH("linear_prepare");
  return CA_OK;
}

// out[t, h * 128 + :] = rmsnorm(o[t, h, :]) * w * silu(z[t, h, :]); z lives at column z_off of rows with pitch ldz (the z part of the
// fused input projection).  One warp per (token, head).
__global__ void gated_rmsnorm_kernel(const bf16* __restrict__ o, const bf16* __restrict__ z, const float* __restrict__ w, bf16* __restrict__ out, int T, int H,
                                     int ldz, int z_off, float eps) {
  pdl_launch(); pdl_wait();
  const int wi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (wi >= T * H) return;
  const int t = wi / H, h = wi % H;
  const uint2 orw = *(const uint2*)(o + ((size_t)t * H + h) * 128 + lane * 4), zr = *(const uint2*)(z + (size_t)t * ldz + z_off + h * 128 + lane * 4);
  const bf16* oe = (const bf16*)&orw; const bf16* ze = (const bf16*)&zr;
  float v[4], ss = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) { v[j] = __bfloat162float(oe[j]); ss += v[j] * v[j]; }
  const float inv = rsqrtf(warp_sum(ss) / 128.f + eps);
  bf16 r[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float zz = __bfloat162float(ze[j]);
    const float n = __bfloat162float(__float2bfloat16(v[j] * inv * w[lane * 4 + j]));        // the norm's bf16 output, as the stand-alone kernel rounds it
    r[j] = __float2bfloat16(n * (zz / (1.f + __expf(-zz))));
  }
  *(uint2*)(out + ((size_t)t * H + h) * 128 + lane * 4) = *(uint2*)r;
}

extern "C" int cuteafd_gated_rmsnorm(const void* o, const void* z, const float* w, void* out, int T, int H, int ldz, int z_off, float eps, cudaStream_t s) {
  CA_REQUIRE(o && z && w && out && ldz % 4 == 0 && z_off % 4 == 0, "gated_rmsnorm: bad arguments");
  if (T <= 0) return CA_OK;
  const long long threads = (long long)T * H * 32;
  CA_LAUNCH_PDL(gated_rmsnorm_kernel, (int)((threads + 255) / 256), 256, 0, s, (const bf16*)o, (const bf16*)z, w, (bf16*)out, T, H, ldz, z_off, eps);
  CA_CHECK_LAUNCH("gated_rmsnorm");
  return CA_OK;
}
