// Wide tcgen05 GEMM for prompt-sized steps on sm_100a:  Y[rows, N] = X[rows, K] * W[N, K]^T  (dense or grouped per expert), bf16, NVFP4,
// MXFP4, and FP8 with one fp32 scale per 128 x 128 weights and 1 x 128 activations.
//
// Decode steps put the weights on the MMA's M side, because few tokens must not waste it.  Here there are tokens enough: a tile is 128 tokens
// (M) x 256 weight rows (N; or 128 rows of the gate and the same 128 of the up weight), which reads 12 KB of shared memory per instruction of
// 128 x 256 outputs - the narrow kernel's 32-token tiles read 5 KB for 128 x 32, and its instructions cost their minimum time whatever N
// (measured: 4096 tokens x 8 of 128 experts, NVFP4, K 4096, 2 x 1536 columns: 1380 us there).  Tokens as tensor-memory lanes also give every
// epilogue thread 64 or 128 consecutive features of ONE row: block maxima and packing of an FP4 output need no shuffles, and every store
// is a whole 32-byte sector.
//
// One persistent CTA per SM, 384 threads: warp 0 loads by TMA, warp 1 issues the MMAs, warp 2 stages FP4 activation scales, warps 4..11 are
// the epilogue (two per tensor-memory lane quarter, one per half of the columns).  Units go round robin, weight tiles innermost, so that the
// units in flight share a few token tiles and read each expert's weights from HBM once and from L2 after that.
//   bf16, FP4: a 256-column accumulator.  The epilogue warps first read all of it into registers (128 per thread) and release it, so only
//   that read (about 400 cycles) lies between two units' MMAs; the arithmetic and the stores run under the next unit's main loop.
//   Of a K in parts every part is read and added to registers before the next one starts.
//   FP8: two 256-column buffers; every 128 channels of K is one product of its own, which the epilogue warps add, times its two scales, to
//   fp32 registers: one FMA per output and scale block, because a thread's row has one activation scale and its 128 columns one weight scale.
// What bounds it: the four products of a stage take 512 cycles whatever the kind, over 48 KB of operands (54 KB with FP4 scales).  Measured cycles a stage, and what the
// issuer waits for in them:
//   bf16, 4096 x 12288 x 2048                    686   operands 549 (the producer 326 for a free stage), accumulator 21
//   NVFP4 / MXFP4, 4096 x 9216 x 4096            987 / 970   operands 531 / 469 (producer 123 / 117), then activation scales 192 / 147, accumulator 30
//   FP8, 2048 x 7168 x 16384; 2048 x 24576 x 1536   754; 1169   accumulator 419; 761 (the epilogue's promotion), operands 153; 193
// So FP4 waits for loads that are in flight, four stages of them (reads from L2 run at 38 % of their peak, in bf16 at 50 %), and FP8 for the epilogue.
#define CA_PDL_CLASS 1
#include "tc_gemm_wide.cuh"
#include "tc_issue.cuh"

namespace {
enum { W_BF16 = 0, W_NVFP4 = 1, W_MXFP4 = 2, W_FP8 = 3 };
enum { WEPI_BF16 = 0, WEPI_BF16_RESIDUAL = 1, WEPI_F32 = 3 };

template <int KIND>
struct WideCfg {
  static constexpr bool FP4 = KIND == W_NVFP4 || KIND == W_MXFP4;
  static constexpr int ISSUE = KIND == W_BF16 ? TI_F16 : KIND == W_NVFP4 ? TI_NVF4 : KIND == W_MXFP4 ? TI_MXF4 : TI_F8;
  static constexpr int X_BYTES = 128 * 128, W_BYTES = 2 * 128 * 128;
  static constexpr int CHUNKS = KIND == W_NVFP4 ? 4 : (KIND == W_MXFP4 ? 2 : 0);       // 512-byte scale chunks per 128 rows and stage
  static constexpr int SFX_BYTES = CHUNKS * 512, SFW_BYTES = 2 * CHUNKS * 512;
  static constexpr int STAGE_BYTES = X_BYTES + W_BYTES + SFX_BYTES + SFW_BYTES;
  static constexpr int NSTAGE = 4;
  static constexpr int SMEM_BYTES = NSTAGE * STAGE_BYTES + 1024;
  static constexpr int K_ELEMS = KIND == W_BF16 ? 64 : (KIND == W_FP8 ? 128 : 256);    // 128 bytes of every row
  static constexpr int KX = KIND == W_BF16 ? 64 : 128;                                 // the same in elements of the descriptors' type
  static constexpr int SF_COL = 256;        // scales, two buffers of 64 columns: 16 of the activations, 32 of the weights
  static_assert(SMEM_BYTES <= 227 * 1024, "stages exceed shared memory");
};

__device__ __forceinline__ void tmem_ld_x32(uint32_t addr, float* r) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
               : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]),
                 "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]),
                 "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31]) : "r"(addr));
}
__device__ __forceinline__ void st_32b(void* p, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}
__device__ __forceinline__ void ld_32b(const void* p, uint32_t* w) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(p) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) { const bf162 h = __floats2bfloat162_rn(a, b); return *(const uint32_t*)&h; }

template <int KIND>
__device__ __forceinline__ uint32_t wide_idesc() {
  uint32_t d = ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  if (KIND == W_BF16) d |= (1u << 4) | (1u << 7) | (1u << 10);             // fp32 accumulator, bf16 x bf16
  else if (KIND == W_FP8) d |= 1u << 4;                                     // fp32 accumulator, E4M3 x E4M3
  else {
    d |= (1u << 7) | (1u << 10);                                            // E2M1 x E2M1
    if (KIND == W_MXFP4) d |= 1u << 23;                                     // UE8M0 scales
  }
  return d;
}

struct Unit { int g, row0, nrows, nt; };
__device__ __forceinline__ Unit unit_of(const WideArgs& a, int w, int n_nt) {
  const int item = w / n_nt;
  Unit u = {0, item * 128, 128, w - item * n_nt};
  if (a.tiles) { const int4 t = a.tiles[item]; u.g = t.x; u.row0 = t.y; u.nrows = t.z; }
  u.nrows = min(u.nrows, a.rows_total - u.row0);
  return u;
}

// A thread's features n0 .. of one output row, from its accumulators: scale, activation, residual, stores.
template <int KIND, bool SWIGLU, bool QOUT, bool PARTS>
__device__ __forceinline__ void wide_finish(const WideArgs& a, float* acc, int g, size_t row, int n0) {
  constexpr int NF = SWIGLU ? 64 : 128;
  const int nf = min(NF, a.N - n0);
  const float al = a.alpha ? a.alpha[g] : 1.f;
  if (SWIGLU) {
    const float al2 = a.alpha2 ? a.alpha2[g] : al;
#pragma unroll
    for (int j = 0; j < 64; ++j) {
      const float v = acc[j] * al, up = acc[64 + j] * al2;
      acc[j] = v / (1.f + __expf(-v)) * up;
    }
  } else {
    if (KIND != W_FP8 && !PARTS) {
#pragma unroll
      for (int j = 0; j < 128; ++j) acc[j] *= al;
    }
    if (!PARTS && a.act) {
#pragma unroll
      for (int j = 0; j < 128; ++j) { const float v = fmaxf(acc[j], 0.f); acc[j] = v * v; }
    }
  }
  if (QOUT) {
    const float inv_gs = (KIND == W_NVFP4 && a.inv_gs_out) ? *a.inv_gs_out : 1.f;
    constexpr int BLK = KIND == W_MXFP4 ? 32 : 16;
    uint32_t codes[8];
    uint32_t scales = 0;
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = __bfloat162float(__float2bfloat16(acc[j]));
#pragma unroll
    for (int b = 0; b < 64 / BLK; ++b) {
      float am = 0.f;
#pragma unroll
      for (int j = 0; j < BLK; ++j) am = fmaxf(am, fabsf(acc[b * BLK + j]));
      float eff; uint8_t sb;
      if (KIND == W_MXFP4) {
        int e = am > 0.f ? (int)((__float_as_uint(am) >> 23) & 0xFF) - 2 : 0;
        e = max(e, 0); e = min(e, 254); sb = (uint8_t)e; eff = ue8m0_to_float(sb);
      } else {
        sb = float_to_e4m3(fminf(am * inv_gs / 6.f, 448.f)); eff = e4m3_to_float(sb) / inv_gs;
      }
      const float inv = eff > 0.f ? 1.f / eff : 0.f;
      scales |= (uint32_t)sb << (8 * b);
#pragma unroll
      for (int o = 0; o < BLK / 8; ++o) {
        float t[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) t[j] = acc[b * BLK + o * 8 + j] * inv;
        codes[b * (BLK / 8) + o] = pack_e2m1x8(t);
      }
    }
    uint8_t* qp = a.q_out + row * (a.N / 2) + n0 / 2;
    uint8_t* sp = a.sf_out + row * a.ldsf_out + n0 / BLK;
    if (nf == 64 && ((uintptr_t)qp & 31) == 0) st_32b(qp, codes);
    else {
#pragma unroll
      for (int o = 0; o < 8; ++o)
        if (o * 8 < nf) *(uint32_t*)(qp + o * 4) = codes[o];
    }
#pragma unroll
    for (int b = 0; b < 64 / BLK; ++b)
      if (b * BLK < nf) sp[b] = (uint8_t)(scales >> (8 * b));
    if (!a.Y) return;
  }
  const size_t o = row * a.ldy + n0;
  const bool aligned = nf == NF && (((uintptr_t)a.Y | ((uintptr_t)a.ldy * (a.epi == WEPI_F32 ? 4 : 2))) & 31) == 0 &&
                       (a.epi != WEPI_BF16_RESIDUAL || ((uintptr_t)a.R & 31) == 0);
  if (aligned) {
    if (a.epi == WEPI_F32) {
#pragma unroll
      for (int j = 0; j < NF; j += 8) st_32b((float*)a.Y + o + j, (const uint32_t*)(acc + j));
    } else {
#pragma unroll
      for (int j = 0; j < NF; j += 16) {
        uint32_t wv[8];
        if (a.epi == WEPI_BF16_RESIDUAL) {
          uint32_t rv[8];
          ld_32b(a.R + o + j, rv);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const bf162 r2 = *(const bf162*)&rv[q];
            wv[q] = pack_bf16(acc[j + 2 * q] + __bfloat162float(r2.x), acc[j + 2 * q + 1] + __bfloat162float(r2.y));
          }
        } else {
#pragma unroll
          for (int q = 0; q < 8; ++q) wv[q] = pack_bf16(acc[j + 2 * q], acc[j + 2 * q + 1]);
        }
        st_32b((bf16*)a.Y + o + j, wv);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < NF; ++j)
      if (j < nf) {
        if (a.epi == WEPI_F32) ((float*)a.Y)[o + j] = acc[j];
        else ((bf16*)a.Y)[o + j] = __float2bfloat16(a.epi == WEPI_BF16_RESIDUAL ? acc[j] + __bfloat162float(a.R[o + j]) : acc[j]);
      }
  }
}

// PARTS (an instance of its own: its registers cost the others 2 %): K in a.parts sums.
template <int KIND, bool SWIGLU, bool QOUT, bool PARTS>
__global__ void __launch_bounds__(384, 1) gemm_wide_kernel(const __grid_constant__ WideArgs a) {
  using C = WideCfg<KIND>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[C::NSTAGE], empty_bar[C::NSTAGE], accf_bar[2], acce_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::NSTAGE; ++s) { mbar_init(&full_bar[s], C::FP4 ? 33 : 1); mbar_init(&empty_bar[s], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&accf_bar[i], 1); mbar_init(&acce_bar[i], 256); }
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_launch();
  pdl_wait();

  const int n_items = a.tiles ? *a.n_tiles : (a.rows_total + 127) / 128;
  const int n_nt = SWIGLU ? (a.N + 127) / 128 : (a.N + 255) / 256;
  const int n_wb = (a.N + 127) / 128;                                       // 128-row blocks of a weight
  const int nkb = (a.K + C::K_ELEMS - 1) / C::K_ELEMS;
  const int total = n_items * n_nt;
  const int parts = PARTS ? a.parts : 1;
  volatile int* abortp = &abort_flag;

  // Registers: 64,512 at launch (384 x 168); 128 x 64 + 256 x 216 = 63,488 of them after the split.
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      if (lane == 0) {
        uint32_t it = 0;
        for (int w = blockIdx.x; w < total && !*abortp; w += gridDim.x) {
          const Unit u = unit_of(a, w, n_nt);
          const CUtensorMap* m0 = a.tmW + u.g;
          const CUtensorMap* m1 = SWIGLU ? a.tmW2 + u.g : m0;
          const int b0 = SWIGLU ? u.nt : u.nt * 2, b1 = SWIGLU ? u.nt : u.nt * 2 + 1;     // the tile's two weight blocks; rows past N are zeros
          for (int kb = 0; kb < nkb; ++kb, ++it) {
            const int s = it % C::NSTAGE;
            if (!mbar_wait_bounded(&empty_bar[s], ((it / C::NSTAGE) & 1) ^ 1, abortp)) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_PRODUCER, w); break; }
            uint8_t* sX = smem + s * C::STAGE_BYTES, *sW = sX + C::X_BYTES, *sSW = sW + C::W_BYTES + C::SFX_BYTES;
            mbar_expect_tx(&full_bar[s], C::X_BYTES + C::W_BYTES + C::SFW_BYTES);
            tma_load_3d(sX, a.tmX, &full_bar[s], kb * C::KX, u.row0, 0);
            tma_load_3d(sW, m0, &full_bar[s], kb * C::KX, b0 * 128, 0);
            tma_load_3d(sW + C::W_BYTES / 2, m1, &full_bar[s], kb * C::KX, b1 * 128, 0);
            if (C::FP4) {
              const size_t o0 = ((size_t)b0 * nkb + kb) * C::SFX_BYTES, o1 = ((size_t)min(b1, n_wb - 1) * nkb + kb) * C::SFX_BYTES;
              bulk_load_1d(sSW, a.sfw[u.g] + o0, C::SFX_BYTES, &full_bar[s]);
              bulk_load_1d(sSW + C::SFX_BYTES, (SWIGLU ? a.sfw2[u.g] : a.sfw[u.g]) + o1, C::SFX_BYTES, &full_bar[s]);
            }
          }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      // (the whole warp, under an elected lane's predicate: tc_issue.cuh)
      uint32_t it = 0, tc = 0;
      const uint32_t x0 = ti_desc(smem_u32(smem)), sx0 = ti_desc_sf(smem_u32(smem) + C::X_BYTES + C::W_BYTES);
      bool ok = true;
      for (int w = blockIdx.x; ok && w < total && !__any_sync(0xffffffffu, *abortp); w += gridDim.x)
      for (int part = 0; part < parts; ++part) {
        const int kb0 = PARTS ? (int)((long long)nkb * part / parts) : 0, kb1 = PARTS ? (int)((long long)nkb * (part + 1) / parts) : nkb;
        if (PARTS && kb0 == kb1) continue;
        if (KIND != W_FP8) {
          if (!mbar_wait_warp(&acce_bar[0], (tc & 1) ^ 1, abortp)) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_MMA, w); ok = false; break; }
          tc_fence_after();
        }
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t s = it % C::NSTAGE, b = it & 1;
          if (KIND == W_FP8 && !mbar_wait_warp(&acce_bar[b], ((it >> 1) & 1) ^ 1, abortp)) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_MMA, w); ok = false; break; }
          if (!mbar_wait_warp(&full_bar[s], (it / C::NSTAGE) & 1, abortp)) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_MMA, w); ok = false; break; }
          tc_fence_after();
          const uint32_t off = s * (C::STAGE_BYTES / 16), cx = tmem + C::SF_COL + b * 64, cw = cx + 16;
          if (C::FP4) {
#pragma unroll
            for (int q = 0; q < C::CHUNKS; ++q) {
              const uint32_t chunk = sx0 + off + q * 32;
              ti_cp_sf(cx + 4 * q, chunk);
              ti_cp_sf(cw + 8 * q, chunk + C::SFX_BYTES / 16);
              ti_cp_sf(cw + 8 * q + 4, chunk + C::SFX_BYTES / 8);
            }
          }
          ti_mma4<C::ISSUE, 4, 8>(tmem + (KIND == W_FP8 ? b * 256 : 0), x0 + off, x0 + off + C::X_BYTES / 16, wide_idesc<KIND>(), KIND == W_FP8 ? 0u : (kb > kb0 ? 1u : 0u), cx, cw);
          ti_commit(&empty_bar[s]);
          if (KIND == W_FP8) ti_commit(&accf_bar[b]);
        }
        if (!ok) break;
        ++tc;
        if (KIND != W_FP8) ti_commit(&accf_bar[0]);
      }
      __syncwarp();
    } else if (warp == 2 && C::FP4) {
      // ---------------------------------------------------------------- activation scales
      // A lane's 16 bytes of a 512-byte chunk are four scales each of rows lane, lane + 32, + 64, + 96: it reads the stage's scales of these
      // rows whole, two stages ahead of the ring, and writes one 16-byte word per chunk (4-byte cp.async straight into the layout looked up
      // 512 cache lines a stage and bounded the main loop: 124 us against 98 for 4096 x 9216 x 4096 NVFP4).
      uint32_t it = 0;
      for (int w = blockIdx.x; w < total && !*abortp; w += gridDim.x) {
        const Unit u = unit_of(a, w, n_nt);
        uint32_t v[2][4][4];
        auto fetch = [&](int kb, uint32_t (&r)[4][4]) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = j * 32 + lane;
            const bool live = c < u.nrows && kb < nkb;
            const uint8_t* src = a.sfx + (size_t)(u.row0 + c) * a.ldsfx + (size_t)kb * (C::CHUNKS * 4);
            if (C::CHUNKS == 4) {
              const uint4 t = live ? *(const uint4*)src : make_uint4(0u, 0u, 0u, 0u);
              r[j][0] = t.x; r[j][1] = t.y; r[j][2] = t.z; r[j][3] = t.w;
            } else {
              const uint2 t = live ? *(const uint2*)src : make_uint2(0u, 0u);
              r[j][0] = t.x; r[j][1] = t.y;
            }
          }
        };
        fetch(0, v[0]);
        fetch(1, v[1]);
        bool ok = true;
        for (int kb0 = 0; kb0 < nkb && ok; kb0 += 2) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int kb = kb0 + e;
            if (kb >= nkb || !ok) break;
            const int s = it % C::NSTAGE;
            ok = mbar_wait_bounded(&empty_bar[s], ((it / C::NSTAGE) & 1) ^ 1, abortp);
            if (!ok) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_PRODUCER, w); break; }
            uint8_t* sSX = smem + s * C::STAGE_BYTES + C::X_BYTES + C::W_BYTES + lane * 16;
#pragma unroll
            for (int q = 0; q < C::CHUNKS; ++q) *(uint4*)(sSX + q * 512) = make_uint4(v[e][0][q], v[e][1][q], v[e][2][q], v[e][3][q]);
            fence_proxy_async_smem();
            mbar_arrive(&full_bar[s]);
            ++it;
            fetch(kb + 2, v[e]);
          }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------------------------------------------ epilogue
    const int q4 = warp & 3, h = (warp - 4) >> 2;
    const uint32_t tbase = tmem + ((uint32_t)(q4 * 32) << 16);
    uint32_t it = 0, tc = 0;
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
      if (__any_sync(0xffffffffu, *abortp)) break;                         // the warp stays together
      const Unit u = unit_of(a, w, n_nt);
      const int trow = q4 * 32 + lane;
      const bool live = trow < u.nrows;
      const size_t row = (size_t)(u.row0 + trow);
      float acc[128];
      bool ok = true;
      if (KIND == W_FP8) {
#pragma unroll
        for (int j = 0; j < 128; ++j) acc[j] = 0.f;
        const int wb = min(SWIGLU ? u.nt : u.nt * 2 + h, n_wb - 1);
        const float* swp = a.sw + (size_t)wb * nkb;
        const float* sxp = a.sx + (live ? row : 0) * nkb;
        // scales of four blocks at a time, the next four on their way under them (one row's scales are strided by the row: every load of
        // a warp is 32 sectors, and one block ahead was not enough to hide it)
        const bool vec = nkb % 4 == 0 && (((uintptr_t)a.sx | (uintptr_t)a.sw) & 15) == 0;
        auto fetch = [&](int kb, float (&x)[4], float (&y)[4]) {
          if (vec) {
            if (kb < nkb) {
              const float4 fx = *(const float4*)(sxp + kb), fy = *(const float4*)(swp + kb);
              x[0] = fx.x; x[1] = fx.y; x[2] = fx.z; x[3] = fx.w;
              y[0] = fy.x; y[1] = fy.y; y[2] = fy.z; y[3] = fy.w;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (kb + e < nkb) { x[e] = sxp[kb + e]; y[e] = swp[kb + e]; }
          }
        };
        float sx[4] = {}, sw[4] = {}, sxn[4] = {}, swn[4] = {};
        fetch(0, sx, sw);
        for (int kb0 = 0; kb0 < nkb && ok; kb0 += 4) {
          fetch(kb0 + 4, sxn, swn);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (kb0 + e >= nkb) break;
            const int b = it & 1;
            const float sc = sx[e] * sw[e];
            ok = mbar_wait_bounded(&accf_bar[b], (it >> 1) & 1, abortp);
            ok = __all_sync(0xffffffffu, ok);                              // tensor-memory loads stay warp-uniform
            if (!ok) break;
            tc_fence_after();
            float p[2][16];                                                // the next 16 columns are on their way under these 16's FMAs
            tmem_ld_x16(tbase + b * 256 + h * 128, (uint32_t*)p[0]);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              tc_wait_ld();
              if (c < 7) tmem_ld_x16(tbase + b * 256 + h * 128 + (c + 1) * 16, (uint32_t*)p[(c + 1) & 1]);
              else { tc_fence_before(); mbar_arrive(&acce_bar[b]); }
#pragma unroll
              for (int j = 0; j < 16; ++j) acc[c * 16 + j] = fmaf(p[c & 1][j], sc, acc[c * 16 + j]);
            }
            ++it;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) { sx[e] = sxn[e]; sw[e] = swn[e]; }
        }
        if (!ok) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_EPILOGUE, w); break; }
      } else if (PARTS) {
        // every part times the output scale, one after the other to fp32 registers: the sums that a split over CTAs adds up, without its trip through
        // memory (the read of a part's accumulator, 400 cycles, is not hidden)
        const float al = a.alpha ? a.alpha[u.g] : 1.f;
#pragma unroll
        for (int j = 0; j < 128; ++j) acc[j] = 0.f;
        for (int part = 0; part < parts; ++part) {
          if ((long long)nkb * part / parts == (long long)nkb * (part + 1) / parts) continue;
          ok = mbar_wait_bounded(&accf_bar[0], tc & 1, abortp);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          float p[2][16];
          tmem_ld_x16(tbase + h * 128, (uint32_t*)p[0]);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            tc_wait_ld();
            if (c < 7) tmem_ld_x16(tbase + h * 128 + (c + 1) * 16, (uint32_t*)p[(c + 1) & 1]);
            else { tc_fence_before(); mbar_arrive(&acce_bar[0]); }
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[c * 16 + j] = __fadd_rn(acc[c * 16 + j], __fmul_rn(p[c & 1][j], al));
          }
          ++tc;
        }
        if (!ok) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_EPILOGUE, w); break; }
      } else {
        ok = mbar_wait_bounded(&accf_bar[0], tc & 1, abortp);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { ca_dev_fail(a.status, CA_DEV_TIMEOUT_EPILOGUE, w); break; }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 4; ++c)      // two-weight form: 64 columns of the gate, then the same 64 of the up half
          tmem_ld_x32(tbase + (SWIGLU ? (c >> 1) * 128 + h * 64 + (c & 1) * 32 : h * 128 + c * 32), acc + c * 32);
        tc_wait_ld();
        tc_fence_before();
        mbar_arrive(&acce_bar[0]);
        ++tc;
      }
      const int n0 = SWIGLU ? u.nt * 128 + h * 64 : u.nt * 256 + h * 128;
      if (live && n0 < a.N) wide_finish<KIND, SWIGLU, QOUT, PARTS>(a, acc, u.g, row, n0);
      __syncwarp();
    }
  }

  // ------------------------------------------------------------------ teardown
  if (*abortp && warp == 0) {
    // give copies already in flight time to land before shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int KIND, bool SWIGLU, bool QOUT, bool PARTS = false>
int launch_wide(const WideArgs& a, int grid, cudaStream_t stream) {
  using C = WideCfg<KIND>;
  auto kern = gemm_wide_kernel<KIND, SWIGLU, QOUT, PARTS>;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return ca_cuda(e, "cudaFuncSetAttribute(gemm_wide)");
    attr_set[dev & 63] = true;
  }
  CA_LAUNCH_PDL(kern, grid, 384, C::SMEM_BYTES, stream, a);
  return CA_OK;
}
}  // namespace

int ca_gemm_wide(int kind, bool swiglu, const WideArgs& a, long long max_items, cudaStream_t stream) {
  const long long units = max_items * (swiglu ? (a.N + 127) / 128 : (a.N + 255) / 256);
  const int grid = (int)(units < ca_sm_count() ? (units > 0 ? units : 1) : ca_sm_count());
  if (a.parts > 1) {
    if (swiglu || a.tiles || a.act) return ca_fail(CA_ERR_ARG, "gemm_wide: parts of K belong to plain dense products");
    if (kind == W_BF16) return launch_wide<W_BF16, false, false, true>(a, grid, stream);
#ifndef CA_TC_BF16_ONLY
    if (kind == W_NVFP4) return launch_wide<W_NVFP4, false, false, true>(a, grid, stream);
    if (kind == W_MXFP4) return launch_wide<W_MXFP4, false, false, true>(a, grid, stream);
#endif
    return ca_fail(CA_ERR_UNSUPPORTED, "gemm_wide: no kernel in parts for operand kind %d", kind);
  }
  if (kind == W_BF16) return swiglu ? launch_wide<W_BF16, true, false>(a, grid, stream) : launch_wide<W_BF16, false, false>(a, grid, stream);
#ifndef CA_TC_BF16_ONLY
  if (kind == W_FP8) return launch_wide<W_FP8, false, false>(a, grid, stream);
  if (kind == W_NVFP4) return !swiglu ? launch_wide<W_NVFP4, false, false>(a, grid, stream) : a.q_out ? launch_wide<W_NVFP4, true, true>(a, grid, stream) : launch_wide<W_NVFP4, true, false>(a, grid, stream);
  if (kind == W_MXFP4) return !swiglu ? launch_wide<W_MXFP4, false, false>(a, grid, stream) : a.q_out ? launch_wide<W_MXFP4, true, true>(a, grid, stream) : launch_wide<W_MXFP4, true, false>(a, grid, stream);
#endif
  return ca_fail(CA_ERR_UNSUPPORTED, "gemm_wide: no kernel for operand kind %d", kind);
}
