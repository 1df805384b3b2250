// Split-KV partial merge shared by the SIMT and the tensor-core paged attention kernels.
#pragma once
#include "common.cuh"
#include "attn_extras.cuh"

// Merge split partials: out = sum_s o_s * exp(m_s - M) / sum_s l_s * exp(m_s - M)  (+ sink term).
// Splits that saw no key carry m = -inf, l = 0 and drop out.  Partials of rows a split never touched are
// ignored through the `valid` test on m.
static __global__ void attn_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, const float* __restrict__ sink,
                                  bf16* __restrict__ out, int T, int Hq, int D, int n_splits) {
  pdl_launch(); pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y;
  float M = sink ? sink[h] : -INFINITY;
  for (int s = 0; s < n_splits; ++s) M = fmaxf(M, part_ml[(((size_t)s * T + t) * Hq + h) * 2]);
  float L = sink ? __expf(sink[h] - M) : 0.f;
  for (int s = 0; s < n_splits; ++s) {
    const float* ml = part_ml + (((size_t)s * T + t) * Hq + h) * 2;
    if (ml[0] != -INFINITY) L += ml[1] * __expf(ml[0] - M);
  }
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float o = 0.f;
    for (int s = 0; s < n_splits; ++s) {
      const float m = part_ml[(((size_t)s * T + t) * Hq + h) * 2];
      if (m != -INFINITY) o += part_o[(((size_t)s * T + t) * Hq + h) * D + d] * __expf(m - M);
    }
    out[((size_t)t * Hq + h) * D + d] = __float2bfloat16(L > 0.f ? o / L : 0.f);
  }
}

// The merge for eight output elements of one (row, head): partial i lies at row0 + i * step of `part_ml` (pairs) and `part_o` (D columns), its
// columns from d0 on.  FRESH: other blocks of this kernel have just written them (no read-only cache).  Leaves the unnormalised sum in o and
// its denominator in L.
// Up to eight partials at a time, every load issued before the first use: the (m, l) pairs and the partial rows are in flight together (a loop
// that reads m, branches, then loads the row is one L2 round trip per partial on a decode step's critical path).  Partial rows of empty
// splits (m = -inf) are loaded but not used; the buffers always cover every split.
template <bool FRESH>
__device__ __forceinline__ void attn_merge8(const float* part_o, const float* part_ml, bool sink, float sk, size_t row0, size_t step, int n, int D, int d0, float (&o)[8], float& L) {
  float M = sk;
  L = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) o[q] = 0.f;
  for (int s0 = 0; s0 < n; s0 += 8) {
    float2 ml[8]; float4 pa[8], pb[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const size_t row = row0 + min(s0 + j, n - 1) * step;
      const float2* pm = (const float2*)(part_ml + row * 2);
      const float4* po = (const float4*)(part_o + row * D + d0);
      if (FRESH) { ml[j] = __ldcg(pm); pa[j] = __ldcg(po); pb[j] = __ldcg(po + 1); }
      else { ml[j] = __ldg(pm); pa[j] = __ldg(po); pb[j] = __ldg(po + 1); }
    }
    float Mn = M;
#pragma unroll
    for (int j = 0; j < 8; ++j) if (s0 + j < n) Mn = fmaxf(Mn, ml[j].x);
    if (s0 == 0) {
      if (sink) L = __expf(sk - Mn);                    // the sink's share first, as the one-pass form adds it
    } else if (Mn != M && M != -INFINITY) {           // a later batch raised the maximum: rescale what was accumulated
      const float r = __expf(M - Mn);
      L *= r;
#pragma unroll
      for (int q = 0; q < 8; ++q) o[q] *= r;
    }
    M = Mn;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (s0 + j < n && ml[j].x != -INFINITY) {
        const float e = __expf(ml[j].x - M);
        L += ml[j].y * e;
        o[0] += pa[j].x * e; o[1] += pa[j].y * e; o[2] += pa[j].z * e; o[3] += pa[j].w * e;
        o[4] += pb[j].x * e; o[5] += pb[j].y * e; o[6] += pb[j].z * e; o[7] += pb[j].w * e;
      }
    }
  }
}

// Eight merged elements -> bf16 `ob` and the output row (the first Dout of a head's D columns, head h at column h * Dout of rows ldo apart).
__device__ __forceinline__ void attn_store8(const AttnExtras<bf16>& x, bf16* out, int t, int h, int d0, int Dout, int ldo, float (&o)[8], float L, bf16 (&ob)[8]) {
  const float inv = (L > 0.f ? 1.f / L : 0.f) * x.head_factor(t, h);
  if (x.gate && x.gate_values) {
#pragma unroll
    for (int j = 0; j < 8; ++j) if (d0 + j < Dout) o[j] *= x.value_factor(t, h * Dout + d0 + j);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) ob[j] = __float2bfloat16(o[j] * inv);
  bf16* dst = out + (size_t)t * ldo + (size_t)h * Dout + d0;
  if (((Dout | ldo) & 7) == 0) { if (d0 < Dout) *(uint4*)dst = *(uint4*)ob; }
  else {
#pragma unroll
    for (int j = 0; j < 8; ++j) if (d0 + j < Dout) dst[j] = ob[j];
  }
}

// That merge as a launch, eight output elements per thread, optionally also writing the merged row quantised to FP4 for the
// output projection that follows (qkind 1 NVFP4 / 2 MXFP4; needs Hq * D % 256 == 0).  grid (T, ceil(Hq * D / 8 / 128)).
static __global__ void attn_merge8_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, const AttnExtras<bf16> x,
                                          bf16* __restrict__ out, int T, int Hq, int D, int Dout, int ldo, int n_splits, uint8_t* __restrict__ q,
                                          uint8_t* __restrict__ sf, int ldsf, const float* __restrict__ inv_gs_ptr, int qkind) {
  pdl_launch(); pdl_wait();
  const int t = blockIdx.x, vi = blockIdx.y * blockDim.x + threadIdx.x, vpr = D / 8;
  if (vi >= Hq * vpr) return;                     // whole warps leave together (Hq * D / 8 is a multiple of 32 with FP4 output)
  const int h = vi / vpr, d0 = (vi % vpr) * 8;
  float o[8], L;
  attn_merge8<false>(part_o, part_ml, x.sink != nullptr, x.sink ? x.sink[h] : -INFINITY, (size_t)t * Hq + h, (size_t)T * Hq, n_splits, D, d0, o, L);
  bf16 ob[8];
  attn_store8(x, out, t, h, d0, Dout, ldo, o, L, ob);
  if (qkind) {
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(ob[j]);
    quant8_store(f, qkind, inv_gs_ptr ? *inv_gs_ptr : 1.f, q + (size_t)t * (Hq * D / 2), sf + (size_t)t * ldsf, h * D + d0);
  }
}

static __global__ void attn_fill_ml_kernel(float* ml, long long n) {
  pdl_launch(); pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ml[i] = (i & 1) ? 0.f : -INFINITY;
}

