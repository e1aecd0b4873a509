// Differential attention in single precision, register-tiled: head_dim 32, 64 or 128, 16-byte aligned rows.
//
// One CTA = one (state, query head, query tile); its WARPS warps split the keys: warp w takes the 32-key tiles w, w+WARPS,
// ... of the visible slots followed by the block's own tokens (causal), each with a running softmax of its own, and the
// partial results are merged once at the end (fixed order, no atomics).  The ROWS rows of a tile are the queries'
// signal vectors followed by their noise vectors, so both streams use every staged K/V element.  Per tile a warp
// computes S as 4 row groups x 8 key groups of TM x 4 register tiles (K and Q read from shared memory as 16-byte
// vectors along Dh), leaves P transposed in its own shared memory, and accumulates P.V as TM rows x Dh/8 columns per
// lane.  K and V sit in one buffer each, refilled by cp.async as soon as the tile's Q.K^T (P.V) is done, so a refill
// has the other half of the tile's arithmetic to arrive in; warps never wait for one another inside the loop.
// Bound: FMA issue.  A row per warp and a key per lane (attend_generic) reads shared memory once per FMA and keeps
// few warps in flight.
// 256 queries of 8 heads over 384 slots + their own block, Dh 64: 219 -> 35 us.
// The instance follows the call, not the batch (a state's result does not depend on its neighbours):
// * queries per CTA: 8 (TM = 4) for blocks, 4 (TM = 2) and 2 (TM = 1) for calls of up to four and two, whose
//   larger tile would be padding;
// * warps: four, or as many as there are key tiles (one, two).  A warp without a tile still holds its buffers, and at Dh 128
//   four warps' are a whole SM's: 800 heads of one query over 64 slots take 19.1 us with two warps, 46.1 with four (generic:
//   34.7); over 32 slots 10.1 with one, 45.6 with four (19.0).
#include "coda_common.cuh"
#include "attend_f32.h"
#include <type_traits>

namespace {

constexpr int AF_TK = 32;        // keys per warp tile

__device__ __forceinline__ void cp16(void* dst, const void* src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = ok ? 16 : 0;     // 0: the destination is filled with zeros, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int DH, int TM, int WARPS>
struct AfLayout {
  static constexpr int ROWS = 4 * TM;          // rows of a tile, both streams
  static constexpr int BQ = ROWS / 2;          // queries of a tile
  static constexpr int QS = DH + 4;            // row strides in floats: 16-byte vectors of 8 neighbouring rows hit
  static constexpr int KS = DH + 4;            // different banks
  static constexpr int PS = ROWS + 4;
  static constexpr int WARP = AF_TK * KS + AF_TK * DH + AF_TK * PS;     // floats of one warp: K, V, P
  static constexpr int FLOATS = ROWS * QS + WARPS * WARP + 2 * WARPS * ROWS;
};

template <int DH, int TM, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) attend_f32_kernel(AttnParams p) {
  typedef AfLayout<DH, TM, WARPS> Lay;
  constexpr int ROWS = Lay::ROWS, BQ = Lay::BQ, QS = Lay::QS, KS = Lay::KS, PS = Lay::PS;
  constexpr int CH = DH / 4;                   // 16-byte chunks per row
  constexpr int NC = DH / 32;                  // 16-byte column chunks of the output per lane
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = lane >> 3, kg = lane & 7;
  const int b = blockIdx.z, h = blockIdx.y, hk = h / (p.H / p.Hkv), q0 = blockIdx.x * BQ;
  float* Qs = sm;                              // [ROWS][QS]
  float* Ks = Qs + ROWS * QS + warp * Lay::WARP;   // [TK][KS]
  float* Vs = Ks + AF_TK * KS;                 // [TK][DH]
  float* Ps = Vs + AF_TK * DH;                 // [TK][PS]
  float* Ms = sm + ROWS * QS + WARPS * Lay::WARP;   // [WARPS][ROWS] maxima, then sums
  float* Ls = Ms + WARPS * ROWS;

  const bool has_blk = p.kblk != nullptr;
  const int nblk_keys = has_blk ? min(q0 + BQ, p.Lq) : 0;
  const int nkeys = p.Lbuf + nblk_keys, ntiles = (nkeys + AF_TK - 1) / AF_TK;
  const float* kbase = (const float*)p.kbuf + ((long long)b * p.Hkv + hk) * p.Lbuf * DH;
  const float* vbase = (const float*)p.vbuf + ((long long)b * p.Hkv + hk) * p.Lbuf * DH;
  const float* kblk = (const float*)p.kblk + (long long)b * p.kb_bs + hk * DH;
  const float* vblk = (const float*)p.vblk + (long long)b * p.vb_bs + hk * DH;
  const uint8_t* al = p.allowed + (long long)b * p.Lbuf;

  // visibility of key j as far as it is the same for every query: slots, and block tokens up to the tile's last query
  auto key_ok = [&](int j) { return j < p.Lbuf ? (!p.mask_unused || al[j] != 0) : j < nkeys; };
  // the first tile at or after t (of this warp's) with such a key, and its mask
  auto next_tile = [&](int t, unsigned& bits) {
    for (; t < ntiles; t += WARPS) {
      bits = __ballot_sync(0xffffffffu, key_ok(t * AF_TK + lane));
      if (bits != 0u) break;
    }
    return t;
  };
  auto load = [&](float* dst, int stride, const float* base, const float* blk, long long blk_rs, int t) {
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int c = lane + 32 * i, r = c / CH, cc = c % CH, j = t * AF_TK + r;
      const float* src = j < p.Lbuf ? base + (long long)j * DH : blk + (long long)(j - p.Lbuf) * blk_rs;
      cp16(dst + r * stride + cc * 4, j < nkeys ? src + cc * 4 : base, j < nkeys);
    }
    cp_commit();
  };

  grid_chain();
  unsigned bits = 0u;
  int t = next_tile(warp, bits);
  if (t < ntiles) { load(Ks, KS, kbase, kblk, p.kb_rs, t); load(Vs, DH, vbase, vblk, p.vb_rs, t); }
  for (int c = tid; c < ROWS * CH; c += WARPS * 32) {
    const int r = c / CH, cc = c % CH, q = q0 + (r % BQ);
    const float* src = r < BQ ? (const float*)p.q + (long long)b * p.q_bs + (long long)q * p.q_rs
                              : (const float*)p.qn + (long long)b * p.qn_bs + (long long)q * p.qn_rs;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q < p.Lq) x = *reinterpret_cast<const float4*>(src + h * DH + cc * 4);
    *reinterpret_cast<float4*>(Qs + r * QS + cc * 4) = x;
  }
  __syncthreads();

  float m[TM], l[TM], acc[TM][NC * 4];
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < NC * 4; ++c) acc[i][c] = 0.f;
  }
  while (t < ntiles) {
    const bool nok = t + WARPS < ntiles && key_ok((t + WARPS) * AF_TK + lane);   // (arrives under Q.K^T)
    cp_wait<1>();                              // this tile's K (V is the younger group)
    __syncwarp();
    float s[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i) { s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f; }
#pragma unroll 4
    for (int d = 0; d < CH; ++d) {
      float4 kv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(Ks + (kg + 8 * j) * KS + d * 4);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 qv = *reinterpret_cast<const float4*>(Qs + (rg * TM + i) * QS + d * 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = fmaf(qv.x, kv[j].x, s[i][j]); s[i][j] = fmaf(qv.y, kv[j].y, s[i][j]);
          s[i][j] = fmaf(qv.z, kv[j].z, s[i][j]); s[i][j] = fmaf(qv.w, kv[j].w, s[i][j]);
        }
      }
    }
    __syncwarp();
    int tn = t + WARPS;
    unsigned nbits = __ballot_sync(0xffffffffu, nok);
    if (nbits == 0u) tn = next_tile(tn + WARPS, nbits);
    if (tn < ntiles) load(Ks, KS, kbase, kblk, p.kb_rs, tn); else cp_commit();
    // visibility (the causal limit differs between the queries), running maximum, probabilities
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int lim = p.Lbuf + q0 + (rg * TM + i) % BQ;             // block keys j <= lim are visible to this row
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kk = kg + 8 * j;
        const bool vis = ((bits >> kk) & 1u) && (t * AF_TK + kk < p.Lbuf || t * AF_TK + kk <= lim);
        s[i][j] = vis ? s[i][j] * p.scale_log2 : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
      const float nm = fmaxf(m[i], mx);
      const float ref = nm == -INFINITY ? 0.f : nm;                 // nothing visible to this row yet: all weights 0
      const float a = exp2f(m[i] - ref);
      m[i] = nm;
      l[i] *= a;
#pragma unroll
      for (int j = 0; j < 4; ++j) { s[i][j] = exp2f(s[i][j] - ref); l[i] += s[i][j]; }
#pragma unroll
      for (int c = 0; c < NC * 4; ++c) acc[i][c] *= a;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float* pr = Ps + (kg + 8 * j) * PS + rg * TM;
      if constexpr (TM == 4) *reinterpret_cast<float4*>(pr) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
      else {
#pragma unroll
        for (int i = 0; i < TM; ++i) pr[i] = s[i][j];
      }
    }
    cp_wait<1>();                              // this tile's V (the next K is the younger group)
    __syncwarp();
    // A key behind a row's causal limit is left out, not multiplied by its zero weight: a token whose values are
    // infinite or not a number must not reach the outputs of the tokens before it.  Only the tiles that hold the
    // diagonal ask.
    auto accumulate = [&](auto diagonal) {
#pragma unroll 4
      for (int kk = 0; kk < AF_TK; ++kk) {
        float w[TM];
        if constexpr (TM == 4) {
          const float4 pv = *reinterpret_cast<const float4*>(Ps + kk * PS + rg * 4);
          w[0] = pv.x; w[1] = pv.y; w[2] = pv.z; w[3] = pv.w;
        } else {
#pragma unroll
          for (int i = 0; i < TM; ++i) w[i] = Ps[kk * PS + rg * TM + i];
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const float4 vv = *reinterpret_cast<const float4*>(Vs + kk * DH + (kg + 8 * c) * 4);
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            if (diagonal.value && t * AF_TK + kk > p.Lbuf + q0 + (rg * TM + i) % BQ) continue;
            acc[i][4 * c] = fmaf(w[i], vv.x, acc[i][4 * c]); acc[i][4 * c + 1] = fmaf(w[i], vv.y, acc[i][4 * c + 1]);
            acc[i][4 * c + 2] = fmaf(w[i], vv.z, acc[i][4 * c + 2]); acc[i][4 * c + 3] = fmaf(w[i], vv.w, acc[i][4 * c + 3]);
          }
        }
      }
    };
    if ((t + 1) * AF_TK > p.Lbuf + q0 + 1 && has_blk) accumulate(std::true_type());
    else accumulate(std::false_type());
    __syncwarp();
    if (tn < ntiles) load(Vs, DH, vbase, vblk, p.vb_rs, tn); else cp_commit();
    t = tn; bits = nbits;
  }
  cp_wait<0>();

  // ---- merge of the four warps: exponents moved to the common maximum, partial O left where the warp's K was ----
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 4);
    if (kg == 0) { Ms[warp * ROWS + rg * TM + i] = m[i]; Ls[warp * ROWS + rg * TM + i] = l[i]; }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = rg * TM + i;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, Ms[w * ROWS + r]);
    const float f = m[i] == -INFINITY ? 0.f : exp2f(m[i] - mm);
#pragma unroll
    for (int c = 0; c < NC; ++c)
      *reinterpret_cast<float4*>(Ks + r * DH + (kg + 8 * c) * 4) =
          make_float4(acc[i][4 * c] * f, acc[i][4 * c + 1] * f, acc[i][4 * c + 2] * f, acc[i][4 * c + 3] * f);
  }
  __syncthreads();

  // ---- epilogue: sig - lam*noise, optional RMSNorm over Dh (attention.py:463-464, primitives.py:23-27); a warp per query
  for (int qi = warp; qi < BQ && q0 + qi < p.Lq; qi += WARPS) {
    const int row = q0 + qi;
    const float lam = p.lam[(long long)b * p.lam_bs + (long long)row * p.lam_rs + h];
    float il[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int r = s * BQ + qi;
      float mm = -INFINITY, ll = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, Ms[w * ROWS + r]);
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const float mw = Ms[w * ROWS + r];
        ll += mw == -INFINITY ? 0.f : Ls[w * ROWS + r] * exp2f(mw - mm);
      }
      il[s] = ll > 0.f ? 1.f / ll : 0.f;
    }
    float diff[NC], sq = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      float o[2] = {0.f, 0.f};
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const float* po = sm + ROWS * QS + w * Lay::WARP;
        o[0] += po[qi * DH + lane + 32 * c];
        o[1] += po[(BQ + qi) * DH + lane + 32 * c];
      }
      diff[c] = t_sub<float>(o[0] * il[0], t_mul<float>(lam, o[1] * il[1]));
      sq += diff[c] * diff[c];
    }
    float* op = (float*)p.out + (long long)b * p.out_bs + (long long)row * p.out_rs + h * DH;
    const float rs = p.norm_full ? rsqrtf(warp_sum(sq) / (float)DH + p.eps) : 1.f;
#pragma unroll
    for (int c = 0; c < NC; ++c)
      op[lane + 32 * c] = p.norm_full ? t_mul<float>(t_mul<float>(diff[c], rs), ((const float*)p.norm_w)[lane + 32 * c]) : diff[c];
  }
}

template <int DH, int TM, int WARPS>
int launch(const AttnParams& p, cudaStream_t s) {
  typedef AfLayout<DH, TM, WARPS> Lay;
  static_assert(Lay::ROWS <= AF_TK, "partial rows are left in the K buffer");
  constexpr int bytes = Lay::FLOATS * 4;
  static coda_device_once once;
  coda_on_first_use(once, [] { cudaFuncSetAttribute(attend_f32_kernel<DH, TM, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); });
  coda_launch_chained(attend_f32_kernel<DH, TM, WARPS>, dim3((p.Lq + Lay::BQ - 1) / Lay::BQ, p.H, p.B), dim3(WARPS * 32), bytes, s, 1, p);
  CODA_CHECK_LAUNCH("attend (f32)");
  return CODA_OK;
}

template <int DH, int TM>
int launch_warps(const AttnParams& p, cudaStream_t s) {
  const int tiles = (p.Lbuf + (p.kblk != nullptr ? p.Lq : 0) + AF_TK - 1) / AF_TK;
  return tiles <= 1 ? launch<DH, TM, 1>(p, s) : tiles <= 2 ? launch<DH, TM, 2>(p, s) : launch<DH, TM, 4>(p, s);
}

template <int DH>
int launch_rows(const AttnParams& p, cudaStream_t s) {
  return p.Lq <= 2 ? launch_warps<DH, 1>(p, s) : p.Lq <= 4 ? launch_warps<DH, 2>(p, s) : launch_warps<DH, 4>(p, s);
}

}  // namespace

bool coda_attend_f32_supported(const AttnParams& p) {
  if (p.Dh != 32 && p.Dh != 64 && p.Dh != 128) return false;
  const uintptr_t ptrs = (uintptr_t)p.q | (uintptr_t)p.qn | (uintptr_t)p.kbuf | (uintptr_t)p.vbuf | (uintptr_t)p.kblk | (uintptr_t)p.vblk;
  long long strides = p.q_bs | p.q_rs | p.qn_bs | p.qn_rs;
  if (p.kblk != nullptr) strides |= p.kb_bs | p.kb_rs | p.vb_bs | p.vb_rs;
  return ptrs % 16 == 0 && strides % 4 == 0;
}

int coda_attend_f32(const AttnParams& p, cudaStream_t s) {
  return p.Dh == 32 ? launch_rows<32>(p, s) : p.Dh == 64 ? launch_rows<64>(p, s) : launch_rows<128>(p, s);
}
