// Projection post-processing: RoPE on q/k, the theta-rotated noise query, lambda / gate sigmoids.
// HBM-bound elementwise work (reads q,k once, writes q,k,q_noise once).
// Two kernels with the same arithmetic: prep_vec_kernel moves 16-byte vectors (a thread owns whole RoPE pairs AND
// whole noise-rotation pairs, so nothing crosses threads) and is used whenever rows are 16-byte aligned and the head
// dimension allows, a CTA per tile of positions x states; prep_kernel is the element-wise fallback for any layout, a CTA per token.
#include "coda_common.cuh"

struct PrepParams {
  int B, L, H, Hkv, Dh, interleaved, gated;
  coda_ring_pos rp; int W;
  void* q; long long q_bs, q_rs;
  void* k; long long k_bs, k_rs;
  void* qn;
  const void* lam_logit; long long lam_bs, lam_rs; float* lam;
  const void* gate_logit; long long gate_bs, gate_rs; float* gate;
  const float* inv_freq; const void* cos_t; const void* sin_t;
};

// T: activation dtype, A: dtype the angles are evaluated in.
template <typename T, typename A>
__global__ void __launch_bounds__(256) prep_kernel(PrepParams p) {
  extern __shared__ float sm[];
  const int half = p.Dh >> 1;
  float* cs = sm;                 // [half] cos, rounded to T
  float* sn = sm + half;          // [half] sin
  float* qrow = sm + 2 * half;    // [H*Dh] rotated query row (noise rotation pairs cross RoPE pairs)
  const int tid = threadIdx.x, NT = blockDim.x;
  const long long ntok = (long long)p.B * p.L;
  // In a decode graph the position comes from the step counter; prefill passes step_dev == NULL.
  const long long pos_base = ring_now(p.rp, p.W).pos;
  for (long long tok = blockIdx.x; tok < ntok; tok += gridDim.x) {
    const int b = (int)(tok / p.L), t = (int)(tok % p.L);
    const long long pos = pos_base + t;
    for (int i = tid; i < half; i += NT) {
      // upstream primitives.py:51-54: t = arange(dtype=inv_freq.dtype); freqs = t (x) inv_freq; cos().to(dtype)
      float ta = El<A>::rnd((float)pos);
      float inv = El<A>::rnd(p.inv_freq[i]);
      float ang = El<A>::rnd(__fmul_rn(ta, inv));
      cs[i] = El<T>::rnd(El<A>::rnd(cosf(ang)));
      sn[i] = El<T>::rnd(El<A>::rnd(sinf(ang)));
    }
    __syncthreads();
    T* qt = (T*)p.q + (long long)b * p.q_bs + (long long)t * p.q_rs;
    T* kt = p.k ? (T*)p.k + (long long)b * p.k_bs + (long long)t * p.k_rs : nullptr;
    const int nq = p.H * half, nk = p.k ? p.Hkv * half : 0;
    for (int w = tid; w < nq + nk; w += NT) {
      const bool isq = w < nq;
      const int ww = isq ? w : w - nq;
      const int h = ww / half, i = ww % half;
      T* row = (isq ? qt : kt) + h * p.Dh;
      const float c = cs[i], s = sn[i];
      int ia, ib;
      float oa, ob;
      if (p.interleaved) {                  // primitives.py:99-106
        ia = 2 * i; ib = 2 * i + 1;
        const float xe = El<T>::ld(row + ia), xo = El<T>::ld(row + ib);
        oa = t_sub<T>(t_mul<T>(xe, c), t_mul<T>(xo, s));
        ob = t_add<T>(t_mul<T>(xe, s), t_mul<T>(xo, c));
      } else {                              // primitives.py:108-113: x*cos_full + rotate_half(x)*sin_full
        ia = i; ib = i + half;
        const float x1 = El<T>::ld(row + ia), x2 = El<T>::ld(row + ib);
        oa = t_add<T>(t_mul<T>(x1, c), t_mul<T>(-x2, s));
        ob = t_add<T>(t_mul<T>(x2, c), t_mul<T>(x1, s));
      }
      El<T>::st(row + ia, oa);
      El<T>::st(row + ib, ob);
      if (isq) { qrow[h * p.Dh + ia] = oa; qrow[h * p.Dh + ib] = ob; }
    }
    __syncthreads();
    T* qnt = (T*)p.qn + tok * (long long)(p.H * p.Dh);
    for (int w = tid; w < nq; w += NT) {    // primitives.py:58-80, always (even, odd) pairs
      const int h = w / half, i = w % half;
      const float qe = qrow[h * p.Dh + 2 * i], qo = qrow[h * p.Dh + 2 * i + 1];
      const float ct = El<T>::ld((const T*)p.cos_t + h * half + i);
      const float st = El<T>::ld((const T*)p.sin_t + h * half + i);
      El<T>::st(qnt + h * p.Dh + 2 * i, t_sub<T>(t_mul<T>(qe, ct), t_mul<T>(qo, st)));
      El<T>::st(qnt + h * p.Dh + 2 * i + 1, t_add<T>(t_mul<T>(qe, st), t_mul<T>(qo, ct)));
    }
    for (int h = tid; h < p.H; h += NT) {
      const float z = El<T>::ld((const T*)p.lam_logit + (long long)b * p.lam_bs + (long long)t * p.lam_rs + h);
      p.lam[tok * p.H + h] = t_sigmoid<T>(z);
    }
    if (tid == 0 && p.gate != nullptr) {
      float g = 1.0f;                       // write_policy "none": attention.py:407-408
      if (p.gated) g = t_sigmoid<T>(El<T>::ld((const T*)p.gate_logit + (long long)b * p.gate_bs + (long long)t * p.gate_rs));
      p.gate[tok] = g;
    }
    __syncthreads();
  }
}

// Vectorised variant.  Work item = one 16-byte chunk of a head row (interleaved pairs) or the two chunks c and
// c + Dh/2 that hold each other's RoPE partners (half-split pairs).  The noise query always rotates (even, odd)
// neighbours of the ROTATED row (primitives.py:58-80), which lie inside one chunk, so an item is self-contained.
//
// One CTA = a tile of `tt` consecutive positions of `nb` states: the states of a batch stand at the same positions, so
// the cos / sin tables of the tile are evaluated once, all entries at the same time (an accurate sine is a chain of
// some thousand cycles; one table per token is what bounded this kernel), and the tile's (token, item) pairs are dealt
// out flat, so that a narrow layer's tokens, which have fewer items than a CTA has threads, leave none idle.
// Bound: HBM (q and k in, q, k and the noise query out); what hides its latency is the number of resident threads, hence
// the register limit and no per-thread state across items (tables from shared memory, the learned rotation from L1).
// Measured, cold L2: 131072 tokens of a 512-wide layer 516 -> 123 us (3.8 TB/s), 131072 of a 576-wide 520 -> 118 us,
// 16384 of a 4096-wide 102 -> 85 us, 8192 of an 8192-wide 86 -> 79 us (5.5 TB/s); three CTAs per SM with item state kept
// in registers 98..130 us at 4096, five (32 registers, spilling) 97 us.
template <typename T> struct Item;
template <> struct Item<bf16> {             // tables as packed words; the arithmetic is one instruction per element pair
  uint4 cv, sv;                             // half-split: cos / sin of angles 8c..8c+7; interleaved: pairs 4c..4c+3, each word duplicated
  uint2 ca, sa, cb, sb;                     // learned rotation of the first / second chunk's four pairs
  static __device__ __forceinline__ uint2 ld2(const bf16* p) { return *reinterpret_cast<const uint2*>(p); }
  static __device__ __forceinline__ uint4 dup4(const uint2& w) { return make_uint4(bdup_lo(w.x), bdup_hi(w.x), bdup_lo(w.y), bdup_hi(w.y)); }
  static __device__ __forceinline__ uint4 turn(const uint4& x, const uint4& c, const uint4& s) {
    return make_uint4(brot(x.x, c.x, s.x), brot(x.y, c.y, s.y), brot(x.z, c.z, s.z), brot(x.w, c.w, s.w));
  }
  static __device__ __forceinline__ uint4 mix(const uint4& a, const uint4& c, const uint4& b, const uint4& s) {   // a c + b s
    return make_uint4(badd2(bmul2(a.x, c.x), bmul2(b.x, s.x)), badd2(bmul2(a.y, c.y), bmul2(b.y, s.y)),
                      badd2(bmul2(a.z, c.z), bmul2(b.z, s.z)), badd2(bmul2(a.w, c.w), bmul2(b.w, s.w)));
  }
  __device__ __forceinline__ void tables(const bf16* csb, const bf16* snb, bool inter, int c) {
    if (inter) { cv = dup4(ld2(csb + 4 * c)); sv = dup4(ld2(snb + 4 * c)); }
    else { cv = *reinterpret_cast<const uint4*>(csb + 8 * c); sv = *reinterpret_cast<const uint4*>(snb + 8 * c); }
  }
  __device__ __forceinline__ void theta(const bf16* cth, const bf16* sth, bool inter, int c, int half) {
    ca = ld2(cth + 4 * c); sa = ld2(sth + 4 * c);
    if (!inter) { cb = ld2(cth + (half >> 1) + 4 * c); sb = ld2(sth + (half >> 1) + 4 * c); }
  }
  __device__ __forceinline__ uint4 rope_pairs(const uint4& x) const { return turn(x, cv, sv); }
  __device__ __forceinline__ void rope_halves(const uint4& x1, const uint4& x2, uint4& oa, uint4& ob) const {     // x1 c + (-x2) s ; x2 c + x1 s
    oa = mix(x1, cv, make_uint4(bneg2(x2.x), bneg2(x2.y), bneg2(x2.z), bneg2(x2.w)), sv);
    ob = mix(x2, cv, x1, sv);
  }
  __device__ __forceinline__ uint4 noise_a(const uint4& o) const { return turn(o, dup4(ca), dup4(sa)); }
  __device__ __forceinline__ uint4 noise_b(const uint4& o) const { return turn(o, dup4(cb), dup4(sb)); }
};
template <> struct Item<float> {
  float c[4], s[4];                         // half-split: angles 4c..4c+3; interleaved: pairs 2c, 2c+1 (first two)
  float ta[2], ua[2], tb[2], ub[2];         // learned rotation cos / sin of the two pairs of the first / second chunk
  static __device__ __forceinline__ float f(uint32_t w) { return __uint_as_float(w); }
  static __device__ __forceinline__ uint32_t u(float v) { return __float_as_uint(v); }
  static __device__ __forceinline__ uint4 turn(const uint4& x, float c0, float s0, float c1, float s1) {
    return make_uint4(u(t_sub<float>(t_mul<float>(f(x.x), c0), t_mul<float>(f(x.y), s0))), u(t_add<float>(t_mul<float>(f(x.x), s0), t_mul<float>(f(x.y), c0))),
                      u(t_sub<float>(t_mul<float>(f(x.z), c1), t_mul<float>(f(x.w), s1))), u(t_add<float>(t_mul<float>(f(x.z), s1), t_mul<float>(f(x.w), c1))));
  }
  __device__ __forceinline__ void tables(const float* cs, const float* sn, bool inter, int ch) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = inter ? 2 * ch + (e & 1) : 4 * ch + e;
      c[e] = cs[i]; s[e] = sn[i];
    }
  }
  __device__ __forceinline__ void theta(const float* cth, const float* sth, bool inter, int ch, int half) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      ta[e] = cth[2 * ch + e]; ua[e] = sth[2 * ch + e];
      if (!inter) { tb[e] = cth[(half >> 1) + 2 * ch + e]; ub[e] = sth[(half >> 1) + 2 * ch + e]; }
    }
  }
  __device__ __forceinline__ uint4 rope_pairs(const uint4& x) const { return turn(x, c[0], s[0], c[1], s[1]); }
  __device__ __forceinline__ void rope_halves(const uint4& x1, const uint4& x2, uint4& oa, uint4& ob) const {
    const uint32_t a[4] = {x1.x, x1.y, x1.z, x1.w}, b[4] = {x2.x, x2.y, x2.z, x2.w};
    uint32_t p[4], q[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      p[e] = u(t_add<float>(t_mul<float>(f(a[e]), c[e]), t_mul<float>(-f(b[e]), s[e])));
      q[e] = u(t_add<float>(t_mul<float>(f(b[e]), c[e]), t_mul<float>(f(a[e]), s[e])));
    }
    oa = make_uint4(p[0], p[1], p[2], p[3]); ob = make_uint4(q[0], q[1], q[2], q[3]);
  }
  __device__ __forceinline__ uint4 noise_a(const uint4& o) const { return turn(o, ta[0], ua[0], ta[1], ua[1]); }
  __device__ __forceinline__ uint4 noise_b(const uint4& o) const { return turn(o, tb[0], ub[0], tb[1], ub[1]); }
};

// ONE: the tile is one token (calls with no more tokens than give every CTA slot of two waves one): the divisions that deal the
// tile out are left out, where nothing hides them (64 to 2048 tokens of a 512-wide fp32 layer 3.6 .. 11.3 -> 3.2 .. 9.1 us).
template <typename T, typename A, bool INTER, bool ONE>
__global__ void __launch_bounds__(320, 4) prep_vec_kernel(PrepParams p, int tt, int nb) {
  constexpr int N = 16 / (int)sizeof(T);    // elements per 16-byte chunk
  extern __shared__ __align__(16) unsigned char prep_sm[];
  const int half = p.Dh >> 1;
  T* tab = reinterpret_cast<T*>(prep_sm);   // [tt][cos half | sin half], entries rounded to T
  const int tid = threadIdx.x, NT = blockDim.x;
  const int t0 = ONE ? blockIdx.x : blockIdx.x * tt, tn = ONE ? 1 : min(tt, p.L - t0);
  const int b0 = ONE ? blockIdx.y : blockIdx.y * nb, bn = ONE ? 1 : min(nb, p.B - b0);
  constexpr int CH = INTER ? 1 : 2;         // chunks of an item
  const int per_head = p.Dh / (N * CH);     // items per head row
  const int nq = p.H * per_head, nit = nq + (p.k ? p.Hkv * per_head : 0), ntok = tn * bn;
  const long long pos = ring_now(p.rp, p.W).pos + t0;
  for (int i = tid; i < tn * half; i += NT) {
    // upstream primitives.py:51-54: t = arange(dtype=inv_freq.dtype); freqs = t (x) inv_freq; cos().to(dtype)
    const int ti = ONE ? 0 : i / half, j = i - ti * half;
    float ta = El<A>::rnd((float)(pos + ti));
    float inv = El<A>::rnd(p.inv_freq[j]);
    float ang = El<A>::rnd(__fmul_rn(ta, inv));
    float cc, ss; sincos_call(ang, &ss, &cc);
    El<T>::st(tab + ti * p.Dh + j, El<T>::rnd(El<A>::rnd(cc)));
    El<T>::st(tab + ti * p.Dh + half + j, El<T>::rnd(El<A>::rnd(ss)));
  }
  // lambda and gate sigmoids of the tile's tokens: item (token, head), the head after the last one being the gate
  for (int i = tid; i < ntok * (p.H + 1); i += NT) {
    const int u = ONE ? 0 : i / (p.H + 1), hh = i - u * (p.H + 1), tq = ONE ? 0 : u / bn, bq = b0 + u - tq * bn, ta = t0 + tq;
    const long long tok = (long long)bq * p.L + ta;
    if (hh < p.H) {
      p.lam[tok * p.H + hh] = t_sigmoid<T>(El<T>::ld((const T*)p.lam_logit + (long long)bq * p.lam_bs + (long long)ta * p.lam_rs + hh));
    } else if (p.gate != nullptr) {
      float g = 1.0f;                       // write_policy "none": attention.py:407-408
      if (p.gated) g = t_sigmoid<T>(El<T>::ld((const T*)p.gate_logit + (long long)bq * p.gate_bs + (long long)ta * p.gate_rs));
      p.gate[tok] = g;
    }
  }
  __syncthreads();
  for (int i = tid; i < ntok * nit; i += NT) {
    const int u = ONE ? 0 : i / nit, w = i - u * nit, t = ONE ? 0 : u / bn, b = b0 + u - t * bn;
    const bool isq = w < nq;
    const int ww = isq ? w : w - nq, h = ww / per_head, c = ww - h * per_head;
    T* row = (isq ? (T*)p.q : (T*)p.k) + (long long)b * (isq ? p.q_bs : p.k_bs) + (long long)(t0 + t) * (isq ? p.q_rs : p.k_rs) + h * p.Dh + c * N;
    T* nrow = (T*)p.qn + ((long long)b * p.L + t0 + t) * (long long)(p.H * p.Dh) + h * p.Dh + c * N;
    Item<T> it;
    if (INTER) {                            // primitives.py:99-106: pairs (2i, 2i+1) share cos/sin i
      const uint4 x = *reinterpret_cast<const uint4*>(row);
      if (isq) it.theta((const T*)p.cos_t + h * half, (const T*)p.sin_t + h * half, INTER, c, half);
      it.tables(tab + t * p.Dh, tab + t * p.Dh + half, INTER, c);
      const uint4 o = it.rope_pairs(x);
      *reinterpret_cast<uint4*>(row) = o;
      if (isq) *reinterpret_cast<uint4*>(nrow) = it.noise_a(o);
    } else {                                // primitives.py:108-113: x*cos_full + rotate_half(x)*sin_full
      const uint4 x1 = *reinterpret_cast<const uint4*>(row), x2 = *reinterpret_cast<const uint4*>(row + half);
      if (isq) it.theta((const T*)p.cos_t + h * half, (const T*)p.sin_t + h * half, INTER, c, half);
      it.tables(tab + t * p.Dh, tab + t * p.Dh + half, INTER, c);
      uint4 oa, ob;
      it.rope_halves(x1, x2, oa, ob);
      *reinterpret_cast<uint4*>(row) = oa;
      *reinterpret_cast<uint4*>(row + half) = ob;
      if (isq) { *reinterpret_cast<uint4*>(nrow) = it.noise_a(oa); *reinterpret_cast<uint4*>(nrow + half) = it.noise_b(ob); }
    }
  }
}

extern "C" int coda_b200_prep(const coda_layer_cfg* cfg, int32_t L, coda_ring_pos rp,
                              void* q, int64_t q_bs, int64_t q_rs,
                              void* k, int64_t k_bs, int64_t k_rs,
                              void* q_noise,
                              const void* lam_logit, int64_t lam_bs, int64_t lam_rs, float* lam,
                              const void* gate_logit, int64_t gate_bs, int64_t gate_rs, float* gate,
                              const float* inv_freq, const void* cos_theta, const void* sin_theta,
                              coda_stream_t stream) {
  CODA_REQUIRE(coda_cfg_ok(cfg), CODA_ERR_ARG, "prep: invalid layer configuration");
  CODA_REQUIRE(L >= 0, CODA_ERR_ARG, "prep: negative L");
  if (L == 0) return CODA_OK;
  CODA_REQUIRE(q && q_noise && lam_logit && lam && inv_freq && cos_theta && sin_theta, CODA_ERR_ARG, "prep: null pointer");
  CODA_REQUIRE(!(cfg->gated && gate && !gate_logit), CODA_ERR_ARG, "prep: gated write policy needs gate logits");
  PrepParams p;
  p.B = cfg->B; p.L = L; p.H = cfg->H; p.Hkv = cfg->Hkv; p.Dh = cfg->Dh;
  p.interleaved = cfg->rope_interleaved; p.gated = cfg->gated; p.rp = rp; p.W = cfg->W;
  p.q = q; p.q_bs = q_bs; p.q_rs = q_rs; p.k = k; p.k_bs = k_bs; p.k_rs = k_rs; p.qn = q_noise;
  p.lam_logit = lam_logit; p.lam_bs = lam_bs; p.lam_rs = lam_rs; p.lam = lam;
  p.gate_logit = gate_logit; p.gate_bs = gate_bs; p.gate_rs = gate_rs; p.gate = gate;
  p.inv_freq = inv_freq; p.cos_t = cos_theta; p.sin_t = sin_theta;
  const long long ntok = (long long)cfg->B * L;
  const int grid = (int)(ntok < 148LL * 16 ? ntok : 148LL * 16);
  const size_t smem = sizeof(float) * (size_t)(cfg->Dh + cfg->H * cfg->Dh);
  CODA_REQUIRE(smem <= 200 * 1024, CODA_ERR_LIMIT, "prep: H*Dh = %d exceeds the shared-memory row limit", cfg->H * cfg->Dh);
  cudaStream_t s = (cudaStream_t)stream;
  // 16-byte vectors need aligned rows and chunks that do not straddle a RoPE half / head row
  const int vn = cfg->dtype == CODA_F32 ? 4 : 8;
  const bool vec = ((cfg->rope_interleaved ? cfg->Dh : cfg->Dh / 2) % vn) == 0 && ((uintptr_t)q | (uintptr_t)q_noise) % 16 == 0 &&
                   (q_bs | q_rs) % vn == 0 && (k == nullptr || ((uintptr_t)k % 16 == 0 && (k_bs | k_rs) % vn == 0));
  // Tile of a CTA: positions so that the tables' entries keep the threads busy once, then states; no larger than leaves
  // two waves of four CTAs per SM.
  const long long share = ntok / (148LL * 8) > 1 ? ntok / (148LL * 8) : 1;
  int tt = 320 / (cfg->Dh / 2);
  tt = tt < 1 ? 1 : (tt > 8 ? 8 : tt);
  if (tt > share) tt = (int)share;
  if (tt > L) tt = L;
  long long nb = share / tt;
  nb = nb < 1 ? 1 : (nb > cfg->B ? cfg->B : nb);
  while ((cfg->B + nb - 1) / nb > 65535) ++nb;
#define LAUNCH(T, A) do { \
    if (vec) { \
      const dim3 vgrid((unsigned)((L + tt - 1) / tt), (unsigned)((cfg->B + nb - 1) / nb)); \
      const size_t vsmem = sizeof(T) * (size_t)cfg->Dh * tt; \
      if (tt == 1 && nb == 1) { \
        if (cfg->rope_interleaved) prep_vec_kernel<T, A, true, true><<<vgrid, 320, vsmem, s>>>(p, 1, 1); \
        else prep_vec_kernel<T, A, false, true><<<vgrid, 320, vsmem, s>>>(p, 1, 1); \
        break; \
      } \
      if (cfg->rope_interleaved) prep_vec_kernel<T, A, true, false><<<vgrid, 320, vsmem, s>>>(p, tt, (int)nb); \
      else prep_vec_kernel<T, A, false, false><<<vgrid, 320, vsmem, s>>>(p, tt, (int)nb); \
      break; \
    } \
    if (smem > 48 * 1024) cudaFuncSetAttribute(prep_kernel<T, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    prep_kernel<T, A><<<grid, 256, smem, s>>>(p); } while (0)
  if (cfg->dtype == CODA_F32) {
    CODA_REQUIRE(cfg->angle_dtype == CODA_F32, CODA_ERR_ARG, "prep: fp32 activations need fp32 angles");
    LAUNCH(float, float);
  } else if (cfg->angle_dtype == CODA_BF16) {
    LAUNCH(bf16, bf16);
  } else {
    LAUNCH(bf16, float);
  }
#undef LAUNCH
  CODA_CHECK_LAUNCH("prep");
  return CODA_OK;
}
