// Routing caches of a fresh state: the unit vectors of every bank slot (values of the exact bank, the phase-safe half of the
// keys of the summary bank), as upstream's two F.normalize calls per state (attention.py:300-317).
// Bound: launches.  As tensor operations this is ten of them (norm, clamp, division, copies, twice) on a few hundred KB,
// some 70 us of host time in the first call of every new sequence; here one, a warp per (slot, head).
#include "coda_common.cuh"

namespace {

template <typename T>
__global__ void __launch_bounds__(128) bank_norms_kernel(coda_layer_cfg c, coda_state_ptrs st) {
  const int lane = threadIdx.x & 31, b = blockIdx.y;
  const int W = c.W, Me = c.Me, Ms = c.Ms, Dh = c.Dh, lf = Dh / 2, Lbuf = W + Me + Ms;
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= (Me + Ms) * c.Hkv) return;
  const int h = item / (Me + Ms), m = item % (Me + Ms);
  const bool exact = m < Me;
  const int n = exact ? Dh : Dh - lf;
  const T* row = (const T*)(exact ? st.v_buf : st.k_buf) + (((long long)b * c.Hkv + h) * Lbuf + W + m) * Dh + (exact ? 0 : lf);
  T* out = exact ? (T*)st.exact_v_norm + (((long long)b * c.Hkv + h) * Me + m) * Dh
                 : (T*)st.sum_lf_k_norm + (((long long)b * c.Hkv + h) * Ms + m - Me) * n;
  float ss = 0.f;
  for (int d = lane; d < n; d += 32) { const float v = El<T>::ld(row + d); ss = fmaf(v, v, ss); }
  const float den = fmaxf(El<T>::rnd(sqrtf(warp_sum(ss))), El<T>::rnd(1e-6f));
  for (int d = lane; d < n; d += 32) El<T>::st(out + d, t_div<T>(El<T>::ld(row + d), den));
}

}  // namespace

extern "C" int coda_b200_bank_norms(const coda_layer_cfg* cfg, const coda_state_ptrs* st, coda_stream_t stream) {
  CODA_REQUIRE(coda_cfg_ok(cfg) && st, CODA_ERR_ARG, "bank_norms: invalid layer configuration");
  const int slots = cfg->Me + cfg->Ms;
  if (slots == 0) return CODA_OK;
  CODA_REQUIRE(st->k_buf && st->v_buf && (cfg->Me == 0 || st->exact_v_norm) && (cfg->Ms == 0 || st->sum_lf_k_norm) && cfg->B <= 65535,
               CODA_ERR_ARG, "bank_norms: null pointer or too many states");
  const dim3 grid((slots * cfg->Hkv + 3) / 4, cfg->B);
  if (cfg->dtype == CODA_F32) bank_norms_kernel<float><<<grid, 128, 0, (cudaStream_t)stream>>>(*cfg, *st);
  else bank_norms_kernel<bf16><<<grid, 128, 0, (cudaStream_t)stream>>>(*cfg, *st);
  CODA_CHECK_LAUNCH("bank_norms");
  return CODA_OK;
}
