// Bank + ring update with one prefill block, as four chained launches:
//   route_score   cosine scores of every candidate against the routing caches as they were before the block (a
//                 register-tiled fp32 mini-GEMM per bank); per candidate the best exact slot/score and the summary argmax go
//                 to a small global scratch.  Grid (2, B, Hkv), the heads of a state in one cluster, for 2..8 KV heads;
//                 (2, B) otherwise.
//   route_decide  grid (B): the order-dependent decisions (LRU victim ranking, novel-rank assignment,
//                 stamps, per-slot candidate lists) -> a small per-state plan in global scratch.
//   route_apply   values + cache re-normalisation of the written bank slots: a group of one, two or eight warps per slot, by
//                 the length of its rows; a CTA holds four, two or one group.
//   ring_rewrite  grid (2*Hkv, B): kept ring rows shift to the front, the block's tail is appended.
// Semantics: upstream memory_banks.py:438-564 (block write), 633-742 (exact), 853-932 (summary).
#include "coda_common.cuh"
#include "topk_warp.cuh"
#include "tma_utils.cuh"
#include "bank_score.cuh"
#include <mutex>

struct RouteParams {
  coda_layer_cfg c;
  coda_state_ptrs st;
  int fill, blk, n_ev, te, ts;          // ring occupancy before the block; evicted count; candidates used
  long long pos_first;                  // position of evicted token 0
  const void* kblk; long long kb_bs, kb_rs;
  const void* vblk; long long vb_bs, vb_rs;
  const float* gates; long long gates_bs, gate_ev0;
  const int* cand; long long cand_bs;
  const float* eta_logit;
  float* ex_best; int* ex_bi; int* su_idx;   // scratch: [B][Te], [B][Te], [B][Ts]
  int* plan;                                 // scratch: per-state plan (see Plan)
};

// Row of evicted token e (ring slot e when e < fill, else row e-fill of the block), head h.
template <typename T>
__device__ __forceinline__ const T* src_row(const RouteParams& p, const void* buf, const void* blkp,
                                            long long bbs, long long brs, int b, int e, int h) {
  const int Lbuf = p.c.W + p.c.Me + p.c.Ms, Dh = p.c.Dh;
  if (e < p.fill) return (const T*)buf + (((long long)b * p.c.Hkv + h) * Lbuf + e) * Dh;
  return (const T*)blkp + (long long)b * bbs + (long long)(e - p.fill) * brs + (long long)h * Dh;
}

// ---- scores: a register-tiled fp32 mini-GEMM per state and bank ----
// S[candidate][slot] = mean over heads of the dtype-rounded per-head dot products of the unit-norm candidate
// with the bank's unit-norm cache row; the kernel keeps only the row-wise first-index argmax (and, for the
// exact bank, the best score).  Grid (2, B): x = 0 exact bank (V rows, n = Dh), x = 1 summary bank (LF half of
// the K rows, n = Dh/2).  Tiles: RS_ROWS candidates x 64 slots x 64-element K chunks of one head, staged
// transposed ([k][row]) in shared memory as fp32; 256 threads, each TM x 4 outputs.
constexpr int RS_KC = 64;
constexpr int RS_COLS = 64;

template <typename T, int TM>
__device__ __forceinline__ void route_score_bank(const RouteParams& p, int b, bool exact, float* sm) {
  constexpr int ROWS = 16 * TM;
  const coda_layer_cfg& c = p.c;
  const int tid = threadIdx.x;
  const int Hkv = c.Hkv, Dh = c.Dh, lf = Dh / 2, W = c.W, Me = c.Me, Ms = c.Ms;
  const int n = exact ? Dh : Dh - lf, M = exact ? Me : Ms, Tn = exact ? p.te : p.ts;
  const int active = exact ? c.active_exact : c.active_summary;
  const T* cache = exact ? (const T*)p.st.exact_v_norm + (long long)b * Hkv * Me * Dh
                         : (const T*)p.st.sum_lf_k_norm + (long long)b * Hkv * Ms * n;
  const uint8_t* al = p.st.allowed + (long long)b * (W + Me + Ms);
  float* As = sm;                                  // [RS_KC][ROWS]
  float* Bs = As + RS_KC * ROWS;                   // [RS_KC][RS_COLS]
  float* Ss = Bs + RS_KC * RS_COLS;                // [ROWS][RS_COLS + 1]
  float* den = Ss + ROWS * (RS_COLS + 1);          // [ROWS][Hkv]
  int* cidx = reinterpret_cast<int*>(den + ROWS * Hkv);   // [ROWS]
  const int ty = tid >> 4, tx = tid & 15;          // 16 x 16 thread grid

  for (int r0 = 0; r0 < Tn; r0 += ROWS) {
    const int nrows = min(ROWS, Tn - r0);
    __syncthreads();
    for (int r = tid; r < ROWS; r += 256) cidx[r] = r < nrows ? p.cand[(long long)b * p.cand_bs + r0 + r] : -1;
    __syncthreads();
    // ||x|| of every (candidate, head) of the tile: one thread per pair, batched loads  (memory_banks.py:498-500)
    for (int it = tid; it < ROWS * Hkv; it += 256) {
      const int r = it / Hkv, h = it % Hkv;
      float ss = 0.f;
      if (cidx[r] >= 0) {
        const T* row = exact ? src_row<T>(p, p.st.v_buf, p.vblk, p.vb_bs, p.vb_rs, b, cidx[r], h)
                             : src_row<T>(p, p.st.k_buf, p.kblk, p.kb_bs, p.kb_rs, b, cidx[r], h) + lf;
        int d = 0;
        for (; d + 16 <= n; d += 16) {
          float x[16];
          load_run<T, 16>(row + d, x);
#pragma unroll
          for (int i = 0; i < 16; ++i) ss = fmaf(x[i], x[i], ss);
        }
        for (; d < n; ++d) { const float v = El<T>::ld(row + d); ss = fmaf(v, v, ss); }
      }
      den[it] = fmaxf(El<T>::rnd(sqrtf(ss)), 1e-6f);
    }
    float best = 0.f; int bi = 0;                  // running first-index argmax of row `tid` (tid < ROWS)
    for (int c0 = 0; c0 < M; c0 += RS_COLS) {
      float tot[TM][4];
#pragma unroll
      for (int i = 0; i < TM; ++i) { tot[i][0] = tot[i][1] = tot[i][2] = tot[i][3] = 0.f; }
      for (int h = 0; h < Hkv; ++h) {
        float acc[TM][4];
#pragma unroll
        for (int i = 0; i < TM; ++i) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f; }
        for (int k0 = 0; k0 < n; k0 += RS_KC) {
          __syncthreads();
          // stage: candidates (normalised, dtype-rounded) and cache rows, both transposed to [k][row];
          // every thread owns a run of KRUN consecutive k of one row and loads it in one batch
          {
            constexpr int KRUN_A = RS_KC * ROWS / 256;          // 16 (64-row tile) or 4 (16-row tile)
            const int r = tid % ROWS, kq0 = (tid / ROWS) * KRUN_A;
            float x[KRUN_A];
#pragma unroll
            for (int i = 0; i < KRUN_A; ++i) x[i] = 0.f;
            if (cidx[r] >= 0) {
              const T* row = exact ? src_row<T>(p, p.st.v_buf, p.vblk, p.vb_bs, p.vb_rs, b, cidx[r], h)
                                   : src_row<T>(p, p.st.k_buf, p.kblk, p.kb_bs, p.kb_rs, b, cidx[r], h) + lf;
              if (k0 + kq0 + KRUN_A <= n) load_run<T, KRUN_A>(row + k0 + kq0, x);
              else
                for (int i = 0; i < KRUN_A; ++i) if (k0 + kq0 + i < n) x[i] = El<T>::ld(row + k0 + kq0 + i);
              const float dn = den[r * Hkv + h];
              // (the division out of line: inlined, the reciprocal form made this loop 4 % slower, 98 -> 102 us for 16 states of 16 heads)
#pragma unroll
              for (int i = 0; i < KRUN_A; ++i) x[i] = El<T>::rnd(div_rn_call(x[i], dn));
            }
#pragma unroll
            for (int i = 0; i < KRUN_A; ++i) As[(kq0 + i) * ROWS + r] = x[i];
          }
          {
            constexpr int KRUN_B = RS_KC * RS_COLS / 256;       // 16
            const int col = tid % RS_COLS, kq0 = (tid / RS_COLS) * KRUN_B, m = c0 + col;
            float x[KRUN_B];
#pragma unroll
            for (int i = 0; i < KRUN_B; ++i) x[i] = 0.f;
            if (m < M) {
              const T* row = cache + ((long long)h * M + m) * n;
              if (k0 + kq0 + KRUN_B <= n) load_run<T, KRUN_B>(row + k0 + kq0, x);
              else
                for (int i = 0; i < KRUN_B; ++i) if (k0 + kq0 + i < n) x[i] = El<T>::ld(row + k0 + kq0 + i);
            }
#pragma unroll
            for (int i = 0; i < KRUN_B; ++i) Bs[(kq0 + i) * RS_COLS + col] = x[i];
          }
          __syncthreads();
#pragma unroll 8
          for (int kq = 0; kq < RS_KC; ++kq) {
            float a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kq * ROWS + ty * TM + i];
            const float4 bv = *reinterpret_cast<const float4*>(Bs + kq * RS_COLS + tx * 4);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
              acc[i][0] = fmaf(a[i], bv.x, acc[i][0]); acc[i][1] = fmaf(a[i], bv.y, acc[i][1]);
              acc[i][2] = fmaf(a[i], bv.z, acc[i][2]); acc[i][3] = fmaf(a[i], bv.w, acc[i][3]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) tot[i][jj] += El<T>::rnd(acc[i][jj]);
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const int m = c0 + tx * 4 + jj;
          float s = El<T>::rnd(tot[i][jj] / (float)Hkv);
          if (m >= M) s = -INFINITY;                                   // padding column: never wins
          else if (m >= active || (exact && !al[W + m])) s = -1e9f;    // (:646-650, :875-877)
          Ss[(ty * TM + i) * (RS_COLS + 1) + tx * 4 + jj] = s;
        }
      __syncthreads();
      if (tid < nrows) {
        for (int col = 0; col < RS_COLS && c0 + col < M; ++col) {
          const float s = Ss[tid * (RS_COLS + 1) + col];
          if ((c0 == 0 && col == 0) || s > best) { best = s; bi = c0 + col; }
        }
      }
    }
    if (tid < nrows) {
      if (exact) { p.ex_best[(long long)b * c.Te + r0 + tid] = best; p.ex_bi[(long long)b * c.Te + r0 + tid] = bi; }
      else p.su_idx[(long long)b * c.Ts + r0 + tid] = bi;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) route_score_kernel(RouteParams p) {
  extern __shared__ float sm[];
  grid_chain();
  const bool exact = blockIdx.x == 0;
  if (exact) { if (p.te > 0 && p.c.Me > 0) route_score_bank<T, 1>(p, blockIdx.y, true, sm); }
  else if (p.ts > 0 && p.c.Ms > 0) route_score_bank<T, 4>(p, blockIdx.y, false, sm);
}

// ---- the same scores with the KV heads side by side: one CTA per (bank, state, head), the heads of a state in one cluster ----
// route_score_bank walks the heads one after the other (2 x Hkv tile loads per output tile, each a memory round
// trip); here CTA h computes head h's rounded dot products only, leaves them in its shared memory, and after one
// cluster barrier every CTA finishes the output rows r with r % Hkv == h, a warp per row: it adds the Hkv partials in head
// order (the order route_score_bank adds them in, so the results are the same bits), takes the mean, applies the slot
// masks and keeps the running first-index argmax of its rows.
// Bound: issue slots of many small CTAs (staging, the rounded division per element, the products), so the tile
// follows the bank: ROWS candidates x COLS slots x KC elements with COLS = 32 where both banks have at most 32 slots,
// and KC = 32 where the phase-safe half of a key has at most 32 elements.
// Per block: 17 -> 12 us (64 states, 2 heads of 64, 64 slots a bank), 94 -> 54 us (512 states, 3 heads of 64, 32 slots),
// 25.5 -> 24 us (32 states, 8 heads of 128, 64 slots).
template <typename T, int ROWS, int COLS, int KC>
__device__ __forceinline__ void route_score_bank_heads(const RouteParams& p, int b, bool exact, float* sm) {
  constexpr int TX = COLS / 4, RG = 256 / TX;                 // threads along the columns (4 each) / row groups
  constexpr int TM = ROWS > RG ? ROWS / RG : 1;               // rows per thread; row groups beyond ROWS only stage
  const coda_layer_cfg& c = p.c;
  const int tid = threadIdx.x, h = blockIdx.z, lane = tid & 31, warp = tid >> 5;
  const int Hkv = c.Hkv, Dh = c.Dh, lf = Dh / 2, W = c.W, Me = c.Me, Ms = c.Ms;
  const int n = exact ? Dh : Dh - lf, M = exact ? Me : Ms, Tn = exact ? p.te : p.ts;
  const int active = exact ? c.active_exact : c.active_summary;
  const T* cache = exact ? (const T*)p.st.exact_v_norm + (long long)b * Hkv * Me * Dh
                         : (const T*)p.st.sum_lf_k_norm + (long long)b * Hkv * Ms * n;
  const uint8_t* al = p.st.allowed + (long long)b * (W + Me + Ms);
  float* As = sm;                                  // [KC][ROWS]
  float* Bs = As + KC * ROWS;                      // [KC][COLS]
  float* Ps = Bs + KC * COLS;                      // [ROWS][COLS]   this head's rounded dots (read by the whole cluster)
  float* den = Ps + ROWS * COLS;                   // [ROWS]
  float* rbest = den + ROWS;                       // [ROWS] running best score and slot of the rows this CTA owns
  int* rbi = reinterpret_cast<int*>(rbest + ROWS);
  int* cidx = rbi + ROWS;                          // [ROWS]
  const int ty = tid / TX, tx = tid % TX;
  const bool one_chunk = n <= KC;

  for (int r0 = 0; r0 < Tn; r0 += ROWS) {
    const int nrows = min(ROWS, Tn - r0);
    __syncthreads();
    for (int r = tid; r < ROWS; r += 256) cidx[r] = r < nrows ? p.cand[(long long)b * p.cand_bs + r0 + r] : -1;
    __syncthreads();
    auto row_at = [&](int r) {
      return exact ? src_row<T>(p, p.st.v_buf, p.vblk, p.vb_bs, p.vb_rs, b, cidx[r], h)
                   : src_row<T>(p, p.st.k_buf, p.kblk, p.kb_bs, p.kb_rs, b, cidx[r], h) + lf;
    };
    // ||x|| of every candidate of the tile for this head (memory_banks.py:498-500): the fp32 sum of squares runs over the
    // elements in order, one thread per row, as route_score_bank's does.  Rows that one chunk holds are summed from
    // shared memory below instead.
    if (!one_chunk && tid < ROWS) {
      float ss = 0.f;
      if (cidx[tid] >= 0) {
        const T* row = row_at(tid);
        int d = 0;
        for (; d + 16 <= n; d += 16) {
          float x[16];
          load_run<T, 16>(row + d, x);
#pragma unroll
          for (int i = 0; i < 16; ++i) ss = fmaf(x[i], x[i], ss);
        }
        for (; d < n; ++d) { const float v = El<T>::ld(row + d); ss = fmaf(v, v, ss); }
      }
      den[tid] = fmaxf(El<T>::rnd(sqrtf(ss)), 1e-6f);
    }
    for (int c0 = 0; c0 < M; c0 += COLS) {
      float acc[TM][4];
#pragma unroll
      for (int i = 0; i < TM; ++i) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f; }
      for (int k0 = 0; k0 < n; k0 += KC) {
        __syncthreads();
        // stage: candidates (normalised, dtype-rounded) and cache rows, both transposed to [k][row]; every thread owns a
        // run of consecutive k of one row of each and loads it in one batch
        constexpr int KRUN_A = KC * ROWS / 256, KRUN_B = KC * COLS / 256;
        const int ar = tid % ROWS, ak = (tid / ROWS) * KRUN_A, bc = tid % COLS, bk = (tid / COLS) * KRUN_B;
        float xa[KRUN_A], xb[KRUN_B];
#pragma unroll
        for (int i = 0; i < KRUN_B; ++i) xb[i] = 0.f;
        if (c0 + bc < M) {
          const T* row = cache + ((long long)h * M + c0 + bc) * n + k0 + bk;
          if (k0 + bk + KRUN_B <= n) load_run<T, KRUN_B>(row, xb);
          else
            for (int i = 0; i < KRUN_B; ++i) if (k0 + bk + i < n) xb[i] = El<T>::ld(row + i);
        }
#pragma unroll
        for (int i = 0; i < KRUN_A; ++i) xa[i] = 0.f;
        const bool have = cidx[ar] >= 0;
        if (have) {
          const T* row = row_at(ar) + k0 + ak;
          if (k0 + ak + KRUN_A <= n) load_run<T, KRUN_A>(row, xa);
          else
            for (int i = 0; i < KRUN_A; ++i) if (k0 + ak + i < n) xa[i] = El<T>::ld(row + i);
        }
#pragma unroll
        for (int i = 0; i < KRUN_B; ++i) Bs[(bk + i) * COLS + bc] = xb[i];
        if (one_chunk && c0 == 0) {
#pragma unroll
          for (int i = 0; i < KRUN_A; ++i) As[(ak + i) * ROWS + ar] = xa[i];
          __syncthreads();
          if (tid < ROWS) {
            float ss = 0.f;
#pragma unroll 8
            for (int d = 0; d < n; ++d) { const float v = As[d * ROWS + tid]; ss = fmaf(v, v, ss); }
            den[tid] = fmaxf(El<T>::rnd(sqrtf(ss)), 1e-6f);
          }
          __syncthreads();
        }
        if (have) {
          const float dn = den[ar];
#pragma unroll
          for (int i = 0; i < KRUN_A; ++i) xa[i] = t_div<T>(xa[i], dn);
        }
#pragma unroll
        for (int i = 0; i < KRUN_A; ++i) As[(ak + i) * ROWS + ar] = xa[i];
        __syncthreads();
        if (ty < ROWS / TM) {
          const int kend = min(KC, n - k0);
#pragma unroll 8
          for (int kq = 0; kq < kend; ++kq) {
            float a[TM];
            const float* ap = As + kq * ROWS + ty * TM;
            if constexpr (TM == 4) { const float4 v = *reinterpret_cast<const float4*>(ap); a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w; }
            else if constexpr (TM == 2) { const float2 v = *reinterpret_cast<const float2*>(ap); a[0] = v.x; a[1] = v.y; }
            else a[0] = ap[0];
            const float4 bv = *reinterpret_cast<const float4*>(Bs + kq * COLS + tx * 4);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
              acc[i][0] = fmaf(a[i], bv.x, acc[i][0]); acc[i][1] = fmaf(a[i], bv.y, acc[i][1]);
              acc[i][2] = fmaf(a[i], bv.z, acc[i][2]); acc[i][3] = fmaf(a[i], bv.w, acc[i][3]);
            }
          }
        }
      }
      // every CTA of the cluster has read the previous tile's partials before they are overwritten
      __syncwarp();
      if (r0 > 0 || c0 > 0) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      if (ty < ROWS / TM) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
          *reinterpret_cast<float4*>(Ps + (ty * TM + i) * COLS + tx * 4) =
              make_float4(El<T>::rnd(acc[i][0]), El<T>::rnd(acc[i][1]), El<T>::rnd(acc[i][2]), El<T>::rnd(acc[i][3]));
      }
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      // rows r = h, h + Hkv, ... of the tile are finished here, a warp per row: partials of all heads, in head order
      for (int r = h + warp * Hkv; r < nrows; r += 8 * Hkv) {
        float best = -INFINITY, first = 0.f;
        int bi = 0x7fffffff;
#pragma unroll
        for (int cc = 0; cc < COLS / 32; ++cc) {
          const int col = lane + 32 * cc, m = c0 + col;
          const uint32_t local = tma::smem_u32(Ps + r * COLS + col);
          float pv[8];                                 // all requests first, then the sum in head order
#pragma unroll
          for (int hh = 0; hh < 8; ++hh) {
            pv[hh] = 0.f;
            if (hh < Hkv) {
              uint32_t remote;
              asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(hh));
              asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(pv[hh]) : "r"(remote) : "memory");
            }
          }
          float tot = 0.f;
#pragma unroll
          for (int hh = 0; hh < 8; ++hh) if (hh < Hkv) tot += pv[hh];
          if (m < M) {
            float sc = El<T>::rnd(tot / (float)Hkv);
            if (m >= active || (exact && !al[W + m])) sc = -1e9f;         // (:646-650, :875-877)
            if (cc == 0) first = sc;
            if (sc > best || bi == 0x7fffffff) { best = sc != sc ? -INFINITY : sc; bi = m; }
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        // a score that is not a number wins only from the very first slot, where the running maximum starts
        if (lane == 0) {
          if (c0 == 0) { const bool nan0 = first != first; rbest[r] = nan0 ? first : best; rbi[r] = nan0 ? 0 : bi; }
          else if (best > rbest[r]) { rbest[r] = best; rbi[r] = bi; }
        }
      }
    }
    __syncwarp();
    if (lane == 0) {
      for (int r = h + warp * Hkv; r < nrows; r += 8 * Hkv) {
        if (exact) { p.ex_best[(long long)b * c.Te + r0 + r] = rbest[r]; p.ex_bi[(long long)b * c.Te + r0 + r] = rbi[r]; }
        else p.su_idx[(long long)b * c.Ts + r0 + r] = rbi[r];
      }
    }
  }
  // no CTA may leave while another still reads its partials
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int COLS, int KCS>
constexpr size_t route_score_heads_floats() {
  const size_t e = (size_t)RS_KC * 16 + RS_KC * COLS + 16 * COLS + 4 * 16, s = (size_t)KCS * 64 + KCS * COLS + 64 * COLS + 4 * 64;
  return e > s ? e : s;
}

template <typename T, int COLS, int KCS>
__global__ void __launch_bounds__(256, 4) route_score_heads_kernel(RouteParams p) {
  extern __shared__ __align__(16) float sm[];
  grid_chain();
  const bool exact = blockIdx.x == 0;
  // (both branches are uniform over a cluster: its CTAs differ in blockIdx.z only)
  if (exact) { if (p.te > 0 && p.c.Me > 0) route_score_bank_heads<T, 16, COLS, RS_KC>(p, blockIdx.y, true, sm); }
  else if (p.ts > 0 && p.c.Ms > 0) route_score_bank_heads<T, 64, COLS, KCS>(p, blockIdx.y, false, sm);
}

template <typename T, int COLS, int KCS>
static cudaError_t launch_score_heads(const RouteParams& p, cudaStream_t s) {
  const size_t smem = sizeof(float) * route_score_heads_floats<COLS, KCS>();
  if (smem > 48 * 1024) cudaFuncSetAttribute(route_score_heads_kernel<T, COLS, KCS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return coda_launch_chained(route_score_heads_kernel<T, COLS, KCS>, dim3(2, p.c.B, p.c.Hkv), dim3(256), smem, s, p.c.Hkv, p);
}

// Per-state plan written by route_decide and consumed by route_apply (all int32 / fp32, in global scratch).
struct Plan {
  int* e_tgt; int* e_flag;            // [Te]  target slot; bit0 overwrite, bit1 touch, bit2 first overwriter of its slot
  float* s_w; int* s_ord;             // [Ts]  summary weights and evicted indices, grouped by slot in candidate order
  int* s_start; float* s_cnt; int* s_was;   // [Ms+1], [Ms], [Ms]
};
__device__ __forceinline__ Plan plan_of(const RouteParams& p, int b) {
  const int Te = p.c.Te > 0 ? p.c.Te : 0, Ts = p.c.Ts > 0 ? p.c.Ts : 0, Ms = p.c.Ms;
  const size_t per = (size_t)(2 * Te + 2 * Ts + 3 * Ms + 1);
  int* base = p.plan + (size_t)b * per;
  Plan pl;
  pl.e_tgt = base; pl.e_flag = base + Te;
  pl.s_w = reinterpret_cast<float*>(base + 2 * Te); pl.s_ord = base + 2 * Te + Ts;
  pl.s_start = base + 2 * Te + 2 * Ts; pl.s_cnt = reinterpret_cast<float*>(pl.s_start + Ms + 1);
  pl.s_was = pl.s_start + Ms + 1 + Ms;
  return pl;
}

// ---- decisions: the order-dependent part, one small CTA per state ----
// Warp 0 decides for the exact bank, the other warps keep the summary bank's books.  What looks serial is a prefix
// count or a per-slot extremum: the rank of a novel candidate is the number of novel kept candidates up to it, the
// first overwriter of a slot is the smallest candidate index and its stamp the largest position among those that
// touch it (shared-memory min / max: independent of the order).  Only a slot's weight sum is rounded after each term; a
// thread per slot walks the candidates for it.
// Bound: latency of one short CTA per state; one thread walking these loops in shared memory took
// 23 us per block for 64 states (256-token blocks, 8 + 64 candidates), this 9 us.
constexpr int RD_THREADS = 160;

template <typename T>
__global__ void __launch_bounds__(RD_THREADS) route_decide_kernel(RouteParams p) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const coda_layer_cfg& c = p.c;
  const int b = blockIdx.x, tid = threadIdx.x, NT = blockDim.x, lane = tid & 31;
  const int Me = c.Me, Ms = c.Ms, W = c.W, Lbuf = W + Me + Ms;
  const int te = (Me > 0) ? p.te : 0, ts = (Ms > 0) ? p.ts : 0, tmax = te > ts ? te : ts;
  typedef topk_order::Item<long long> It64;
  It64* lruq = reinterpret_cast<It64*>(smraw);                       // [Me]
  float* c_g = reinterpret_cast<float*>(lruq + (Me > 0 ? Me : 1));   // [tmax] gates
  float* x_best = c_g + (tmax > 0 ? tmax : 1);                       // [te]
  float* w_s = x_best + (te > 0 ? te : 1);                           // [ts] summary weights
  int* c_e = reinterpret_cast<int*>(w_s + (ts > 0 ? ts : 1));        // [tmax] evicted index
  int* x_bi = c_e + (tmax > 0 ? tmax : 1);                           // [te]
  int* s_idx = x_bi + (te > 0 ? te : 1);                             // [ts]
  int* n_first = s_idx + (ts > 0 ? ts : 1);                          // [Me] first overwriting candidate of a slot
  int* n_e = n_first + (Me > 0 ? Me : 1);                            // [Me] largest touching evicted index, -1: none
  int* start_s = n_e + (Me > 0 ? Me : 1);                            // [Ms+1]
  uint16_t* qscr = reinterpret_cast<uint16_t*>(start_s + Ms + 1);    // [2*Me] partition scratch
  unsigned char* s_used = reinterpret_cast<unsigned char*>(qscr + 2 * (Me > 0 ? Me : 1));   // [Me + Ms]
  const uint8_t* al = p.st.allowed + (long long)b * Lbuf;
  long long* last = (long long*)p.st.mem_last_exact + (long long)b * Me;
  Plan pl = plan_of(p, b);
  const int Ae = c.active_exact;
  // All but the scores was there before the scoring kernel passed its own wait (it lets this one come only then) and is not
  // written by it: candidates, gates, flags and stamps are read (through L2), and the victims ranked, while it still runs.
  for (int t = tid; t < tmax; t += NT) {
    const int e = __ldcg(p.cand + (long long)b * p.cand_bs + t);
    c_e[t] = e;
    c_g[t] = __ldcg(p.gates + (long long)b * p.gates_bs + p.gate_ev0 + e);
  }
  for (int m = tid; m < Ms; m += NT) s_used[Me + m] = __ldcg(al + W + Me + m);
  int used_here = 0;
  for (int m = tid; m < Me; m += NT) {
    const bool used = __ldcg(al + W + m) != 0;
    const long long stamp = __ldcg(last + m);
    s_used[m] = used;
    lruq[m].v = (used && m < Ae) ? stamp : -(1LL << 62);
    lruq[m].i = m;
    n_first[m] = 0x7fffffff; n_e[m] = -1;
    used_here |= used ? 1 : 0;
  }
  const bool any_used = __syncthreads_or(used_here) != 0;
  const int n_lru = te < Ae ? te : Ae;
  if (tid < 32 && te > 0) topk_order::topk_queue_warp<long long, false>(lruq, Me, n_lru, true, qscr);   // victims = lruq[0..n_lru).i
  grid_chain();
  for (int t = tid; t < te; t += NT) { x_best[t] = p.ex_best[(long long)b * c.Te + t]; x_bi[t] = p.ex_bi[(long long)b * c.Te + t]; }
  for (int t = tid; t < ts; t += NT) s_idx[t] = p.su_idx[(long long)b * c.Ts + t];
  // routing-event record of this call (optional): cleared here, filled by the deciding warps below
  int32_t* evw = p.st.events != nullptr ? p.st.events + (long long)b * CODA_EVENT_WORDS : nullptr;
  if (evw != nullptr && tid < CODA_EVENT_WORDS) evw[tid] = 0;
  __syncthreads();
  if (tid < 32) {
    if (te > 0) {
      // ---- exact bank (memory_banks.py:635-697) ----
      const float tn = El<T>::rnd(c.tau_novel), tm = El<T>::rnd(c.tau_match);
      int ranked = 0, n_gated = 0, n_hit = 0, n_ins = 0, n_ow = 0, n_frus = 0;
      for (int t0 = 0; t0 < te; t0 += 32) {
        const int t = t0 + lane;
        const bool in = t < te;
        const float best = in ? x_best[t] : 0.f;
        const bool keep = in && (c.gated ? (c_g[t] >= c.tau_gate_exact) : true);
        const bool novel = !any_used || best < tn;
        const bool hit = any_used && best >= tm;
        const bool nk = novel && keep;
        const unsigned nkb = __ballot_sync(0xffffffffu, nk);
        const int rank = ranked + __popc(nkb & (0xffffffffu >> (31 - lane))) - 1;
        ranked += __popc(nkb);
        const bool capped = nk && rank < Ae;
        int r = rank < 0 ? 0 : rank;
        if (r > n_lru - 1) r = n_lru - 1 > 0 ? n_lru - 1 : 0;
        const int tgt = capped ? lruq[r].i : (in ? x_bi[t] : 0);
        const bool touch = keep && (!novel || capped);
        const bool ow = c.refresh_on_hit ? (keep && (capped || hit)) : capped;
        if (ow) atomicMin(&n_first[tgt], t);
        if (touch) atomicMax(&n_e[tgt], c_e[t]);
        __syncwarp();
        // (an earlier chunk's candidates are in already, a later one's are larger: the minimum is final for this chunk)
        if (in) { pl.e_tgt[t] = tgt; pl.e_flag[t] = (ow ? 1 : 0) | (touch ? 2 : 0) | (ow && n_first[tgt] == t ? 4 : 0); }
        if (evw != nullptr) {
          n_gated += __popc(__ballot_sync(0xffffffffu, in && c.gated && !keep)); n_hit += __popc(__ballot_sync(0xffffffffu, hit && keep));
          n_ins += __popc(__ballot_sync(0xffffffffu, capped)); n_ow += __popc(__ballot_sync(0xffffffffu, ow));
          n_frus += __popc(__ballot_sync(0xffffffffu, nk && !capped));
        }
      }
      if (evw != nullptr && lane == 0) { evw[0] = n_gated; evw[1] = n_hit; evw[2] = n_ins; evw[3] = n_ow; evw[4] = n_frus; }
      __syncwarp();
      // stamps: per slot the largest position among touching candidates replaces the old stamp (:682-697)
      for (int m = lane; m < Me; m += 32) {
        if (n_e[m] >= 0) last[m] = p.pos_first + n_e[m];
      }
    }
    return;
  }
  if (ts <= 0) return;
  // ---- summary bank bookkeeping (memory_banks.py:880-885, 906): weights, per-slot candidate lists ----
  constexpr int NS = RD_THREADS - 32;
  const int sid = tid - 32;
  auto sync_s = [] { asm volatile("bar.sync 1, %0;" ::"n"(NS) : "memory"); };
  for (int t = sid; t < ts; t += NS) {
    float w = El<T>::rnd(c_g[t]);
    if (c.gated && !(c_g[t] >= c.tau_gate_summary)) w = 0.f;             // (:518-523)
    w_s[t] = w;
  }
  sync_s();
  for (int m = sid; m < Ms; m += NS) {
    float cnt = 0.f;
    int n = 0;
#pragma unroll 4
    for (int t = 0; t < ts; ++t)
      if (s_idx[t] == m) { cnt = t_add<T>(cnt, w_s[t]); ++n; }
    pl.s_cnt[m] = cnt;
    pl.s_was[m] = s_used[Me + m] != 0;
    start_s[m + 1] = n;
    s_used[Me + m] = (s_used[Me + m] != 0 ? 1 : 0) | (cnt > 0.f ? 2 : 0);    // for the event record
  }
  if (sid == 0) start_s[0] = 0;
  sync_s();
  if (tid < 64) {                                                        // inclusive prefix sum over the slots
    int carry = 0;
    for (int m0 = 1; m0 <= Ms; m0 += 32) {
      int v = m0 + lane <= Ms ? start_s[m0 + lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
      v += carry;
      if (m0 + lane <= Ms) start_s[m0 + lane] = v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
  } else if (tid < 96 && evw != nullptr) {
    const int As = c.active_summary;
    int n_upd = 0, n_new = 0; bool all_used = true, incoming = false;
    for (int m = lane; m < Ms; m += 32) {
      const bool got = (s_used[Me + m] & 2) != 0, was = (s_used[Me + m] & 1) != 0;
      n_upd += got ? 1 : 0; n_new += (got && !was) ? 1 : 0;
      if (m < As) { all_used = all_used && (was || got); incoming = incoming || got; }
    }
    n_upd = __reduce_add_sync(0xffffffffu, n_upd); n_new = __reduce_add_sync(0xffffffffu, n_new);
    all_used = __all_sync(0xffffffffu, all_used); incoming = __any_sync(0xffffffffu, incoming);
    if (lane == 0) { evw[5] = n_upd; evw[6] = n_new; evw[7] = all_used ? 1 : 0; evw[8] = incoming ? 1 : 0; }
  }
  sync_s();
  for (int m = sid; m <= Ms; m += NS) pl.s_start[m] = start_s[m];
  for (int m = sid; m < Ms; m += NS) {                                   // stable grouping by slot
    int a = start_s[m];
    if (start_s[m + 1] == a) continue;
#pragma unroll 4
    for (int t = 0; t < ts; ++t)
      if (s_idx[t] == m) { pl.s_ord[a] = c_e[t]; pl.s_w[a] = w_s[t]; ++a; }
  }
}

// ---- slot writes ----
// One group of WPS warps per written slot (exact: per overwriting candidate group; summary: per slot).  The slot's K
// and V rows are cut into 8-element chunks, each owned by one thread, which reads the old values and the candidates'
// rows (NB candidates in flight) and adds them in list order.  The candidate list is read 32 at a time by the lanes of
// every warp and handed round by shuffles.
// In bf16 the sums are packed: one instruction per element pair for the weighted row and one for the sum, each result the
// rounding of the exact value, which is what the reference's op-by-op bf16 arithmetic gives.
// A group has a thread for each chunk of rows of up to 1024 elements over all heads (one warp up to 128 elements, two up
// to 256, else eight; larger rows loop), so that old rows and candidates are one round trip.  A CTA per slot of a narrow
// layer left three threads in four idle and the chip waiting on CTA launches.
// Per block: 40 -> 12.5 us (64 states, 2 x 64 elements a row), 233 -> 91 us (512 states, 3 x 64), 31 -> 22 us (32 states, 8 x 128).
template <typename T, int WPS, bool PACKED>
__global__ void __launch_bounds__(WPS == 8 ? 256 : 128, WPS == 8 ? 4 : WPS == 1 ? 8 : 6) route_apply_kernel(RouteParams p, int nslots) {
  extern __shared__ float stash_all[];                               // [groups of the CTA][Hkv*Dh] new rows for re-normalising
  const coda_layer_cfg& c = p.c;
  constexpr int GT = 32 * WPS, GROUPS = (WPS == 8 ? 256 : 128) / GT; // threads of a slot's group, groups per CTA
  const int b = blockIdx.y, lane = threadIdx.x & 31, gid = threadIdx.x / GT, tid = threadIdx.x % GT;
  const int job = blockIdx.x * GROUPS + gid;
  grid_chain();
  if (job >= nslots) return;
  const int Hkv = c.Hkv, Dh = c.Dh, HD = Hkv * Dh, lf = Dh / 2, lfd = Dh - lf;
  float* stash = stash_all + gid * HD;
  const int Me = c.Me, Ms = c.Ms, W = c.W, Lbuf = W + Me + Ms;
  const int te = (Me > 0) ? p.te : 0;
  const Plan pl = plan_of(p, b);
  const bool exact = job < te;
  int slot, first, last;                                             // slot of its bank; range of the list scanned for it
  float cden = 1.f; bool fresh = false;
  if (exact) {
    // ---- exact bank write (memory_banks.py:707-742): candidates that overwrite this slot, in list order ----
    if ((pl.e_flag[job] & 5) != 5) return;                           // not the first overwriter of its slot
    slot = pl.e_tgt[job];
    first = job; last = te;
  } else {
    // ---- summary bank EMA of one slot (memory_banks.py:887-932) ----
    slot = job - te;
    const float cnt = pl.s_cnt[slot];
    if (!(cnt > 0.f)) return;
    first = pl.s_start[slot]; last = pl.s_start[slot + 1];
    cden = fmaxf(cnt, El<T>::rnd(1e-6f));
    fresh = c.overwrite_on_insert && !pl.s_was[slot];
  }
  // candidates a0 + 0..31 of the list in the lanes: a mask of those that count, their rows and weights
  auto list_at = [&](int a0, int& ce, float& w) {
    const int a = a0 + lane;
    bool on = a < last;
    ce = 0; w = 1.f;
    if (on) {
      if (exact) { on = (pl.e_flag[a] & 1) && pl.e_tgt[a] == slot; ce = p.cand[(long long)b * p.cand_bs + a]; }
      else { ce = pl.s_ord[a]; w = pl.s_w[a]; }
    }
    return __ballot_sync(0xffffffffu, on);
  };
  const int gslot = W + (exact ? 0 : Me) + slot;
  T* const kbuf = (T*)p.st.k_buf + (long long)b * Hkv * Lbuf * Dh;
  T* const vbuf = (T*)p.st.v_buf + (long long)b * Hkv * Lbuf * Dh;
  constexpr int R = 8;
  const bool runs = PACKED || (Dh % R) == 0;
  const int nch = (HD + R - 1) / R;                                  // chunks of the K row, then as many of the V row
  for (int x0 = 0; x0 < 2 * nch; x0 += GT) {
    const int x = x0 + tid;
    const bool isv = x >= nch;
    const int e0 = (isv ? x - nch : x) * R, h = e0 / Dh, d0 = e0 % Dh;
    // a chunk below the phase-safe half of a summary key is left alone
    const bool live = x < 2 * nch && !(runs && !exact && !isv && d0 + R <= lf);
    T* const buf = isv ? vbuf : kbuf;
    const void* sblk = isv ? p.vblk : p.kblk;
    const void* sbuf = isv ? p.st.v_buf : p.st.k_buf;
    const long long sbs = isv ? p.vb_bs : p.kb_bs, srs = isv ? p.vb_rs : p.kb_rs;
    auto at = [&](int e) { return buf + ((long long)(e / Dh) * Lbuf + gslot) * Dh + e % Dh; };
    float old[R], acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) { old[i] = 0.f; acc[i] = 0.f; }
    uint32_t oldw[R / 2], accw[R / 2];                               // (bf16 runs: the same, two elements a word)
    if (PACKED && live) {
      const uint4 t = *reinterpret_cast<const uint4*>(buf + ((long long)h * Lbuf + gslot) * Dh + d0);
      oldw[0] = t.x; oldw[1] = t.y; oldw[2] = t.z; oldw[3] = t.w;
      accw[0] = accw[1] = accw[2] = accw[3] = 0u;
#pragma unroll
      for (int i = 0; i < R / 2; ++i) { old[2 * i] = __uint_as_float(oldw[i] << 16); old[2 * i + 1] = __uint_as_float(oldw[i] & 0xffff0000u); }
    } else if (live) {
      if (runs) load_run<T, R>(buf + ((long long)h * Lbuf + gslot) * Dh + d0, old);
      else for (int i = 0; i < R; ++i) if (e0 + i < HD) old[i] = El<T>::ld(at(e0 + i));
    }
    auto row_of = [&](int ce, float (&y)[R]) {
      if (runs) { load_run<T, R>(src_row<T>(p, sbuf, sblk, sbs, srs, b, ce, h) + d0, y); return; }
      for (int i = 0; i < R; ++i)
        y[i] = e0 + i < HD ? El<T>::ld(src_row<T>(p, sbuf, sblk, sbs, srs, b, ce, (e0 + i) / Dh) + (e0 + i) % Dh) : 0.f;
    };
    for (int a0 = first; a0 < last; a0 += 32) {
      int lce; float lw;
      unsigned on = list_at(a0, lce, lw);
      while (on != 0u) {
        constexpr int NB = 4;
        if constexpr (PACKED) {
          uint4 y[NB];
          uint32_t w2[NB];
          bool have[NB];
#pragma unroll
          for (int q = 0; q < NB; ++q) {
            have[q] = on != 0u;
            const int src = have[q] ? __ffs(on) - 1 : 0;
            on &= on - 1u;
            const int ce = __shfl_sync(0xffffffffu, lce, src);
            w2[q] = __float_as_uint(__shfl_sync(0xffffffffu, lw, src));      // a bf16 value: its word's upper half
            w2[q] |= w2[q] >> 16;
            if (have[q] && live) y[q] = *reinterpret_cast<const uint4*>(src_row<T>(p, sbuf, sblk, sbs, srs, b, ce, h) + d0);
          }
#pragma unroll
          for (int q = 0; q < NB; ++q) {
            if (!have[q] || !live) continue;
            const uint32_t yw[4] = {y[q].x, y[q].y, y[q].z, y[q].w};
#pragma unroll
            for (int i = 0; i < R / 2; ++i)
              accw[i] = badd2(accw[i], exact ? badd2(yw[i], bneg2(oldw[i])) : bmul2(yw[i], w2[q]));
          }
        } else {
          // one candidate at a time: single precision, unaligned rows, head sizes that are no multiple of a chunk
          const int src = __ffs(on) - 1;
          on &= on - 1u;
          const int ce = __shfl_sync(0xffffffffu, lce, src);
          const float w = __shfl_sync(0xffffffffu, lw, src);
          if (live) {
            float y[R];
            row_of(ce, y);
#pragma unroll
            for (int i = 0; i < R; ++i) {
              if (exact) acc[i] = t_add<T>(acc[i], t_sub<T>(y[i], old[i]));
              else acc[i] = t_add<T>(acc[i], t_mul<T>(y[i], w));
            }
          }
        }
      }
    }
    if (!live) continue;
    if constexpr (PACKED) {
#pragma unroll
      for (int i = 0; i < R / 2; ++i) { acc[2 * i] = __uint_as_float(accw[i] << 16); acc[2 * i + 1] = __uint_as_float(accw[i] & 0xffff0000u); }
    }
    // the slot's EMA rate depends on the head only: one sigmoid per run, not one per element
    const float eta_run = (exact || fresh) ? 1.f : t_sigmoid<T>(p.eta_logit[h]);
    float nv[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int e = e0 + i;
      nv[i] = old[i];
      if (e >= HD) continue;
      const int hh = runs ? h : e / Dh, dd = runs ? d0 + i : e % Dh;
      if (exact) {                                                     // mem + sum of deltas
        nv[i] = t_add<T>(old[i], acc[i]);
        if (isv) stash[e] = nv[i];
      } else {                                                         // phase-safe EMA
        const float eta = fresh ? 1.f : (runs ? eta_run : t_sigmoid<T>(p.eta_logit[hh]));
        if (isv) nv[i] = t_add<T>(old[i], t_mul<T>(eta, t_sub<T>(t_div<T>(acc[i], cden), old[i])));
        else if (dd >= lf) {
          const float inc = El<T>::rnd(__fmul_rn(t_div<T>(acc[i], cden), c.energy_scale));
          nv[i] = t_add<T>(old[i], t_mul<T>(eta, t_sub<T>(inc, old[i])));
          stash[hh * lfd + dd - lf] = nv[i];
        }
      }
    }
    if (runs) store_run<T, R>(buf + ((long long)h * Lbuf + gslot) * Dh + d0, nv);
    else
      for (int i = 0; i < R; ++i)
        if (e0 + i < HD) El<T>::st(at(e0 + i), nv[i]);
  }
  if (tid == 0) p.st.allowed[(long long)b * Lbuf + gslot] = 1;
  if constexpr (WPS == 1) __syncwarp();
  else if constexpr (WPS == 8) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + gid), "n"(GT) : "memory");     // (a group may have left)
  const int nn_norm = exact ? Dh : lfd;
  T* cachep = exact ? (T*)p.st.exact_v_norm + (long long)b * Hkv * Me * Dh : (T*)p.st.sum_lf_k_norm + (long long)b * Hkv * Ms * lfd;
  const int Mb = exact ? Me : Ms;
  for (int h = tid >> 5; h < Hkv; h += WPS) {
    float ss = 0.f;
    for (int d = lane; d < nn_norm; d += 32) { const float v = stash[h * nn_norm + d]; ss += v * v; }
    const float den = fmaxf(El<T>::rnd(sqrtf(warp_sum(ss))), 1e-6f);
    for (int d = lane; d < nn_norm; d += 32)
      El<T>::st(cachep + ((long long)h * Mb + slot) * nn_norm + d, t_div<T>(stash[h * nn_norm + d], den));
  }
}

// Ring rewrite (memory_banks.py:152-177, 554-563): with the ring in chronological order the kept rows
// [drop, fill) move down to [0, fill-drop) and block rows [bstart, blk) follow them.  One CTA per
// (plane, K|V); 16-byte vectors when rows allow it; the in-place shift goes chunk by chunk in ascending order.
template <typename T, typename V>
__device__ __forceinline__ void ring_plane(T* ring, const T* src, long long src_rs, int Dh, int drop, int kept,
                                           int bstart, int nnew, int tid, int NT) {
  constexpr int PER = 4;
  constexpr int EV = sizeof(V) / sizeof(T);
  const int rowv = Dh / EV;                                            // vectors per row
  V* rv = reinterpret_cast<V*>(ring);
  if (drop > 0 && kept > 0) {
    const long long n = (long long)kept * rowv, off = (long long)drop * rowv;
    for (long long c0 = 0; c0 < n; c0 += (long long)NT * PER) {
      V tmp[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) { const long long x = c0 + (long long)i * NT + tid; if (x < n) tmp[i] = rv[off + x]; }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < PER; ++i) { const long long x = c0 + (long long)i * NT + tid; if (x < n) rv[x] = tmp[i]; }
      __syncthreads();
    }
  }
  for (long long x = tid; x < (long long)nnew * rowv; x += NT) {
    const int r = (int)(x / rowv), dv = (int)(x % rowv);
    rv[(long long)(kept + r) * rowv + dv] = *reinterpret_cast<const V*>(src + (long long)(bstart + r) * src_rs + (long long)dv * EV);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) ring_rewrite_kernel(RouteParams p, int vec16) {
  const coda_layer_cfg& c = p.c;
  const int h = blockIdx.x >> 1, pass = blockIdx.x & 1, b = blockIdx.y, tid = threadIdx.x, NT = blockDim.x;
  const int W = c.W, Dh = c.Dh, Lbuf = W + c.Me + c.Ms;
  const int drop = p.n_ev < p.fill ? p.n_ev : p.fill;
  const int kept = p.fill - drop;
  const int bstart = p.n_ev > p.fill ? p.n_ev - p.fill : 0;
  const int nnew = p.blk - bstart;
  T* ring = (T*)(pass ? p.st.v_buf : p.st.k_buf) + ((long long)b * c.Hkv + h) * Lbuf * Dh;
  const T* src = (const T*)(pass ? p.vblk : p.kblk) + (long long)b * (pass ? p.vb_bs : p.kb_bs) + (long long)h * Dh;
  const long long rs = pass ? p.vb_rs : p.kb_rs;
  grid_chain();
  if (vec16) ring_plane<T, uint4>(ring, src, rs, Dh, drop, kept, bstart, nnew, tid, NT);
  else ring_plane<T, T>(ring, src, rs, Dh, drop, kept, bstart, nnew, tid, NT);
  if (blockIdx.x == 0) {
    float* gr = p.st.g_recent + (long long)b * W;
    uint8_t* al = p.st.allowed + (long long)b * Lbuf;
    if (drop > 0 && kept > 0) {
      for (int c0 = 0; c0 < kept; c0 += NT) {
        const int x = c0 + tid;
        float tmp = 0.f;
        if (x < kept) tmp = gr[drop + x];
        __syncthreads();
        if (x < kept) gr[x] = tmp;
        __syncthreads();
      }
    }
    const float* gsrc = p.gates + (long long)b * p.gates_bs + p.gate_ev0 + p.fill + bstart;
    for (int x = tid; x < nnew; x += NT) gr[kept + x] = gsrc[x];
    for (int x = tid; x < kept + nnew; x += NT) al[x] = 1;
  }
}

static size_t route_scratch_bytes(const coda_layer_cfg* c) {
  const size_t te = c->Te > 0 ? c->Te : 0, ts = c->Ts > 0 ? c->Ts : 0, ms = c->Ms;
  return (size_t)c->B * 4 * (2 * te + ts + (2 * te + 2 * ts + 3 * ms + 1)) + 64;
}

extern "C" int64_t coda_b200_route_scratch_bytes(const coda_layer_cfg* cfg) {
  if (!coda_cfg_ok(cfg)) return -1;
  return (int64_t)route_scratch_bytes(cfg);
}

// K and V rows of the state and of the block can be read and written as 16-byte vectors
template <typename T>
static int rows_vec16(const RouteParams& p) {
  return (p.c.Dh * sizeof(T)) % 16 == 0 && ((uintptr_t)p.st.k_buf % 16 == 0) && ((uintptr_t)p.st.v_buf % 16 == 0) &&
         ((uintptr_t)p.kblk % 16 == 0) && ((uintptr_t)p.vblk % 16 == 0) && (p.kb_rs * sizeof(T)) % 16 == 0 &&
         (p.vb_rs * sizeof(T)) % 16 == 0 && (p.kb_bs * sizeof(T)) % 16 == 0 && (p.vb_bs * sizeof(T)) % 16 == 0;
}

template <typename T, bool PACKED>
static void launch_apply(const RouteParams& p, int nslots, cudaStream_t s) {
  const int HD = p.c.Hkv * p.c.Dh;
  const size_t smem = sizeof(float) * (size_t)HD * (HD <= 128 ? 4 : HD <= 256 ? 2 : 1);
  if (HD <= 128) coda_launch_chained(route_apply_kernel<T, 1, PACKED>, dim3((nslots + 3) / 4, p.c.B), dim3(128), smem, s, 1, p, nslots);
  else if (HD <= 256) coda_launch_chained(route_apply_kernel<T, 2, PACKED>, dim3((nslots + 1) / 2, p.c.B), dim3(128), smem, s, 1, p, nslots);
  else {
    if (smem > 48 * 1024) cudaFuncSetAttribute(route_apply_kernel<T, 8, PACKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    coda_launch_chained(route_apply_kernel<T, 8, PACKED>, dim3(nslots, p.c.B), dim3(256), smem, s, 1, p, nslots);
  }
}

template <typename T>
// phase 0: everything; 1: scores and decisions only (they read the state and write the scratch and the LRU
// stamps: nothing the attention of the same block reads is touched); 2: slot updates and the ring rewrite only.
static int launch_route(RouteParams& p, cudaStream_t s, int phase = 0) {
  const coda_layer_cfg& c = p.c;
  const int HD = c.Hkv * c.Dh;
  if ((p.te > 0 || p.ts > 0) && phase != 2) {
    const size_t smem1 = sizeof(float) * (size_t)(RS_KC * 64 + RS_KC * RS_COLS + 64 * (RS_COLS + 1) + 64 * c.Hkv + 64);
    CODA_REQUIRE(smem1 <= 200 * 1024, CODA_ERR_LIMIT, "route_block: %d KV heads too many for the scoring tile", c.Hkv);
    if (smem1 > 48 * 1024) cudaFuncSetAttribute(route_score_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
    if (c.Hkv >= 2 && c.Hkv <= 8 && c.B <= 65535) {
      // the heads of a state side by side: clusters of Hkv CTAs along z
      const bool narrow = c.Me <= 32 && c.Ms <= 32, low = c.Dh - c.Dh / 2 <= 32;
      const cudaError_t e = narrow ? (low ? launch_score_heads<T, 32, 32>(p, s) : launch_score_heads<T, 32, 64>(p, s))
                                   : (low ? launch_score_heads<T, 64, 32>(p, s) : launch_score_heads<T, 64, 64>(p, s));
      if (e != cudaSuccess) { coda_set_error("route_block (score): %s", cudaGetErrorString(e)); return CODA_ERR_LAUNCH; }
    } else {
      coda_launch_chained(route_score_kernel<T>, dim3(2, c.B), dim3(256), smem1, s, 1, p);
      CODA_CHECK_LAUNCH("route_block (score)");
    }
    const int tmax = p.te > p.ts ? p.te : p.ts;
    const size_t me1 = c.Me > 0 ? c.Me : 1;
    const size_t smem2 = me1 * (16 + 4 + 4 + 4) + 4 * ((size_t)2 * (tmax + 1) + 2 * (size_t)(p.te + 1) + 2 * (size_t)(p.ts + 1) +
                         (size_t)c.Ms + 2) + c.Me + c.Ms + 64;
    CODA_REQUIRE(smem2 <= 200 * 1024, CODA_ERR_LIMIT, "route_block: decision stage needs %zu bytes of shared memory", smem2);
    if (smem2 > 48 * 1024) cudaFuncSetAttribute(route_decide_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
    // route_decide reads candidates, gates, slot flags and stamps BEFORE its grid_chain().  That is sound because the launch
    // just before it on the stream is the scoring kernel above, every CTA of which lets it come only after its own wait (so
    // whatever wrote these is complete) and which writes ex_best, ex_bi and su_idx only.  No launch may go between the two.
    coda_launch_chained(route_decide_kernel<T>, dim3(c.B), dim3(RD_THREADS), smem2, s, 1, p);
    CODA_CHECK_LAUNCH("route_block (decide)");
  }
  if (phase == 1) return CODA_OK;
  if (p.te > 0 || p.ts > 0) {
    const int tmax = p.te > p.ts ? p.te : p.ts;
    // The entry point's documented limit.  (The kernel itself needs the new rows only: 4 bytes an element and group.)
    const size_t most = sizeof(float) * (size_t)HD + 8 * (size_t)(tmax > 0 ? tmax : 1);
    CODA_REQUIRE(most <= 200 * 1024, CODA_ERR_LIMIT, "route_block: Hkv*Dh = %d with %d candidates per block exceeds the limit (4 * Hkv*Dh + 8 * candidates = %zu, at most 204800)", HD, tmax, most);
    const int nslots = (c.Me > 0 ? p.te : 0) + (c.Ms > 0 && p.ts > 0 ? c.Ms : 0);
    if (nslots > 0) {
      if constexpr (sizeof(T) == 2) { if (rows_vec16<T>(p)) launch_apply<T, true>(p, nslots, s); else launch_apply<T, false>(p, nslots, s); }
      else launch_apply<T, false>(p, nslots, s);
      CODA_CHECK_LAUNCH("route_block (apply)");
    }
  }
  const int vec16 = rows_vec16<T>(p);
  coda_launch_chained(ring_rewrite_kernel<T>, dim3(2 * c.Hkv, c.B), dim3(256), 0, s, 1, p, vec16);
  CODA_CHECK_LAUNCH("route_block (ring)");
  return CODA_OK;
}

// ---- allocation-free variant -------------------------------------------------------------------------------
// Scratch for callers that are not allowed to allocate device memory: a fixed array in the library's own
// device image.  Every GPU that loads the library carries these bytes until the process exits.
constexpr size_t CODA_STATIC_SCRATCH_BYTES = 1u << 20;
static __device__ __align__(256) unsigned char g_route_scratch[CODA_STATIC_SCRATCH_BYTES];

extern "C" int64_t coda_b200_route_static_scratch_bytes(void) { return (int64_t)CODA_STATIC_SCRATCH_BYTES; }

// In host code `g_route_scratch` is only a handle for the symbol, not a device address; the address is looked
// up once per device (with that device current) and remembered.
static void* static_scratch_for_current_device() {
  constexpr int MAX_DEV = 64;
  static void* ptrs[MAX_DEV] = {nullptr};
  static std::mutex mu;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEV) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (ptrs[dev] == nullptr) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_route_scratch) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    ptrs[dev] = ptr;
  }
  return ptrs[dev];
}

extern "C" int coda_b200_route_block(const coda_layer_cfg* cfg, const coda_state_ptrs* st,
                                     int32_t ring_fill, int32_t blk, int64_t pos0,
                                     const void* k_blk, int64_t kb_bs, int64_t kb_rs,
                                     const void* v_blk, int64_t vb_bs, int64_t vb_rs,
                                     const float* gates, int64_t gates_bs, int64_t gate_ev0,
                                     const int32_t* cand, int64_t cand_bs,
                                     const float* eta_logit, void* scratch, coda_stream_t stream);

extern "C" int coda_b200_route_block_noalloc(const coda_layer_cfg* cfg, const coda_state_ptrs* st,
                                             int32_t ring_fill, int32_t blk, int64_t pos0,
                                             const void* k_blk, int64_t kb_bs, int64_t kb_rs,
                                             const void* v_blk, int64_t vb_bs, int64_t vb_rs,
                                             const float* gates, int64_t gates_bs, int64_t gate_ev0,
                                             const int32_t* cand, int64_t cand_bs,
                                             const float* eta_logit, coda_stream_t stream) {
  CODA_REQUIRE(coda_cfg_ok(cfg), CODA_ERR_ARG, "route_block_noalloc: invalid layer configuration");
  const size_t need = route_scratch_bytes(cfg);
  CODA_REQUIRE(need <= CODA_STATIC_SCRATCH_BYTES, CODA_ERR_LIMIT,
               "route_block_noalloc: this configuration needs %zu bytes of scratch, the built-in buffer holds %zu "
               "(fewer states per call, or use coda_b200_route_block with caller-provided scratch)",
               need, CODA_STATIC_SCRATCH_BYTES);
  void* scratch = static_scratch_for_current_device();
  CODA_REQUIRE(scratch != nullptr, CODA_ERR_LAUNCH, "route_block_noalloc: cudaGetSymbolAddress failed for the built-in scratch");
  return coda_b200_route_block(cfg, st, ring_fill, blk, pos0, k_blk, kb_bs, kb_rs, v_blk, vb_bs, vb_rs,
                               gates, gates_bs, gate_ev0, cand, cand_bs, eta_logit, scratch, stream);
}

extern "C" int coda_b200_route_block(const coda_layer_cfg* cfg, const coda_state_ptrs* st,
                                     int32_t ring_fill, int32_t blk, int64_t pos0,
                                     const void* k_blk, int64_t kb_bs, int64_t kb_rs,
                                     const void* v_blk, int64_t vb_bs, int64_t vb_rs,
                                     const float* gates, int64_t gates_bs, int64_t gate_ev0,
                                     const int32_t* cand, int64_t cand_bs,
                                     const float* eta_logit, void* scratch, coda_stream_t stream) {
  return coda_b200_route_block_phase(cfg, st, ring_fill, blk, pos0, k_blk, kb_bs, kb_rs, v_blk, vb_bs, vb_rs, gates, gates_bs,
                                     gate_ev0, cand, cand_bs, eta_logit, scratch, 0, stream);
}

extern "C" int coda_b200_route_block_phase(const coda_layer_cfg* cfg, const coda_state_ptrs* st,
                                           int32_t ring_fill, int32_t blk, int64_t pos0,
                                           const void* k_blk, int64_t kb_bs, int64_t kb_rs,
                                           const void* v_blk, int64_t vb_bs, int64_t vb_rs,
                                           const float* gates, int64_t gates_bs, int64_t gate_ev0,
                                           const int32_t* cand, int64_t cand_bs,
                                           const float* eta_logit, void* scratch, int32_t phase, coda_stream_t stream) {
  CODA_REQUIRE(coda_cfg_ok(cfg) && st, CODA_ERR_ARG, "route_block: invalid layer configuration");
  CODA_REQUIRE(phase >= 0 && phase <= 2, CODA_ERR_ARG, "route_block: phase %d is not 0, 1 or 2", phase);
  CODA_REQUIRE(blk > 0 && ring_fill >= 0 && ring_fill <= cfg->W, CODA_ERR_ARG, "route_block: bad block / ring sizes");
  CODA_REQUIRE(st->k_buf && st->v_buf && st->allowed && st->g_recent && k_blk && v_blk && gates, CODA_ERR_ARG,
               "route_block: null pointer");
  RouteParams p;
  p.c = *cfg; p.st = *st; p.fill = ring_fill; p.blk = blk;
  const int total = ring_fill + blk;
  const int keep = total < cfg->W ? total : cfg->W;
  p.n_ev = total - keep;
  const bool do_e = cfg->Me > 0 && cfg->Te > 0, do_s = cfg->Ms > 0 && cfg->Ts > 0;
  p.te = do_e ? (cfg->Te < p.n_ev ? cfg->Te : p.n_ev) : 0;
  p.ts = do_s ? (cfg->Ts < p.n_ev ? cfg->Ts : p.n_ev) : 0;
  p.pos_first = pos0 - ring_fill;
  p.kblk = k_blk; p.kb_bs = kb_bs; p.kb_rs = kb_rs; p.vblk = v_blk; p.vb_bs = vb_bs; p.vb_rs = vb_rs;
  p.gates = gates; p.gates_bs = gates_bs; p.gate_ev0 = gate_ev0;
  p.cand = cand; p.cand_bs = cand_bs; p.eta_logit = eta_logit;
  if (p.te > 0 || p.ts > 0) {
    CODA_REQUIRE(cand && scratch, CODA_ERR_ARG, "route_block: candidate list / scratch missing");
    CODA_REQUIRE(!do_e || (st->mem_last_exact && st->exact_v_norm), CODA_ERR_ARG, "route_block: exact bank pointers missing");
    CODA_REQUIRE(!do_s || (st->sum_lf_k_norm && eta_logit), CODA_ERR_ARG, "route_block: summary bank pointers missing");
    const size_t te_all = cfg->Te > 0 ? cfg->Te : 0;
    char* sp = (char*)scratch;
    p.ex_best = (float*)sp; sp += (size_t)cfg->B * te_all * 4;
    p.ex_bi = (int*)sp; sp += (size_t)cfg->B * te_all * 4;
    p.su_idx = (int*)sp; sp += (size_t)cfg->B * (cfg->Ts > 0 ? cfg->Ts : 0) * 4;
    p.plan = (int*)sp;
  } else {
    p.ex_best = nullptr; p.ex_bi = nullptr; p.su_idx = nullptr; p.plan = nullptr;
  }
  cudaStream_t s = (cudaStream_t)stream;
  return cfg->dtype == CODA_F32 ? launch_route<float>(p, s, phase) : launch_route<bf16>(p, s, phase);
}
