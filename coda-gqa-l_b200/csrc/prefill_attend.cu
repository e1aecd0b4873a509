// Chunked-prefill differential attention on the 5th-generation tensor cores (tcgen05 + TMEM), bf16.
//
// One CTA = one (state, query head, 64-row query tile) and BOTH streams, stacked as the 128 rows of every MMA: rows
// 0..63 carry the signal Q, rows 64..127 the theta-rotated noise Q of the same tokens, so the two streams share every
// K/V tile.  Keys are the layer's Lbuf slots (masked by `allowed`; 64-key tiles without a visible slot are skipped)
// followed by the block's own tokens (causal).  Per 64-key tile:
//     S = Q . K^T          tcgen05.mma  M=128 N=64 K=Dh    A, B from shared memory, S in TMEM
//     P = exp2(S - m)      softmax warps: tcgen05.ld, lazy-rescaled online softmax, bf16 P written back over S
//     O += P . V           tcgen05.mma  M=128 N=Dh K=64    A = P straight from TMEM, B = V from shared memory
// Warp roles: warps 0-7 = softmax / correction / epilogue (two warps per 32 rows, each with 32 of a tile's 64 keys),
// warp 8 = TMA producer (128-byte swizzle, K and V on rings of their own), warp 9 = MMA issuer and TMEM owner.
// What bounds it: the chain of a tile (S from TMEM, maximum, exponentials, P back), 1.6 K cycles a CTA-tile against 0.44 K
// for the exponentials' instructions alone; no pipe is more than half busy.  So everything is arranged to keep that
// chain short and several of them in flight.  S is double-buffered (S0, S1: 128 TMEM columns; with O at most 256), so
// Q.K^T of the next tile runs under the softmax of the present one, and half the tensor memory per CTA lets two CTAs share
// an SM: one CTA's start-up and epilogue (some 7 K cycles) run under the other's tiles.  64-key tiles are what fits twice;
// 64 queries x 2 streams fill the 128 rows of an MMA.
// Measured per block, against two streams of 128 rows in one CTA per SM with 128-key tiles: 64 states x 8 heads x 256
// queries over 384 slots, Dh 64: 109 -> 91 us; 512 x 9 x 128 over 192, Dh 64: 352 -> 254 us; 32 x 32 x 128 over 384, Dh
// 128: 115 -> 95 us; 8 x 64 x 256 over 768, Dh 128: 179 -> 137 us.
// All mbarrier waits are bounded (status word, no hang, TMEM is freed).
#include "coda_common.cuh"
#include "tma_utils.cuh"
#include "tensor_maps.h"

namespace {

constexpr int PF_BM = 64;        // query rows per CTA (each present twice: signal and noise)
constexpr int PF_BN = 64;        // keys per tile
constexpr int PF_M = 128;        // MMA rows
constexpr int PF_SWARPS = 8;     // softmax warps: two per 32 rows, each with half of a tile's keys
constexpr int PF_THREADS = (PF_SWARPS + 2) * 32;  // warps 0-7: softmax, 8: TMA, 9: MMA issuer
constexpr int PF_TMEM_COLS = 256;
constexpr int PF_STAGES = 2;     // K tiles (and V tiles) in flight
constexpr float PF_RESCALE_GAP = 8.0f;   // log2 units the running max may lag before O is rescaled

struct PrefillParams {
  int B, H, Hkv, Lbuf, blk, t0, mask_unused, norm_full;
  float eps, scale_log2;
  const float* lam; long long lam_bs, lam_rs;
  const uint8_t* allowed;
  const bf16* norm_w;
  bf16* out; long long out_bs, out_rs;
  int* status;
};

using tma::smem_u32;

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

// ---- tcgen05 wrappers ----
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
               "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                 "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                 "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(taddr));
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// True in one lane of the (converged) warp, always the same one
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(pred));
  return pred != 0;
}

// Shared-memory matrix descriptor, 128-byte swizzle, version 1 (Blackwell).  K-major operands (rows of 64
// bf16 = 128 bytes, 8-row groups 1024 bytes apart): lbo unused (1), sbo = 1024.  MN-major operands (rows are
// the K index, 64 MN elements per 128-byte row): lbo = distance between 64-element MN groups, sbo = 1024.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: fp32 accumulate, bf16 x bf16, M = 128, N = n, A K-major, B K-major or MN-major.
__device__ __forceinline__ constexpr uint32_t instr_desc(int n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(PF_M >> 4) << 24);
}
// 2^x for x <= 0 on the special-function unit (one MUFU op).
__device__ __forceinline__ float ex2_mufu(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Packed fp32 pairs (one instruction for two lanes of a register pair) and the three-input maximum.
__device__ __forceinline__ uint64_t pk64(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpk64(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2_rm(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rm.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// 2^x for a pair of arguments on the FMA / integer pipes: x = n + f, n = floor(x) left in the low mantissa bits by a
// round-down add of 1.5 * 2^23, 2^f by a cubic, n added into the exponent field.  The cubic is the one with p(0) = 1
// whose largest relative error on [0, 1] is smallest (a linear programme over 20001 points; 8.6e-5, far below the bf16
// rounding of P).  The special-function unit delivers one warp of exponentials per 8 cycles per scheduler; a third of
// the exponentials go this way so that neither pipe bounds the softmax.
__device__ __forceinline__ void ex2_poly2(float x0, float x1, float& y0, float& y1) {
  const uint64_t x = pk64(fmaxf(x0, -127.0f), fmaxf(x1, -127.0f));
  const uint64_t magic = pk64(12582912.0f, 12582912.0f), nmagic = pk64(-12582912.0f, -12582912.0f);
  const uint64_t t = add2_rm(x, magic);
  const uint64_t fl = add2(t, nmagic);                           // floor(x), exact
  const uint64_t mone = pk64(-1.0f, -1.0f);
  const uint64_t f = fma2(fl, mone, x);                          // x - floor(x), exact
  uint64_t r = fma2(f, pk64(0.0770680314f, 0.0770680314f), pk64(0.227643533f, 0.227643533f));
  r = fma2(r, f, pk64(0.695117286f, 0.695117286f));
  r = fma2(r, f, pk64(1.0f, 1.0f));
  float r0, r1, t0, t1;
  unpk64(r, r0, r1);
  unpk64(t, t0, t1);
  y0 = __int_as_float(__float_as_int(r0) + (__float_as_int(t0) << 23));
  y1 = __int_as_float(__float_as_int(r1) + (__float_as_int(t1) << 23));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ void bar_softmax_all() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// The two warps that share 32 rows (barrier 2 + rows / 32): a rendezvous, and one that tells whether `mine` held anywhere
__device__ __forceinline__ void bar_pair(int rows32) { asm volatile("bar.sync %0, 64;" ::"r"(2 + rows32) : "memory"); }
__device__ __forceinline__ bool bar_pair_any(int rows32, bool mine) {
  uint32_t r;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %2, 0;\nbar.red.or.pred p, %1, 64, q;\nselp.u32 %0, 1, 0, p;\n}"
               : "=r"(r) : "r"(2 + rows32), "r"(mine ? 1u : 0u) : "memory");
  return r != 0;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <int DH>
__global__ void __launch_bounds__(PF_THREADS, 2)
prefill_attend_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap qnmap,
                      const __grid_constant__ CUtensorMap kpmap, const __grid_constant__ CUtensorMap vpmap,
                      const __grid_constant__ CUtensorMap kbmap, const __grid_constant__ CUtensorMap vbmap,
                      PrefillParams p) {
  constexpr int STAGES = PF_STAGES;
  constexpr int HALVES = DH / 64;                 // 64-element (128-byte) column groups per row
  constexpr int Q_HALF = PF_M * 128;              // bytes of one column group of the stacked Q tile
  constexpr int Q_BYTES = HALVES * Q_HALF;
  constexpr int KV_HALF = PF_BN * 128;
  constexpr int KV_BYTES = HALVES * KV_HALF;      // one K (or V) tile
  constexpr int KSTEPS_QK = DH / 16;
  constexpr int KSTEPS_PV = PF_BN / 16;
  constexpr uint32_t TM_O = 2 * PF_BN;            // TMEM columns: S0 at 0, S1 at 64, O at 128

  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* sQ = smem;                        // [HALVES][128 rows][128 B]: rows 0..63 signal, 64..127 noise
  unsigned char* sK = sQ + Q_BYTES;                // [STAGES][KV_BYTES]
  unsigned char* sV = sK + STAGES * KV_BYTES;      // [STAGES][KV_BYTES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + STAGES * KV_BYTES);
  uint64_t* q_full = bars;                          // 1
  uint64_t* s_full = bars + 1;                      // [buffer] S complete; K tile n sits in stage n % 2 = buffer, so: K stage free
  uint64_t* p_full = bars + 3;                      // [buffer]
  uint64_t* k_full = bars + 5;                      // [stage]
  uint64_t* v_full = bars + 7;                      // [stage]
  uint64_t* v_empty = bars + 9;                     // [stage] P.V complete: V stage free, O quiescent
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);   // TMEM base, then the number of prefix tiles
  float* sMax = reinterpret_cast<float*>(tmem_slot + 2);   // [2][128] row maxima of the two halves of a tile, when a base may move
  uint32_t* sMask = tmem_slot + 2 + 2 * PF_M;             // [NP][2] visibility bits of the n-th tile that is read
  const int NP = (p.Lbuf + PF_BN - 1) / PF_BN;      // prefix tiles
  unsigned short* sTile = reinterpret_cast<unsigned short*>(sMask + 2 * NP);   // [NP] which tile that is

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x * PF_BM, h = blockIdx.y, b = blockIdx.z;
  const int hk = h / (p.H / p.Hkv);

  __shared__ int s_abort;                          // set by the first bounded wait of this CTA that expires
  int* const abortw = &s_abort;
  // one K (or V) tile, the it-th that is read, into its stage
  auto load_tile = [&](int it, int nv, const CUtensorMap* pm, const CUtensorMap* bm, unsigned char* ring, uint64_t* full) {
    const int st = it % STAGES;
    tma::mbar_expect_tx(&full[st], KV_BYTES);
    unsigned char* dst = ring + st * KV_BYTES;
#pragma unroll
    for (int hf = 0; hf < HALVES; ++hf) {
      if (it < nv) tma_load_3d(dst + hf * KV_HALF, pm, &full[st], hf * 64, (int)sTile[it] * PF_BN, b * p.Hkv + hk);
      else tma_load_4d(dst + hf * KV_HALF, bm, &full[st], hf * 64, hk, p.t0 + (it - nv) * PF_BN, b);
    }
  };
  if (warp == PF_SWARPS) {
    if (lane == 0) {
      s_abort = 0;
      tma::mbar_init(q_full, 1);
      for (int i = 0; i < 2; ++i) {
        tma::mbar_init(&s_full[i], 1); tma::mbar_init(&p_full[i], PF_SWARPS);
        tma::mbar_init(&k_full[i], 1); tma::mbar_init(&v_full[i], 1); tma::mbar_init(&v_empty[i], 1);
      }
      tma::fence_barrier_init();
    }
    grid_chain();
    if (lane == 0) {                                 // (the barriers are this thread's own so far: Q may leave at once)
      tma::mbar_expect_tx(q_full, Q_BYTES);
#pragma unroll
      for (int hf = 0; hf < HALVES; ++hf) {
        tma_load_4d(sQ + hf * Q_HALF, &qmap, q_full, hf * 64, h, p.t0 + r0, b);
        tma_load_4d(sQ + hf * Q_HALF + PF_BM * 128, &qnmap, q_full, hf * 64, h, p.t0 + r0, b);
      }
    }
    // visibility of the prefix slots; tiles with no visible slot drop out
    const uint8_t* al = p.allowed + (long long)b * p.Lbuf;
    int nv = 0;
    for (int j0 = 0; j0 < NP; j0 += 4) {
      bool vis[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = j0 * PF_BN + i * 32 + lane;
        vis[i] = c < p.Lbuf && (!p.mask_unused || al[c] != 0);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned lo = __ballot_sync(0xffffffffu, vis[2 * i]), hi = __ballot_sync(0xffffffffu, vis[2 * i + 1]);
        if ((lo | hi) != 0u) {
          if (lane == 0) { sTile[nv] = (unsigned short)(j0 + i); sMask[2 * nv] = lo; sMask[2 * nv + 1] = hi; }
          ++nv;
        }
      }
    }
    if (lane == 0) {
      tmem_slot[1] = (uint32_t)nv;
      load_tile(0, nv, &kpmap, &kbmap, sK, k_full);
      if (nv + r0 / PF_BN + 1 > 1) load_tile(1, nv, &kpmap, &kbmap, sK, k_full);
      load_tile(0, nv, &vpmap, &vbmap, sV, v_full);
    }
  } else if (warp == PF_SWARPS + 1) {                // TMEM: half of the SM's columns, owned by the MMA warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(PF_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot[0];
  const int NV = (int)tmem_slot[1];                  // prefix tiles that are read
  const int NT = NV + r0 / PF_BN + 1;                // ... and the block tiles up to the diagonal

  if (warp == PF_SWARPS) {
    // =========================== TMA producer ===========================
    // K tile it needs Q.K^T it-2 to be done, long before V tile it needs P.V it-2: K runs one tile ahead
    if (lane == 0) {
      for (int it = 1; it < NT; ++it) {
        if (it + 1 < NT) {
          tma::mbar_wait(&s_full[(it + 1) & 1], ((it - 1) >> 1) & 1, p.status, 11, abortw);
          load_tile(it + 1, NV, &kpmap, &kbmap, sK, k_full);
        }
        if (it >= 2) tma::mbar_wait(&v_empty[it & 1], ((it - 2) >> 1) & 1, p.status, 15, abortw);
        load_tile(it, NV, &vpmap, &vbmap, sV, v_full);
      }
    }
  } else if (warp == PF_SWARPS + 1) {
    // =========================== MMA issuer ===========================
    // The whole warp walks the loop and one elected lane issues: descriptors stay in uniform registers that way.  Under
    // a lane == 0 branch they are moved there one by one, some 100 cycles per MMA (430 + 790 cycles for a tile's P.V and
    // Q.K^T), and the issue becomes the longest chain of the tile.
    constexpr uint32_t IDESC_QK = instr_desc(PF_BN, false);
    constexpr uint32_t IDESC_PV = instr_desc(DH, true);
    const uint64_t qdesc = smem_desc(smem_u32(sQ), 16, 1024), kdesc = smem_desc(smem_u32(sK), 16, 1024);
    const uint64_t vdesc = smem_desc(smem_u32(sV), KV_HALF, 1024);
    // S = Q . K^T into buffer it & 1 (free: the P.V two tiles back, which read P from it, was issued earlier by
    // this same lane and the tensor pipe executes in order)
    auto issue_qk = [&](int it) {
      tma::mbar_wait(&k_full[it & 1], (it >> 1) & 1, p.status, 14, abortw);
      tc_fence_after();
      const uint64_t kd = kdesc + (uint32_t)(it & 1) * (KV_BYTES >> 4);
      const uint32_t dcol = tmem + (uint32_t)(it & 1) * PF_BN;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < KSTEPS_QK; ++kk)
          tc_mma(dcol, qdesc + (((kk >> 2) * Q_HALF + (kk & 3) * 32) >> 4), kd + (((kk >> 2) * KV_HALF + (kk & 3) * 32) >> 4), IDESC_QK, kk > 0 ? 1u : 0u);
        tc_commit(&s_full[it & 1]);
      }
      __syncwarp();
    };
    tma::mbar_wait(q_full, 0, p.status, 13, abortw);
    issue_qk(0);
    if (NT > 1) issue_qk(1);
    for (int it = 0; it < NT; ++it) {
      tma::mbar_wait(&v_full[it & 1], (it >> 1) & 1, p.status, 17, abortw);
      tma::mbar_wait(&p_full[it & 1], (it >> 1) & 1, p.status, 12, abortw);
      tc_fence_after();
      const uint64_t vd = vdesc + (uint32_t)(it & 1) * (KV_BYTES >> 4);
      const uint32_t pcol = tmem + (uint32_t)(it & 1) * PF_BN;      // P (bf16 pairs) sits in the first 32 columns of S
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < KSTEPS_PV; ++kk)
          tc_mma_ts(tmem + TM_O, pcol + kk * 8, vd + ((kk * 2048) >> 4), IDESC_PV, (it > 0 || kk > 0) ? 1u : 0u);
        tc_commit(&v_empty[it & 1]);
      }
      __syncwarp();
      if (it + 2 < NT) issue_qk(it + 2);
    }
  } else {
    // =========================== softmax / correction / epilogue ===========================
    grid_chain();                                         // (lambda and the output rows are this role's)
    const int quarter = warp & 3;                         // TMEM lanes this warp may touch: 32 * quarter ..
    const int hf = warp >> 2;                             // keys 32 * hf .. of every tile
    const int s = quarter >> 1;                           // 0 = signal rows, 1 = noise rows
    const int row = (quarter & 1) * 32 + lane;            // row of the query tile
    const int grow = r0 + row;                            // row inside the block
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t o_col = lane_addr + TM_O;

    // Visibility of this warp's 32 keys of a tile.  The class (2 = all visible, 0 = none, 1 = mixed) is the same for
    // every lane of a warp: prefix slots carry one mask per state, and in a block tile the 32 rows of a warp
    // meet the causal diagonal inside one group only.
    auto visible = [&](int it, uint32_t& vis) {
      if (it < NV) {
        vis = sMask[2 * it + hf];
        return vis == 0xffffffffu ? 2 : (vis == 0u ? 0 : 1);
      }
      const int c0 = (it - NV) * PF_BN + 32 * hf;
      const int nvis = grow - c0 + 1;                     // key c0+i visible iff c0+i <= grow
      const int gd = (r0 + (quarter & 1) * 32 - c0) >> 5; // 0: this group holds the warp's diagonal
      vis = nvis >= 32 ? 0xffffffffu : (nvis <= 0 ? 0u : ((1u << nvis) - 1u));
      return gd > 0 ? 2 : (gd == 0 ? 1 : 0);
    };
    // This warp's part of S of a tile, and the row maximum over its visible keys (the others become -inf)
    auto load_s = [&](int it, uint32_t vis, int cls, uint32_t (&v)[32]) {
      tma::mbar_wait(&s_full[it & 1], (it >> 1) & 1, p.status, 16, abortw);
      tc_fence_after();
      tc_ld32(lane_addr + (uint32_t)(it & 1) * PF_BN + hf * 32, v);
      tc_wait_ld();
      float m0 = -INFINITY, m1 = -INFINITY;
      if (cls == 2) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          m0 = max3(m0, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
          m1 = max3(m1, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
        }
      } else if (cls == 1) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (!((vis >> i) & 1u)) v[i] = 0xff800000u;     // -inf: exp gives 0 below
          m0 = fmaxf(m0, __uint_as_float(v[i]));
        }
      }
      return fmaxf(m0, m1);
    };

    float mb = -INFINITY;                                 // exponent base (lags the true max by < GAP), the same in both halves
    float l = 0.f;                                        // sum over this warp's keys
    // The first base is the maximum over the first TWO tiles (128 keys).  A weight at the base is 1 in bf16 and carries
    // no rounding error; where the base lags, the row's largest weight carries up to 2^-8 of itself, and in a row that one
    // key dominates that is the error of the output.  With one tile's maximum the attention of 130 slots and 64
    // tokens was 2.2e-3 off 64 bits where it now is 2.0e-3, most of it the rounding of the result (queries of standard
    // deviation 2; the rounding of the weights alone: 1.3e-3 against 0.9e-3).
    // It costs a CTA the wait for the second Q.K^T: 88.4 -> 90.8, 242 -> 254, 90.5 -> 95.5 and 131 -> 137 us at the four shapes above.
    float ahead = -INFINITY;
    if (NT > 1) {
      uint32_t vis, v[32];
      const int cls = visible(1, vis);
      ahead = load_s(1, vis, cls, v);
    }
    for (int it = 0; it < NT; ++it) {
      const uint32_t s_col = lane_addr + (uint32_t)(it & 1) * PF_BN;
      uint32_t vis, v[32];
      const int cls = visible(it, vis);
      const float ms = fmaxf(load_s(it, vis, cls, v), ahead);
      ahead = -INFINITY;
      float mx = ms * p.scale_log2;                       // scale > 0: max commutes with the scaling
      // The other half of the row is in another warp.  Most tiles move no base: one barrier says so for the 32 rows (and
      // that both warps hold their part of S in registers, which P may then overwrite); else the maxima are exchanged.
      if (bar_pair_any(quarter, mx > mb + PF_RESCALE_GAP || (mb == -INFINITY && mx > -INFINITY))) {
        sMax[hf * PF_M + quarter * 32 + lane] = mx;
        bar_pair(quarter);
        mx = fmaxf(mx, sMax[(1 - hf) * PF_M + quarter * 32 + lane]);
        float alpha = 1.f;
        if (mx > mb + PF_RESCALE_GAP || (mb == -INFINITY && mx > -INFINITY)) {
          alpha = (mb == -INFINITY) ? 0.f : exp2f(mb - mx);
          mb = mx;
          l *= alpha;
        }
        // Rescale O, each warp half of its columns, when some row moved its exponent base (not for the first tile: the
        // first P.V overwrites O instead of accumulating); O must be quiescent: wait for the previous P.V.  (s_full of
        // tile it was committed behind P.V it-2, so the barrier of P.V it-1 is at most one phase behind and its parity is
        // not ambiguous; the same holds for the last P.V in the epilogue.)
        if (it > 0) {
          tma::mbar_wait(&v_empty[(it - 1) & 1], ((it - 1) >> 1) & 1, p.status, 19, abortw);
          tc_fence_after();
#pragma unroll 1
          for (int c = hf * (DH / 32); c < (hf + 1) * (DH / 32); ++c) {
            uint32_t o[16];
            tc_ld16(o_col + c * 16, o);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tc_st16(o_col + c * 16, o);
          }
        }
      }
      // probabilities, written back over S as packed bf16 (key 2i, 2i+1 -> column i)
      const float nref = mb == -INFINITY ? 0.f : -mb;
      const uint64_t scale2 = pk64(p.scale_log2, p.scale_log2), nref2 = pk64(nref, nref);
      uint64_t sum0 = 0ull, sum1 = 0ull;                  // independent chains of packed pairs
      uint32_t pk[16];
      if (cls == 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[i] = 0u;
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          // exponent arguments of two keys per instruction; two pairs in three on the special-function
          // unit, the third on the FMA pipe
          float x0, x1, a0, a1;
          unpk64(fma2(pk64(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), scale2, nref2), x0, x1);
          if (i % 3 == 2) { ex2_poly2(x0, x1, a0, a1); } else { a0 = ex2_mufu(x0); a1 = ex2_mufu(x1); }
          const uint64_t pr = pk64(a0, a1);
          if (i & 1) sum1 = add2(sum1, pr); else sum0 = add2(sum0, pr);
          pk[i] = pack2(a0, a1);
        }
      }
      tc_st16(s_col + hf * 16, pk);
      {
        float t0, t1;
        unpk64(add2(sum0, sum1), t0, t1);
        l += t0 + t1;
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&p_full[it & 1]);
    }

    // ---- epilogue: signal / l_s - lambda * noise / l_n, head RMSNorm, store ----
    // The two streams of a query row sit 64 TMEM lanes apart.  A thread finishes one quarter of the columns of its query
    // (signal rows the lower half, noise rows the upper, each warp of the pair half of that) and hands the quarter its
    // partner in the other stream finishes, normalised, through the shared memory of the query tile, which is dead once
    // every Q.K^T has completed; row sums and partial sums of squares go through the K ring and the rounded rows
    // through the V ring, so that a warp stores whole rows.  16-byte chunks are XORed with the row so that neither the
    // row-wise writes nor the reads collide in a bank.  fp32 end to end with a single rounding of the result.
    const bool valid = grow < p.blk;
    float lam = 0.f;
    if (valid) lam = bf16_round(p.lam[(long long)b * p.lam_bs + (long long)(p.t0 + grow) * p.lam_rs + h]);
    constexpr int HC = DH / 2, HQ = DH / 4;                // columns per stream, per thread
    tma::mbar_wait(&v_empty[(NT - 1) & 1], ((NT - 1) >> 1) & 1, p.status, 18, abortw);
    tc_fence_after();
    float* xl = reinterpret_cast<float*>(sK);              // [2][128] row sums of the halves
    float* xsq = xl + 2 * PF_M;                            // [4][64] partial sums of squares
    xl[hf * PF_M + quarter * 32 + lane] = l;
    bar_pair(quarter);
    l += xl[(1 - hf) * PF_M + quarter * 32 + lane];
    const float inv = l > 0.f ? 1.f / l : 0.f;
    constexpr int XM = HC / 4 - 1;                         // chunks of 4 floats per exchanged row, minus one
    float4* xown = reinterpret_cast<float4*>(sQ) + (size_t)(s * PF_BM + row) * (HC / 4);
    const float4* xpart = reinterpret_cast<const float4*>(sQ) + (size_t)((1 - s) * PF_BM + row) * (HC / 4);
    auto load_o = [&](int col, uint32_t (&o)[HQ]) {
      if constexpr (HQ == 32) tc_ld32(o_col + col, o); else tc_ld16(o_col + col, o);
      tc_wait_ld();
    };
    {
      uint32_t o[HQ];
      load_o((1 - s) * HC + hf * HQ, o);
#pragma unroll
      for (int i = 0; i < HQ / 4; ++i)
        xown[(hf * (HQ / 4) + i) ^ (row & XM)] = make_float4(__uint_as_float(o[4 * i]) * inv, __uint_as_float(o[4 * i + 1]) * inv,
                                                             __uint_as_float(o[4 * i + 2]) * inv, __uint_as_float(o[4 * i + 3]) * inv);
    }
    bar_softmax_all();
    float dv[HQ];                                          // sig - lam * noise of this thread's columns
    float sq = 0.f;
    {
      uint32_t o[HQ];
      load_o(s * HC + hf * HQ, o);
#pragma unroll
      for (int i = 0; i < HQ / 4; ++i) {
        const float4 x = xpart[(hf * (HQ / 4) + i) ^ (row & XM)];
        const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float own = __uint_as_float(o[4 * i + e]) * inv;
          const float d = s == 0 ? fmaf(-lam, xv[e], own) : fmaf(-lam, own, xv[e]);
          sq = fmaf(d, d, sq);
          dv[4 * i + e] = d;
        }
      }
    }
    float rs = 1.f;
    if (p.norm_full) {
      xsq[(s * 2 + hf) * PF_BM + row] = sq;
      bar_softmax_all();
      rs = rsqrtf(((xsq[row] + xsq[PF_BM + row]) + (xsq[2 * PF_BM + row] + xsq[3 * PF_BM + row])) / (float)DH + p.eps);
    }
    constexpr int RC = DH / 8;                             // 16-byte chunks per output row
    uint4* srow = reinterpret_cast<uint4*>(sV) + (size_t)row * RC;
    const int cbase = (s * 2 + hf) * HQ;                   // first of this thread's columns
#pragma unroll
    for (int i = 0; i < HQ / 8; ++i) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float y0 = dv[8 * i + 2 * e] * rs, y1 = dv[8 * i + 2 * e + 1] * rs;
        if (p.norm_full) {
          const __nv_bfloat162 wv = reinterpret_cast<const __nv_bfloat162*>(p.norm_w)[cbase / 2 + 4 * i + e];
          y0 *= __low2float(wv); y1 *= __high2float(wv);
        }
        w[e] = pack2(y0, y1);
      }
      srow[(cbase / 8 + i) ^ (row & (RC - 1))] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    bar_softmax_all();
    bf16* ob = p.out + (long long)b * p.out_bs + (long long)(p.t0 + r0) * p.out_rs + (long long)h * DH;
#pragma unroll
    for (int i = 0; i < PF_BM * RC / (32 * PF_SWARPS); ++i) {
      const int x = i * 32 * PF_SWARPS + tid, rr = x / RC, cc = x % RC;
      if (r0 + rr < p.blk)
        *reinterpret_cast<uint4*>(ob + (long long)rr * p.out_rs + cc * 8) = reinterpret_cast<const uint4*>(sV)[rr * RC + (cc ^ (rr & (RC - 1)))];
    }
    tc_fence_before();
  }

  __syncthreads();                                     // every role meets here once all tensor work is done
  if (warp == PF_SWARPS + 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(PF_TMEM_COLS) : "memory");
  }
}

template <int DH>
size_t prefill_smem(int Lbuf) {
  const int NP = (Lbuf + PF_BN - 1) / PF_BN;
  return (size_t)(DH / 64) * PF_M * 128 + 2 * PF_STAGES * (size_t)(DH / 64) * PF_BN * 128 +
         11 * 8 + 8 + 2 * PF_M * 4 + (size_t)NP * 10 + 1024 + 16;
}

template <int DH>
int launch_prefill(const CUtensorMap* maps, const PrefillParams& p, cudaStream_t s) {
  const size_t smem = prefill_smem<DH>(p.Lbuf);
  CODA_REQUIRE(smem <= 226 * 1024, CODA_ERR_LIMIT, "prefill_attend: %d slots need %zu bytes of shared memory", p.Lbuf, smem);
  static coda_device_once once;
  coda_on_first_use(once, [] {
    cudaFuncSetAttribute(prefill_attend_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
  });
  dim3 grid((p.blk + PF_BM - 1) / PF_BM, p.H, p.B);
  coda_launch_chained(prefill_attend_kernel<DH>, grid, dim3(PF_THREADS), smem, s, 1, maps[0], maps[1], maps[2], maps[3], maps[4], maps[5], p);
  CODA_CHECK_LAUNCH("prefill_attend");
  return CODA_OK;
}

}  // namespace

extern "C" int coda_b200_prefill_attend_supported(const coda_layer_cfg* cfg) {
  if (!coda_cfg_ok(cfg)) return 0;
  return cfg->dtype == CODA_BF16 && (cfg->Dh == 64 || cfg->Dh == 128) && tmaps::available();
}

extern "C" int coda_b200_prefill_attend(const coda_layer_cfg* cfg, const coda_state_ptrs* st,
                                        int32_t L, int32_t t0, int32_t blk,
                                        const void* q, int64_t q_bs, int64_t q_rs,
                                        const void* q_noise, int64_t qn_bs, int64_t qn_rs,
                                        const float* lam, int64_t lam_bs, int64_t lam_rs,
                                        const void* k_seq, int64_t k_bs, int64_t k_rs,
                                        const void* v_seq, int64_t v_bs, int64_t v_rs,
                                        const void* norm_w, void* out, int64_t out_bs, int64_t out_rs,
                                        int32_t* status, coda_stream_t stream) {
  CODA_REQUIRE(coda_cfg_ok(cfg) && st, CODA_ERR_ARG, "prefill_attend: invalid layer configuration");
  CODA_REQUIRE(coda_b200_prefill_attend_supported(cfg), CODA_ERR_ARG, "prefill_attend: needs bf16 and head_dim 64 or 128");
  CODA_REQUIRE(L > 0 && blk > 0 && t0 >= 0 && t0 + blk <= L, CODA_ERR_ARG, "prefill_attend: block [%d, %d) outside the %d tokens", t0, t0 + blk, L);
  CODA_REQUIRE(q && q_noise && lam && k_seq && v_seq && out && st->k_buf && st->v_buf && st->allowed, CODA_ERR_ARG,
               "prefill_attend: null pointer");
  CODA_REQUIRE(!cfg->head_norm_full || norm_w, CODA_ERR_ARG, "prefill_attend: head-norm weight missing");
  const uintptr_t al = (uintptr_t)q | (uintptr_t)q_noise | (uintptr_t)k_seq | (uintptr_t)v_seq | (uintptr_t)out |
                       (uintptr_t)st->k_buf | (uintptr_t)st->v_buf;
  CODA_REQUIRE(al % 16 == 0 && (q_bs | q_rs | qn_bs | qn_rs | k_bs | k_rs | v_bs | v_rs | out_bs | out_rs) % 8 == 0, CODA_ERR_ARG,
               "prefill_attend: pointers must be 16-byte aligned and strides multiples of 8 elements");
  const int Lbuf = cfg->W + cfg->Me + cfg->Ms, Dh = cfg->Dh;
  CUtensorMap maps[6];
  const bool ok = tmaps::token_map(&maps[0], q, cfg->B, L, cfg->H, Dh, q_bs, q_rs, PF_BM) &&
                  tmaps::token_map(&maps[1], q_noise, cfg->B, L, cfg->H, Dh, qn_bs, qn_rs, PF_BM) &&
                  tmaps::plane_map(&maps[2], st->k_buf, cfg->B * cfg->Hkv, Lbuf, Dh, PF_BN) &&
                  tmaps::plane_map(&maps[3], st->v_buf, cfg->B * cfg->Hkv, Lbuf, Dh, PF_BN) &&
                  tmaps::token_map(&maps[4], k_seq, cfg->B, L, cfg->Hkv, Dh, k_bs, k_rs, PF_BN) &&
                  tmaps::token_map(&maps[5], v_seq, cfg->B, L, cfg->Hkv, Dh, v_bs, v_rs, PF_BN);
  CODA_REQUIRE(ok, CODA_ERR_LAUNCH, "prefill_attend: cuTensorMapEncodeTiled failed");
  PrefillParams p;
  p.B = cfg->B; p.H = cfg->H; p.Hkv = cfg->Hkv; p.Lbuf = Lbuf; p.blk = blk; p.t0 = t0;
  p.mask_unused = cfg->mask_unused; p.norm_full = cfg->head_norm_full; p.eps = cfg->eps;
  p.scale_log2 = 1.4426950408889634f / sqrtf((float)Dh);
  p.lam = lam; p.lam_bs = lam_bs; p.lam_rs = lam_rs; p.allowed = st->allowed; p.norm_w = (const bf16*)norm_w;
  p.out = (bf16*)out; p.out_bs = out_bs; p.out_rs = out_rs; p.status = status;
  cudaStream_t s = (cudaStream_t)stream;
  return Dh == 128 ? launch_prefill<128>(maps, p, s) : launch_prefill<64>(maps, p, s);
}
