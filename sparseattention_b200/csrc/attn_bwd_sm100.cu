// Backward pass of the block-sparse attention forward with TMA + tcgen05 + TMEM (fp16 / bf16, head dim 64 or
// 128, BLOCK_Q 128, BLOCK_K 32 / 64 / 128; everything else runs attn_bwd_mma.cu or attn_bwd_simt.cu).
//
// The reference has no backward (README.md:61-65); the mathematics is that of attn_bwd_simt.cu:
//
//   P_ij  = exp(q_i.k_j * scale - lse_i)  on attended (i, j) of listed tiles, 0 elsewhere
//   D_i   = sum_d dO_id * O_id  (- the incoming gradient of lse_i, when there is one)
//   dV_j  = sum_i P_ij dO_i          dS_ij = P_ij * (dO_i.v_j - D_i)
//   dQ_i  = scale * sum_j dS_ij k_j  dK_j  = scale * sum_i dS_ij q_i
//
// One kernel template in two modes, no atomics (the result does not depend on the order CTAs run in).  A CTA
// owns 128 rows of one side -- query rows (mode 0: dQ) or kv rows (mode 1: dK, dV) -- and walks a list of the
// other side in steps of 128 rows gathered by TMA.  With A1, A2 the owned tiles (Q, dO / K, V) and X, Y the
// streamed ones (K, V / Q, dO), a step is
//
//   S = A1.X^T,  T = A2.Y^T             both operands in shared memory, 128 x 128 fp32 in tensor memory
//   P = exp2(S * scale - lse2),  dS = P * (T - D)     256 threads: a row and one half of the 128 columns each
//   mode 0: acc += dS.X                 dS read as the A operand from tensor memory, X as an MN-major B operand
//   mode 1: acc1 += P.Y, acc2 += dS.X   the same tile of X / Y serves both products
//
// so P and dS never pass through shared memory: in both modes the owned rows are the lanes of tensor memory.
// The walk of mode 1 lists 32-row query chunks per 128 kv rows: the forward's lists are tall along the query
// side, and 32 x 128 tiles keep the density that 128 x 32 tiles have in the forward (128 x 128 tiles of a mask
// of 32 x 32 blocks kept with probability 0.1 would be 81 % listed, these are 34 %).  Its lists and a bit plane
// whose words run along the query side are made by two small kernels from the forward's lists and plane.
//
// What bounds it: a step is 2048 (mode 1) / 1536 (mode 0) cycles of tensor pipe, 2048 / 1792 cycles of shared
// memory at 128 B a cycle (operands and TMA writes) and 1024 cycles of exponential unit.  Shared memory has room
// for the owned tiles and two stages of X and Y, tensor memory (512 columns) for the accumulators, S and T, so
// P overwrites S and dS overwrites T; the products are ordered such that the tensor pipe has one half of a
// step's products to do while the 256 threads work on the other half.
//
// Measured (one B200): B=4 H=8 S=4096 D=128 bf16, 32 x 32 blocks dropped with p = 0.5, lists at (128, 32), forward +
// backward through autograd 5.17 ms with attn_bwd_mma.cu, 1.31 ms with this kernel.  The backward alone is 0.98 ms
// (0.9 PFLOP/s over the seven products of the listed tiles): row statistics and lists 0.04, and with only the CTAs of one
// mode dK / dV 0.47 and dQ 0.48 ms.  Tensor pipe active 44 % of the launch.
//
// A product with an infinite or NaN row of dO or Q reaches every kv row of a listed 32 x 128 tile (0 * inf), as it
// reached those of a listed 128 x 32 tile before.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <mutex>

#include "ptx_sm100.cuh"
#include "sa_common.cuh"
#include "tensor_map.cuh"

namespace sa {
namespace {

constexpr int kOwn = 128;            // rows a CTA owns
constexpr int kStep = 128;           // rows of the other side per step
constexpr int kChunkQ = 32;          // query rows per list entry of mode 1
constexpr int kThreadsB = 384;       // warps: X producer, Y producer, MMA issuer, idle, 8 x element-wise
constexpr int kMathWarp0 = 4;
constexpr int kStagesB = 2;
constexpr uint32_t kPanel = 128u * 128u;      // 128 rows x 64 elements x 2 B
constexpr uint32_t kColS = 0, kColT = 128;    // mode 0: T buffers at 128 and 256, dQ at 384; mode 1: T at 128, dV at 256, dK at 384
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

enum BarB : int {
  BB_OWN = 0,                                    // the owned tiles landed
  BB_X_FULL,                                     // 2: X tile (and mask words, and row statistics in mode 1) landed
  BB_X_EMPTY = BB_X_FULL + kStagesB,             // 2: last product that reads it complete
  BB_Y_FULL = BB_X_EMPTY + kStagesB,
  BB_Y_EMPTY = BB_Y_FULL + kStagesB,
  BB_S_FULL = BB_Y_EMPTY + kStagesB,             // scores of a step complete
  BB_S_DONE,                                     // mode 0: scores read; mode 1: P written over them
  BB_T_FULL,                                     // 2: dO.V^T of a step complete (parity of the step)
  BB_DS_FULL = BB_T_FULL + 2,                    // 2: dS written over it
  BB_ACC = BB_DS_FULL + 2,                       // the accumulators are final
  BB_COUNT
};

template <int D>
struct SmemB {
  static constexpr uint32_t kTile = kPanel * (D / 64);
  static constexpr uint32_t off_a = 0;                                        // A1, A2
  static constexpr uint32_t off_x = 2 * kTile;
  static constexpr uint32_t off_y = off_x + kStagesB * kTile;
  static constexpr uint32_t off_bits = off_y + kStagesB * kTile;              // [stage][4 sub-slots][128 rows] u32
  static constexpr uint32_t off_stat = off_bits + kStagesB * 4 * 128 * 4;     // [stage][-lse2 | D][128] f32 (mode 1)
  static constexpr uint32_t off_bar = off_stat + kStagesB * 2 * 128 * 4;
  static constexpr uint32_t off_misc = off_bar + 8 * 24;                      // TMEM base, abort flag
  static constexpr uint32_t off_ids = off_misc + 16;                          // per producer warp [4 steps][4 entries]
  static constexpr uint32_t total = off_ids + 2 * 64;
  static constexpr uint32_t dynamic_bytes = total + 1024;
};
static_assert(BB_COUNT <= 24, "barrier area too small");
static_assert(SmemB<128>::dynamic_bytes <= 232448, "shared memory");

template <typename T> struct FmtB;
template <> struct FmtB<__half> {
  static constexpr uint32_t umma = 0;
  static __device__ __forceinline__ uint32_t pack2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ float up(__half x) { return __half2float(x); }
};
template <> struct FmtB<__nv_bfloat16> {
  static constexpr uint32_t umma = 1;
  static __device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ float up(__nv_bfloat16 x) { return __bfloat162float(x); }
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct BwdArgs {
  AttnBwdParams p;
  const float* nlse2;            // [B,H,Sq]: -lse in base 2, -inf for a row that attended nothing
  const float* dsum;             // [B,H,Sq]
  // the walk of mode 1: per (plane, 128 kv rows) the listed 32-row query chunks -- those every element of which
  // is attended from the front of the row, the others from its end backwards -- and the counts of both
  const int32_t* t_ids;          // [planes, kv tiles, Sq / 32]
  const int32_t* t_lens;         // [planes, kv tiles, 2]
  const uint32_t* t_bits;        // [planes, Sq / 32, sk_pad]: bit j of word [., c, r] = kv row r is attended by query 32 c + j
  int64_t plane_b, plane_h;      // plane index = b * plane_b + h * plane_h
  int sk_pad;                    // kv rows rounded up to 128
};

// 32 columns of S -> P.  kCol: -lse2 is per column (nl: the 32 values in shared memory) instead of one value.
template <bool kCol, bool kMasked>
__device__ __forceinline__ void probs(const uint32_t (&s)[32], uint32_t w, uint64_t scale2, uint64_t nl_own,
                                      const float* nl, float (&pr)[32]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    uint64_t n0 = nl_own, n1 = nl_own;
    if (kCol) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(nl + 4 * i);
      n0 = v.x; n1 = v.y;
    }
    float x[4];
    ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_u32x2(s[4 * i], s[4 * i + 1]), scale2, n0), x[0], x[1]);
    ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_u32x2(s[4 * i + 2], s[4 * i + 3]), scale2, n1), x[2], x[3]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (kMasked) x[e] = (w >> (4 * i + e)) & 1u ? x[e] : -INFINITY;
      pr[4 * i + e] = ex2(x[e]);
    }
  }
}

template <typename T, int D, int MODE>
__device__ __forceinline__ void bwd_body(const BwdArgs& a, const CUtensorMap* tm_a1, const CUtensorMap* tm_a2,
                                         const CUtensorMap* tm_x, const CUtensorMap* tm_y, const int tile) {
  using L = SmemB<D>;
  const AttnBwdParams& p = a.p;
  const AttnParams& f = p.fwd;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = ptx::smem_u32(smem);
  const uint32_t sA = sbase + L::off_a, sX = sbase + L::off_x, sY = sbase + L::off_y;
  auto bar = [&](int i) { return sbase + L::off_bar + 8u * static_cast<uint32_t>(i); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::off_misc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::off_misc + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int tiles = MODE == 0 ? f.Sq / kOwn : a.sk_pad / kOwn;
  const int bh = tile / tiles, own = tile - bh * tiles;
  const int b = bh / f.H, h = bh - b * f.H;
  const int row0 = own * kOwn;

  // the walk: `n_full` entries of fids (no mask), then `total - n_full` of pids (mask words)
  const int32_t *fids, *pids;
  int64_t fstr, pstr;
  int n_full, total, n_entries;                    // n_entries: ids must lie in [0, n_entries)
  const uint32_t* words;                           // mask words of this CTA's rows: [32-column group][row], pitch words apart
  int64_t pitch;
  if (MODE == 0) {
    fids = f.full_ids + b * f.fis[0] + h * f.fis[1] + static_cast<int64_t>(own) * f.fis[2];
    pids = f.part_ids + b * f.pis[0] + h * f.pis[1] + static_cast<int64_t>(own) * f.pis[2];
    fstr = f.fis[3]; pstr = f.pis[3];
    n_entries = f.Sk / f.BK;
    n_full = min(max(f.full_lens[b * f.fls[0] + h * f.fls[1] + static_cast<int64_t>(own) * f.fls[2]], 0), n_entries);
    total = n_full +
            min(max(f.part_lens[b * f.pls[0] + h * f.pls[1] + static_cast<int64_t>(own) * f.pls[2]], 0), n_entries);
    words = f.bits + b * f.bits_sb + h * f.bits_sh + row0;
    pitch = f.Sq;
  } else {
    const int64_t plane = b * a.plane_b + h * a.plane_h;
    n_entries = f.Sq / kChunkQ;
    fids = a.t_ids + (plane * tiles + own) * n_entries;
    pids = fids + n_entries - 1;
    fstr = 1; pstr = -1;
    n_full = a.t_lens[(plane * tiles + own) * 2];
    total = n_full + a.t_lens[(plane * tiles + own) * 2 + 1];
    words = a.t_bits + plane * n_entries * static_cast<int64_t>(a.sk_pad) + row0;
    pitch = a.sk_pad;
  }
  // entries per step (4, 2, 1) and 32-column groups per entry (1, 2, 4)
  const int eps_shift = MODE == 1 || f.BK == 32 ? 2 : (f.BK == 64 ? 1 : 0);
  const int sps_shift = 2 - eps_shift;
  const int eps = 1 << eps_shift;
  const int entry_rows = kStep >> eps_shift;
  const int n_steps = (total + eps - 1) >> eps_shift;
  const int n_plain = n_full >> eps_shift;         // leading steps without mask words

  if (threadIdx.x == 0) {
    for (int i = 0; i < BB_COUNT; ++i) {
      const bool many = i == BB_S_DONE || i == BB_DS_FULL || i == BB_DS_FULL + 1;
      ptx::mbar_init(bar(i), many ? 8 : 1);        // one arrival per element-wise warp
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), 512u);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (n_steps > 0 && warp < 2) {
    // ------------------------------------------------------------------ producers: warp 0 X, warp 1 Y
    const bool is_x = warp == 0;
    const CUtensorMap* tm = is_x ? tm_x : tm_y;
    const uint32_t s_tiles = is_x ? sX : sY;
    const int bar_full = is_x ? BB_X_FULL : BB_Y_FULL, bar_empty = is_x ? BB_X_EMPTY : BB_Y_EMPTY;
    const int64_t* xs = MODE == 0 ? (is_x ? f.ks : f.vs) : (is_x ? f.qs : p.dos);
    const int cb = xs[0] ? b : 0, ch = xs[1] ? h : 0;
    if (lane == 0) {
      ptx::prefetch_tensormap(tm);
      if (is_x) {
        const int64_t *s1 = MODE == 0 ? f.qs : f.ks, *s2 = MODE == 0 ? p.dos : f.vs;
        ptx::mbar_arrive_expect_tx(bar(BB_OWN), 2 * L::kTile);
#pragma unroll
        for (int pnl = 0; pnl < D / 64; ++pnl) {
          ptx::tma_load_4d(sA + pnl * kPanel, tm_a1, bar(BB_OWN), pnl * 64, row0, s1[1] ? h : 0, s1[0] ? b : 0);
          ptx::tma_load_4d(sA + L::kTile + pnl * kPanel, tm_a2, bar(BB_OWN), pnl * 64, row0, s2[1] ? h : 0, s2[0] ? b : 0);
        }
      }
    }
    __syncwarp();
    constexpr int kPanels = D / 64;
    const int c_of_lane = lane / kPanels, pnl_of_lane = lane % kPanels;
    const bool has_box = c_of_lane < eps;
    const uint32_t slot_bytes = static_cast<uint32_t>(entry_rows) * 128u;
    const uint32_t s_ids = sbase + L::off_ids + static_cast<uint32_t>(warp) * 64u;
    const volatile int* ids_ring = reinterpret_cast<const volatile int*>(smem + L::off_ids + warp * 64);
    // list entries reach a four-step ring in shared memory two steps ahead of their use
    auto fetch_ids = [&](int j) {
      if (lane < eps && j < n_steps) {
        const int e = (j << eps_shift) + lane;
        const int ee = e < total ? e : 0;           // slots past the end re-load the first listed entry
        ptx::cp_async_4(s_ids + static_cast<uint32_t>((j & 3) * 4 + lane) * 4u,
                        ee < n_full ? fids + ee * fstr : pids + (ee - n_full) * pstr);
      }
      ptx::cp_async_commit();
    };
    fetch_ids(0);
    fetch_ids(1);
    bool ok = true, bad = false;
    int issued = 0;
    for (int j = 0; j < n_steps; ++j) {
      fetch_ids(j + 2);
      ptx::cp_async_wait<2>();
      __syncwarp();
      const int st = j & 1;
      const uint32_t full_bar = bar(bar_full + st);
      const bool with_bits = is_x && j >= n_plain;
      uint32_t tx = L::kTile + (MODE == 1 && is_x ? 1024u : 0u);
      if (with_bits) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int e = (j << eps_shift) + (c >> sps_shift);
          tx += (e >= n_full && e < total) ? 512u : 0u;
        }
      }
      if (j >= kStagesB) ok = ptx::mbar_wait(bar(bar_empty + st), ((j >> 1) - 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (lane == 0) ptx::mbar_arrive_expect_tx(full_bar, tx);
      __syncwarp();
      int id = ids_ring[(j & 3) * 4 + (c_of_lane & (eps - 1))];
      if (static_cast<unsigned>(id) >= static_cast<unsigned>(n_entries)) { bad = bad || has_box; id = 0; }
      if (has_box)
        ptx::tma_load_4d(s_tiles + st * L::kTile + pnl_of_lane * kPanel + c_of_lane * slot_bytes, tm, full_bar,
                         pnl_of_lane * 64, id * entry_rows, ch, cb);
      if (is_x && lane < 4) {
        const int e = (j << eps_shift) + (lane >> sps_shift);
        int id_b = ids_ring[(j & 3) * 4 + (lane >> sps_shift)];
        if (static_cast<unsigned>(id_b) >= static_cast<unsigned>(n_entries)) id_b = 0;
        const int64_t group = (static_cast<int64_t>(id_b) << sps_shift) + (lane & ((1 << sps_shift) - 1));
        if (with_bits && e >= n_full && e < total)
          ptx::bulk_load(sbase + L::off_bits + static_cast<uint32_t>(st * 4 + lane) * 512u, words + group * pitch, 512u,
                         full_bar);
        if (MODE == 1) {
          const int64_t at = (static_cast<int64_t>(b) * f.H + h) * f.Sq + static_cast<int64_t>(id_b) * kChunkQ;
          const uint32_t dst = sbase + L::off_stat + static_cast<uint32_t>(st * 2) * 512u + static_cast<uint32_t>(lane) * 128u;
          ptx::bulk_load(dst, a.nlse2 + at, 128u, full_bar);
          ptx::bulk_load(dst + 512u, a.dsum + at, 128u, full_bar);
        }
      }
      __syncwarp();
      issued = j + 1;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0 && f.dev_status != nullptr) atomicMax(f.dev_status, SA_DEV_BAD_INDEX);
    if (!ok && lane == 0) {
      // given up: the copies in flight must have landed before the CTA leaves (bounded, on a flag of its own)
      volatile int* own_flag = reinterpret_cast<volatile int*>(smem + L::off_misc + 8 + 4 * warp);
      *own_flag = 0;
      if (is_x) ptx::mbar_wait_slow(bar(BB_OWN), 0, own_flag, 10000000ull);
      for (int j = issued > kStagesB ? issued - kStagesB : 0; j < issued; ++j)
        ptx::mbar_wait_slow(bar(bar_full + (j & 1)), (j >> 1) & 1, own_flag, 10000000ull);
    }
    __syncwarp();
  } else if (n_steps > 0 && warp == 2) {
    // ------------------------------------------------------------------ MMA issuer (whole warp waits, lane 0 issues)
    constexpr uint32_t idesc_s = ptx::umma_idesc_f16(FmtB<T>::umma, kOwn, kStep, 0);
    constexpr uint32_t idesc_acc = ptx::umma_idesc_f16(FmtB<T>::umma, kOwn, D, 1);
    const uint64_t d0 = ptx::umma_desc_sw128(sA, 16u);
    const uint32_t a1_lo = static_cast<uint32_t>(d0), k_hi = static_cast<uint32_t>(d0 >> 32);
    const uint32_t a2_lo = a1_lo + (L::kTile >> 4);
    const uint32_t x_lo = static_cast<uint32_t>(ptx::umma_desc_sw128(sX, 16u));
    const uint32_t y_lo = static_cast<uint32_t>(ptx::umma_desc_sw128(sY, 16u));
    const uint64_t dx = ptx::umma_desc_sw128(sX, kPanel), dy = ptx::umma_desc_sw128(sY, kPanel);
    const uint32_t xm_lo = static_cast<uint32_t>(dx), ym_lo = static_cast<uint32_t>(dy), m_hi = static_cast<uint32_t>(dx >> 32);
    constexpr uint32_t kStageStep = L::kTile >> 4;
    auto product = [&](uint32_t d_col, uint32_t a_lo, uint32_t b_lo) {      // 128 x 128 over the head dim
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t off = (kk / 4) * (kPanel >> 4) + (kk % 4) * 2u;
        if (kk == 0) ptx::mma_ss_lo<false>(tmem + d_col, a_lo + off, b_lo + off, k_hi, idesc_s);
        else         ptx::mma_ss_lo<true>(tmem + d_col, a_lo + off, b_lo + off, k_hi, idesc_s);
      }
    };
    // 128 x D over the step's 128 rows; the A operand is 16-bit, 32 columns at a_col and 32 at a_col + 64 (each
    // half of the columns is overwritten in place by the threads that read it)
    auto accumulate = [&](uint32_t d_col, uint32_t a_col, uint32_t b_lo, bool first) {
#pragma unroll
      for (int kk = 0; kk < kStep / 16; ++kk) {
        const uint32_t at = tmem + a_col + (kk / 4) * 64u + (kk % 4) * 8u;
        if (kk == 0 && first) ptx::mma_ts_lo<false>(tmem + d_col, at, b_lo + kk * 128u, m_hi, idesc_acc);
        else                  ptx::mma_ts_lo<true>(tmem + d_col, at, b_lo + kk * 128u, m_hi, idesc_acc);
      }
    };
    bool ok = true;
    auto wait = [&](int i, int parity) {
      ok = __all_sync(0xffffffffu, ok && ptx::mbar_wait(bar(i), parity & 1, abort_flag));
      return ok;
    };
    auto issue_s = [&](int j) {
      const int st = j & 1;
      if (!wait(BB_X_FULL + st, j >> 1)) return;
      // Products with different accumulators are not promised to run in the order they are issued: in mode 1 the one
      // that reads P(j - 1) has to be through before these scores overwrite it.
      if (MODE == 1 && j > 0 && !wait(BB_Y_EMPTY + (st ^ 1), (j - 1) >> 1)) return;
      ptx::tc_fence_after();
      if (lane == 0) {
        product(kColS, a1_lo, x_lo + st * kStageStep);
        ptx::mma_commit(bar(BB_S_FULL));
      }
      __syncwarp();
    };
    auto issue_t = [&](int j) {
      const int st = j & 1;
      if (!wait(BB_Y_FULL + st, j >> 1)) return;
      // (dS(j - 1) likewise; mode 0 has two buffers, and dS(j - 2) was read before X(j) could be loaded)
      if (MODE == 1 && j > 0 && !wait(BB_X_EMPTY + (st ^ 1), (j - 1) >> 1)) return;
      ptx::tc_fence_after();
      if (lane == 0) {
        product(MODE == 0 ? kColT + 128u * st : kColT, a2_lo, y_lo + st * kStageStep);
        ptx::mma_commit(bar(BB_T_FULL + st));
        if (MODE == 0) ptx::mma_commit(bar(BB_Y_EMPTY + st));
      }
      __syncwarp();
    };
    wait(BB_OWN, 0);
    if (ok) issue_s(0);
    if (ok) issue_t(0);
    for (int j = 0; j < n_steps && ok; ++j) {
      const int st = j & 1;
      if (!wait(BB_S_DONE, j)) break;
      ptx::tc_fence_after();
      if (MODE == 1) {
        if (lane == 0) {
          accumulate(256u, kColS, ym_lo + st * kStageStep, j == 0);      // dV += P.dO
          ptx::mma_commit(bar(BB_Y_EMPTY + st));
        }
        __syncwarp();
      }
      if (j + 1 < n_steps) issue_s(j + 1);
      if (MODE == 0 && ok && j + 1 < n_steps) issue_t(j + 1);            // into the other T buffer
      if (!ok || !wait(BB_DS_FULL + st, j >> 1)) break;
      ptx::tc_fence_after();
      if (lane == 0) {
        accumulate(384u, MODE == 0 ? kColT + 128u * st : kColT, xm_lo + st * kStageStep, j == 0);   // dQ += dS.K, dK += dS.Q
        ptx::mma_commit(bar(BB_X_EMPTY + st));
        if (j == n_steps - 1) ptx::mma_commit(bar(BB_ACC));
      }
      __syncwarp();
      if (MODE == 1 && j + 1 < n_steps) issue_t(j + 1);
    }
  } else if (warp >= kMathWarp0) {
    // ------------------------------------------------------------------ element-wise work and epilogue
    const int lq = warp & 3, half = (warp - kMathWarp0) >> 2;
    const int row = lq * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(lq * 32) << 16;
    const uint32_t t_s = tmem + lane_off + kColS + 64u * half;
    const uint64_t scale2 = ptx::pack_f32x2(f.scale_log2, f.scale_log2);
    uint64_t nl_own = 0, nd_own = 0;
    if (MODE == 0) {
      const int64_t at = (static_cast<int64_t>(b) * f.H + h) * f.Sq + row0 + row;
      const float nl = a.nlse2[at], nd = -a.dsum[at];
      nl_own = ptx::pack_f32x2(nl, nl);
      nd_own = ptx::pack_f32x2(nd, nd);
    }
    const uint32_t* bits_smem = reinterpret_cast<const uint32_t*>(smem + L::off_bits);
    const float* stat_smem = reinterpret_cast<const float*>(smem + L::off_stat);
    bool live = true;
    for (int j = 0; j < n_steps; ++j) {
      const int st = j & 1;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(bar(BB_S_FULL), j & 1, abort_flag))) { live = false; break; }
      ptx::tc_fence_after();
      uint32_t w[2] = {0xffffffffu, 0xffffffffu};
      if (j >= n_plain) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int ss = half * 2 + c, e = (j << eps_shift) + (ss >> sps_shift);
          const uint32_t word = bits_smem[(st * 4 + ss) * 128 + row];     // stale for a full or padding slot
          w[c] = e < n_full ? 0xffffffffu : (e < total ? word : 0u);
        }
      }
      const float* nl = stat_smem + st * 256 + half * 64;
      float pr[2][32];
      {
        uint32_t s[2][32];
        ptx::tmem_ld32(t_s, s[0]);
        ptx::tmem_ld32(t_s + 32, s[1]);
        ptx::tmem_ld_wait();
        if (MODE == 0) {
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(bar(BB_S_DONE));
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (__all_sync(0xffffffffu, w[c] == 0xffffffffu)) {
            probs<MODE == 1, false>(s[c], w[c], scale2, nl_own, nl + 32 * c, pr[c]);
          } else if (__all_sync(0xffffffffu, w[c] == 0u)) {
#pragma unroll
            for (int i = 0; i < 32; ++i) pr[c][i] = 0.f;
          } else {
            probs<MODE == 1, true>(s[c], w[c], scale2, nl_own, nl + 32 * c, pr[c]);
          }
          if (MODE == 1) {
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[i] = FmtB<T>::pack2(pr[c][2 * i], pr[c][2 * i + 1]);
            ptx::tmem_st16(t_s + 16 * c, pk);
          }
        }
      }
      if (MODE == 1) {
        ptx::tmem_st_wait();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar(BB_S_DONE));
      }
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(bar(BB_T_FULL + st), (j >> 1) & 1, abort_flag))) { live = false; break; }
      ptx::tc_fence_after();
      const uint32_t t_t = tmem + lane_off + kColT + (MODE == 0 ? 128u * st : 0u) + 64u * half;
      const float* ds = nl + 128;
      uint32_t pk[2][16];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t t[32];
        ptx::tmem_ld32(t_t + 32 * c, t);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint64_t n0 = nd_own, n1 = nd_own;
          if (MODE == 1) {
            const float4 v = *reinterpret_cast<const float4*>(ds + 32 * c + 4 * i);
            n0 = ptx::pack_f32x2(-v.x, -v.y);
            n1 = ptx::pack_f32x2(-v.z, -v.w);
          }
          float x[4];
          ptx::unpack_f32x2(ptx::mul_f32x2(ptx::pack_f32x2(pr[c][4 * i], pr[c][4 * i + 1]),
                                           ptx::add_f32x2(ptx::pack_u32x2(t[4 * i], t[4 * i + 1]), n0)), x[0], x[1]);
          ptx::unpack_f32x2(ptx::mul_f32x2(ptx::pack_f32x2(pr[c][4 * i + 2], pr[c][4 * i + 3]),
                                           ptx::add_f32x2(ptx::pack_u32x2(t[4 * i + 2], t[4 * i + 3]), n1)), x[2], x[3]);
          pk[c][2 * i] = FmtB<T>::pack2(x[0], x[1]);
          pk[c][2 * i + 1] = FmtB<T>::pack2(x[2], x[3]);
        }
        // (columns 32.. of this thread's half are still to be read when c = 0: dS goes to the first 32 of its 64)
        ptx::tmem_st16(t_t + 16 * c, pk[c]);
      }
      ptx::tmem_st_wait();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar(BB_DS_FULL + st));
    }
    if (n_steps > 0 && live) {
      live = __all_sync(0xffffffffu, ptx::mbar_wait(bar(BB_ACC), 0, abort_flag));
      ptx::tc_fence_after();
    }
    // this thread's half of a row of an accumulator -> global memory (zeros for an empty walk)
    constexpr int kOC = D / 2;
    auto write_out = [&](uint32_t col, T* base, int64_t row_stride, float factor) {
      uint4* dst = reinterpret_cast<uint4*>(base + static_cast<int64_t>(row) * row_stride + kOC * half);
#pragma unroll
      for (int c = 0; c < kOC / 32; ++c) {
        uint32_t r[32];
        if (n_steps > 0) {
          ptx::tmem_ld32(tmem + lane_off + col + kOC * half + 32 * c, r);
          ptx::tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
        if (MODE == 0 || row0 + row < f.Sk) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            auto v = [&](int k) { return __uint_as_float(r[8 * i + k]) * factor; };
            dst[4 * c + i] = make_uint4(FmtB<T>::pack2(v(0), v(1)), FmtB<T>::pack2(v(2), v(3)),
                                        FmtB<T>::pack2(v(4), v(5)), FmtB<T>::pack2(v(6), v(7)));
          }
        }
      }
    };
    if (live) {
      const float scale = f.scale_log2 * kLn2;
      if (MODE == 0) {
        write_out(384u, static_cast<T*>(p.dq) + b * p.dqs[0] + h * p.dqs[1] + static_cast<int64_t>(row0) * p.dqs[2],
                  p.dqs[2], scale);
      } else {
        write_out(256u, static_cast<T*>(p.dv) + b * p.dvs[0] + h * p.dvs[1] + static_cast<int64_t>(row0) * p.dvs[2],
                  p.dvs[2], 1.f);
        write_out(384u, static_cast<T*>(p.dk) + b * p.dks[0] + h * p.dks[1] + static_cast<int64_t>(row0) * p.dks[2],
                  p.dks[2], scale);
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_dealloc(tmem, 512u);
  }
  if (threadIdx.x == 0 && *abort_flag != 0 && f.dev_status != nullptr) atomicMax(f.dev_status, SA_DEV_WAIT_EXPIRED);
}

struct BwdMaps {
  CUtensorMap q_own, do_own, k_own, v_own;         // boxes of 128 rows
  CUtensorMap q_str, do_str, k_str, v_str;         // boxes of 32 query rows / BLOCK_K kv rows
};

// Both modes in one launch, the longer steps (dK, dV) first: one tail instead of two.
template <typename T, int D>
__global__ void __launch_bounds__(kThreadsB, 1)
attn_bwd_tc_kernel(const __grid_constant__ BwdArgs a, const __grid_constant__ BwdMaps m, const int n_kv_tiles) {
  if (static_cast<int>(blockIdx.x) < n_kv_tiles)
    bwd_body<T, D, 1>(a, &m.k_own, &m.v_own, &m.q_str, &m.do_str, static_cast<int>(blockIdx.x));
  else
    bwd_body<T, D, 0>(a, &m.q_own, &m.do_own, &m.k_str, &m.v_str, static_cast<int>(blockIdx.x) - n_kv_tiles);
}

// D_i = sum_d dO_id O_id (- d_lse_i) and -lse_i in base 2: D / 8 lanes per row, 16 bytes each.
template <typename T, int D>
__global__ void __launch_bounds__(256)
bwd_row_stats_kernel(const AttnBwdParams p, float* __restrict__ nlse2, float* __restrict__ dsum) {
  const AttnParams& f = p.fwd;
  constexpr int kLanes = D / 8;
  const int64_t row = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) / kLanes;
  const int part = threadIdx.x % kLanes;
  const int64_t rows = static_cast<int64_t>(f.B) * f.H * f.Sq;
  float acc = 0.f;
  if (row < rows) {
    const int s = static_cast<int>(row % f.Sq);
    const int bh = static_cast<int>(row / f.Sq);
    const int b = bh / f.H, h = bh - b * f.H;
    const T* o = static_cast<const T*>(f.o) + b * f.os[0] + h * f.os[1] + s * f.os[2] + part * 8;
    const T* g = static_cast<const T*>(p.d_o) + b * p.dos[0] + h * p.dos[1] + s * p.dos[2] + part * 8;
    const uint4 ov = *reinterpret_cast<const uint4*>(o), gv = *reinterpret_cast<const uint4*>(g);
    const T* oe = reinterpret_cast<const T*>(&ov);
    const T* ge = reinterpret_cast<const T*>(&gv);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc = fmaf(FmtB<T>::up(ge[i]), FmtB<T>::up(oe[i]), acc);
  }
#pragma unroll
  for (int s = kLanes / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (row < rows && part == 0) {
    if (p.d_lse != nullptr) acc -= p.d_lse[row];
    dsum[row] = acc;
    const float lse = f.lse[row];
    nlse2[row] = lse == -INFINITY ? -INFINITY : -lse * kLog2e;
  }
}

// The walk of mode 1, first half.  One CTA per (plane, query block of 128 rows): the block's two lists become a
// class per kv block in shared memory; per (128 kv rows, 32-row query chunk) a warp looks at the 4 x 32 mask words
// (all ones for a listed full block, zero for one that is not listed), writes the class of the 32 x 128 tile and,
// for a mixed one, its words transposed (bit = query row, word = kv row).
struct BwdPlan {
  const int32_t *full_ids, *full_lens, *part_ids, *part_lens;
  int64_t fis[4], fls[3], pis[4], pls[3];
  const uint32_t* bits;
  int64_t bits_sb, bits_sh;
  int P1;                        // planes = P0 * P1; plane = p0 * P1 + p1
  int Sq, Sk, BK, sk_pad;
  uint8_t* cls;                  // [planes, kv tiles, Sq / 32]: 0 nothing, 1 some, 2 every element attended
  uint32_t* t_bits;
  int32_t* t_ids;
  int32_t* t_lens;
};

__device__ __forceinline__ uint32_t transpose_32(uint32_t x, int lane) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const uint32_t m = s == 16 ? 0x0000ffffu : s == 8 ? 0x00ff00ffu : s == 4 ? 0x0f0f0f0fu : s == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    x = (lane & s) ? ((x & ~m) | ((y >> s) & m)) : ((x & m) | ((y & m) << s));
  }
  return x;
}

__global__ void __launch_bounds__(256)
bwd_classify_kernel(const BwdPlan a) {
  extern __shared__ uint8_t s_cls[];               // [Sk / BK]
  const int nq = a.Sq / 128, nk = a.Sk / a.BK, n_chunks = a.Sq / kChunkQ, kv_tiles = a.sk_pad / kOwn;
  const int plane = blockIdx.x / nq, qb = blockIdx.x - plane * nq;
  const int p0 = plane / a.P1, p1 = plane - p0 * a.P1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int t = threadIdx.x; t < nk; t += 256) s_cls[t] = 0;
  __syncthreads();
  const int32_t* fids = a.full_ids + p0 * a.fis[0] + p1 * a.fis[1] + qb * a.fis[2];
  const int32_t* pids = a.part_ids + p0 * a.pis[0] + p1 * a.pis[1] + qb * a.pis[2];
  const int nf = min(max(a.full_lens[p0 * a.fls[0] + p1 * a.fls[1] + qb * a.fls[2]], 0), nk);
  const int np = min(max(a.part_lens[p0 * a.pls[0] + p1 * a.pls[1] + qb * a.pls[2]], 0), nk);
  for (int t = threadIdx.x; t < nf; t += 256) {
    const int id = fids[t * a.fis[3]];
    if (static_cast<unsigned>(id) < static_cast<unsigned>(nk)) s_cls[id] = 2;
  }
  for (int t = threadIdx.x; t < np; t += 256) {
    const int id = pids[t * a.pis[3]];
    if (static_cast<unsigned>(id) < static_cast<unsigned>(nk)) s_cls[id] = 1;
  }
  __syncthreads();
  const uint32_t* bits = a.bits + p0 * a.bits_sb + p1 * a.bits_sh + qb * 128 + lane;
  for (int kt = warp; kt < kv_tiles; kt += 8) {
    uint32_t w[4][4];                              // [chunk][32-column group]
    bool inside = true;                            // no kv row of the tile lies past the end
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int col = kt * 128 + g * 32;
      const int cl = col < a.Sk ? s_cls[col / a.BK] : 0;
      inside = inside && col < a.Sk;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        w[c][g] = cl == 1 ? bits[static_cast<int64_t>(col >> 5) * a.Sq + c * 32] : cl == 2 ? 0xffffffffu : 0u;
    }
    uint32_t packed = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const bool any = __any_sync(0xffffffffu, (w[c][0] | w[c][1] | w[c][2] | w[c][3]) != 0u);
      const bool all = __all_sync(0xffffffffu, (w[c][0] & w[c][1] & w[c][2] & w[c][3]) == 0xffffffffu) && inside;
      packed |= (all ? 2u : any ? 1u : 0u) << (8 * c);
      if (any && !all) {
        uint32_t* dst = a.t_bits + (static_cast<int64_t>(plane) * n_chunks + qb * 4 + c) * a.sk_pad + kt * 128 + lane;
#pragma unroll
        for (int g = 0; g < 4; ++g) dst[g * 32] = transpose_32(w[c][g], lane);
      }
    }
    if (lane == 0)
      *reinterpret_cast<uint32_t*>(a.cls + (static_cast<int64_t>(plane) * kv_tiles + kt) * n_chunks + qb * 4) = packed;
  }
}

// Second half: a warp per (plane, kv tile) packs the listed chunks, the plain ones ascending from the front of the
// row, the mixed ones ascending from its end backwards.
__global__ void __launch_bounds__(256)
bwd_lists_kernel(const BwdPlan a, const int rows) {
  const int row = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int n_chunks = a.Sq / kChunkQ;
  const uint8_t* cls = a.cls + static_cast<int64_t>(row) * n_chunks;
  int32_t* ids = a.t_ids + static_cast<int64_t>(row) * n_chunks;
  const uint32_t below = (1u << lane) - 1u;
  int nf = 0, np = 0;
  for (int c0 = 0; c0 < n_chunks; c0 += 32) {
    const int c = c0 + lane;
    const int cl = c < n_chunks ? cls[c] : 0;
    const uint32_t bf = __ballot_sync(0xffffffffu, cl == 2), bp = __ballot_sync(0xffffffffu, cl == 1);
    if (cl == 2) ids[nf + __popc(bf & below)] = c;
    if (cl == 1) ids[n_chunks - 1 - (np + __popc(bp & below))] = c;
    nf += __popc(bf);
    np += __popc(bp);
  }
  if (lane == 0) {
    a.t_lens[2 * row] = nf;
    a.t_lens[2 * row + 1] = np;
  }
}

struct BwdLayout {
  size_t nlse2, dsum, cls, ids, lens, bits, total;
};
BwdLayout bwd_layout(int B, int H, int planes, int Sq, int Sk) {
  const size_t kv_tiles = (static_cast<size_t>(Sk) + kOwn - 1) / kOwn, chunks = static_cast<size_t>(Sq) / kChunkQ;
  const size_t rows = static_cast<size_t>(B) * H * Sq, cells = static_cast<size_t>(planes) * kv_tiles * chunks;
  auto up = [](size_t x) { return (x + 255) & ~static_cast<size_t>(255); };
  BwdLayout l;
  l.nlse2 = 0;
  l.dsum = l.nlse2 + up(4 * rows);
  l.cls = l.dsum + up(4 * rows);
  l.ids = l.cls + up(cells);
  l.lens = l.ids + up(4 * cells);
  l.bits = l.lens + up(8 * static_cast<size_t>(planes) * kv_tiles);
  l.total = l.bits + up(4 * static_cast<size_t>(planes) * chunks * kv_tiles * kOwn);
  return l;
}

template <typename T, int D>
int launch_bwd(const BwdArgs& a, const BwdMaps& m, float* nlse2, float* dsum, int sm_ordinal, cudaStream_t stream) {
  const AttnParams& f = a.p.fwd;
  auto kernel = attn_bwd_tc_kernel<T, D>;
  static std::once_flag once[kMaxDevices];
  static cudaError_t attr[kMaxDevices];
  std::call_once(once[sm_ordinal], [&] {
    attr[sm_ordinal] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(SmemB<D>::dynamic_bytes));
  });
  if (attr[sm_ordinal] != cudaSuccess) return SA_ERR_CUDA;
  const int64_t stat_threads = static_cast<int64_t>(f.B) * f.H * f.Sq * (D / 8);
  bwd_row_stats_kernel<T, D><<<static_cast<unsigned>((stat_threads + 255) / 256), 256, 0, stream>>>(a.p, nlse2, dsum);
  const int n_kv = f.B * f.H * (a.sk_pad / kOwn), n_q = f.B * f.H * (f.Sq / kOwn);
  kernel<<<static_cast<unsigned>(n_kv + n_q), kThreadsB, SmemB<D>::dynamic_bytes, stream>>>(a, m, n_kv);
  return cudaGetLastError() == cudaSuccess ? SA_OK : SA_ERR_CUDA;
}

}  // namespace

size_t attn_bwd_tc_workspace_bytes(int B, int H, int planes, int Sq, int Sk) { return bwd_layout(B, H, planes, Sq, Sk).total; }

int attn_bwd_tc_supported(const AttnBwdParams& p) {
  const AttnParams& f = p.fwd;
  if (f.dtype != SA_DTYPE_F16 && f.dtype != SA_DTYPE_BF16) return 0;
  if (f.D != 64 && f.D != 128) return 0;
  if (f.BQ != kOwn || (f.BK != 32 && f.BK != 64 && f.BK != 128)) return 0;
  if (f.Sq % kOwn != 0 || f.Sk % f.BK != 0 || f.Sk / f.BK > 40 * 1024) return 0;      // classes in 48 KB of shared memory
  if (f.bits == nullptr || reinterpret_cast<uintptr_t>(f.bits) % 16 != 0 || f.bits_sb % 4 != 0 || f.bits_sh % 4 != 0) return 0;
  if (!(f.scale_log2 > 0.f) || !(f.scale_log2 < 1e30f)) return 0;
  auto rows_ok = [](const void* base, const int64_t* st) {
    return reinterpret_cast<uintptr_t>(base) % 16 == 0 && st[3] == 1 && st[2] % 8 == 0 && st[1] % 8 == 0 && st[0] % 8 == 0;
  };
  if (!tma_friendly(f.q, f.qs) || !tma_friendly(f.k, f.ks) || !tma_friendly(f.v, f.vs) || !tma_friendly(p.d_o, p.dos)) return 0;
  if (!rows_ok(f.o, f.os) || !rows_ok(p.dq, p.dqs) || !rows_ok(p.dk, p.dks) || !rows_ok(p.dv, p.dvs)) return 0;
  const long long bh = static_cast<long long>(f.B) * f.H;
  if (bh * (f.Sq / kOwn + f.Sk / kOwn + 1) > 0x7fffffffLL || bh * f.Sq * (f.D / 8) / 256 > 0x7ffffffeLL) return 0;
  return 1;
}

int launch_attn_bwd_tc(const AttnBwdParams& p, int P0, int P1, void* workspace, cudaStream_t stream) {
  const AttnParams& f = p.fwd;
  const DeviceInfo* info = current_device_info();
  if (info == nullptr) return SA_ERR_NO_DEVICE;
  const int planes = P0 * P1;
  const BwdLayout l = bwd_layout(f.B, f.H, planes, f.Sq, f.Sk);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  BwdArgs a;
  a.p = p;
  a.nlse2 = reinterpret_cast<float*>(ws + l.nlse2);
  a.dsum = reinterpret_cast<float*>(ws + l.dsum);
  a.t_ids = reinterpret_cast<int32_t*>(ws + l.ids);
  a.t_lens = reinterpret_cast<int32_t*>(ws + l.lens);
  a.t_bits = reinterpret_cast<uint32_t*>(ws + l.bits);
  a.plane_b = P0 > 1 ? P1 : 0;
  a.plane_h = P1 > 1 ? 1 : 0;
  a.sk_pad = (f.Sk + kOwn - 1) / kOwn * kOwn;

  BwdMaps m;
  if (!make_map(&m.q_own, f.q, f.dtype, f.B, f.H, f.Sq, f.D, f.qs, kOwn) ||
      !make_map(&m.do_own, p.d_o, f.dtype, f.B, f.H, f.Sq, f.D, p.dos, kOwn) ||
      !make_map(&m.k_own, f.k, f.dtype, f.B, f.H, f.Sk, f.D, f.ks, kOwn) ||
      !make_map(&m.v_own, f.v, f.dtype, f.B, f.H, f.Sk, f.D, f.vs, kOwn) ||
      !make_map(&m.q_str, f.q, f.dtype, f.B, f.H, f.Sq, f.D, f.qs, kChunkQ) ||
      !make_map(&m.do_str, p.d_o, f.dtype, f.B, f.H, f.Sq, f.D, p.dos, kChunkQ) ||
      !make_map(&m.k_str, f.k, f.dtype, f.B, f.H, f.Sk, f.D, f.ks, f.BK) ||
      !make_map(&m.v_str, f.v, f.dtype, f.B, f.H, f.Sk, f.D, f.vs, f.BK))
    return SA_ERR_CUDA;

  BwdPlan pl;
  pl.full_ids = f.full_ids; pl.full_lens = f.full_lens; pl.part_ids = f.part_ids; pl.part_lens = f.part_lens;
  for (int i = 0; i < 4; ++i) { pl.fis[i] = f.fis[i]; pl.pis[i] = f.pis[i]; }
  for (int i = 0; i < 3; ++i) { pl.fls[i] = f.fls[i]; pl.pls[i] = f.pls[i]; }
  pl.bits = f.bits; pl.bits_sb = f.bits_sb; pl.bits_sh = f.bits_sh;
  pl.P1 = P1;
  pl.Sq = f.Sq; pl.Sk = f.Sk; pl.BK = f.BK; pl.sk_pad = a.sk_pad;
  pl.cls = ws + l.cls;
  pl.t_bits = reinterpret_cast<uint32_t*>(ws + l.bits);
  pl.t_ids = reinterpret_cast<int32_t*>(ws + l.ids);
  pl.t_lens = reinterpret_cast<int32_t*>(ws + l.lens);
  const int rows = planes * (a.sk_pad / kOwn);
  bwd_classify_kernel<<<static_cast<unsigned>(planes * (f.Sq / kOwn)), 256, static_cast<size_t>(f.Sk / f.BK), stream>>>(pl);
  bwd_lists_kernel<<<static_cast<unsigned>((static_cast<int64_t>(rows) * 32 + 255) / 256), 256, 0, stream>>>(pl, rows);
  if (cudaGetLastError() != cudaSuccess) return SA_ERR_CUDA;

  float* nlse2 = reinterpret_cast<float*>(ws + l.nlse2);
  float* dsum = reinterpret_cast<float*>(ws + l.dsum);
  if (f.dtype == SA_DTYPE_BF16)
    return f.D == 128 ? launch_bwd<__nv_bfloat16, 128>(a, m, nlse2, dsum, info->ordinal, stream)
                      : launch_bwd<__nv_bfloat16, 64>(a, m, nlse2, dsum, info->ordinal, stream);
  return f.D == 128 ? launch_bwd<__half, 128>(a, m, nlse2, dsum, info->ordinal, stream)
                    : launch_bwd<__half, 64>(a, m, nlse2, dsum, info->ordinal, stream);
}

}  // namespace sa
