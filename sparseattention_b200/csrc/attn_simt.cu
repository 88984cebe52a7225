// Stage 2, generic kernel: block-sparse attention forward on the CUDA cores.
//
// Same algorithm as sparseattention/sparse_attn_kernel.py:72-146 (+ inner loop 10-63):
// per query block, loop A over the full list without the mask, loop B over the partial
// list with the boolean mask applied as -inf, online softmax in base 2 with fp32 running
// max / sum / accumulator, P rounded to the V dtype before P.V (line 61), O = acc / l.
// It takes any dtype (fp32 / fp16 / bf16), any strides (0 included), head dims 16, 32, 64
// and 128 and block sizes that are multiples of 32, reads the byte mask
// directly, and is the path for shapes the tcgen05 kernel does not cover.  Rows without
// any attended key come out as 0.
//
// Work split: a CTA owns 32 query rows of one (batch, head).  Its kGroups groups of 128 threads walk the lists in
// chunks of 64 kv rows, group g taking chunks g, g + kGroups, ...; each keeps its own running max, sum and
// accumulator, and they are combined at the end, so that a call with few query rows still has 8 to 16 warps
// per SM.  Within a group a thread forms 4 rows x 4 columns of the scores and 4 rows x D / 16 columns of the
// output in registers: per four steps of the inner dimension 8 (D = 128: 12 in P.V) 16-byte shared-memory loads
// feed 64 (128) FMAs.  That is the bound on a full chip: a 16-byte load returns 512 bytes to a warp at 128 B a
// cycle, so the loads take twice the cycles of the FMAs they feed.  K of the next chunk travels while P.V of this one runs, V while
// the scores are formed (cp.async for 16-byte aligned fp32 rows, plain loads and a conversion otherwise).
// Measured (kernel alone, one B200, fp32, 32 x 32 blocks dropped with p = 0.5, lists at (128, 32); before: a quad of
// threads per row, one scalar load per FMA): B=1 H=4 S=512 D=64 100 -> 35 us (64 CTAs: latency), D=128 168 -> 59 us;
// B=2 H=16 S=2048 D=64 2.68 -> 1.29 ms (25 TFLOP/s), D=128 5.34 -> 2.46 ms.  Error against float64: 3.3e-7 both.
// The 16-bit types, which are converted on the way to shared memory, gain less: B=2 H=16 S=2048, p = 0.7, lists at
// (64, 64), bf16 D=64 2.22 -> 1.39 ms, D=128 4.46 -> 3.19 (fp32 2.23 -> 1.10, 4.50 -> 2.04); rows that are not dense
// (D=128 fp32) 6.85 -> 4.91.  At D 16 to 64 the 512 threads of a CTA have 128 registers each and 12 to 68 bytes of a
// thread's state are spilled (D = 128: 150 to 174 registers, none).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <mutex>
#include <type_traits>

#include "ptx_sm100.cuh"
#include "sa_common.cuh"

namespace sa {
namespace {

constexpr int kRows = 32;       // query rows per CTA
constexpr int kKeys = 64;       // kv rows per chunk: two units of 32, each from one listed block
constexpr int kGroupThreads = 128;

template <int D>
struct SimtSmem {
  static constexpr int kGroups = D == 128 ? 2 : 4;
  static constexpr int kLdK = D + 4, kLdP = kKeys + 4;       // 16 bytes of padding: 8 lanes reading 8 rows hit 8 bank groups
  static constexpr int q = 0;                                // floats
  static constexpr int group0 = kRows * kLdK;
  static constexpr int k = 0, v = kKeys * kLdK, pr = v + kKeys * D;      // within a group
  static constexpr int group_floats = pr + kRows * kLdP;
  static constexpr size_t bytes = sizeof(float) * (group0 + static_cast<size_t>(kGroups) * group_floats);
  // the end of the walk: a group's row max, row sum, weight and accumulator lie over its K and V
  static_assert(3 * kRows + kRows * kLdK <= v + kKeys * D, "combine area");
};

template <typename T> __device__ __forceinline__ float to_f32(T x);
template <> __device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

__device__ __forceinline__ void simt_cp_async_16(float* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_u32(dst)), "l"(src) : "memory");
}

template <typename T, int D>
__global__ void __launch_bounds__(SimtSmem<D>::kGroups * kGroupThreads)
attn_simt_kernel(const AttnParams p, const int vec) {
  using L = SimtSmem<D>;
  constexpr int kGroups = L::kGroups, kLdK = L::kLdK, kLdP = L::kLdP;
  constexpr int kOC = D / 16;                            // output columns per thread
  extern __shared__ __align__(16) float simt_smem[];

  const int tid = threadIdx.x % kGroupThreads, group = threadIdx.x / kGroupThreads;
  const int cg = tid & 15, rg = tid >> 4;                // 16 column groups, 8 row groups of 4 rows
  float* Qs = simt_smem + L::q;
  float* Ks = simt_smem + L::group0 + group * L::group_floats + L::k;
  float* Vs = Ks + L::v;
  float* Ps = Ks + L::pr;

  const int row_groups = p.Sq / kRows;                   // 1-D grid: (batch * head, group of 32 query rows)
  const int row0 = static_cast<int>(blockIdx.x % row_groups) * kRows;
  const int bh = static_cast<int>(blockIdx.x / row_groups);
  const int b = bh / p.H, h = bh % p.H;
  const int qblk = row0 / p.BQ;
  const int nk = p.Sk / p.BK;
  const int units = p.BK / 32;                           // units per listed block

  const T* q = static_cast<const T*>(p.q) + b * p.qs[0] + h * p.qs[1] + static_cast<int64_t>(row0) * p.qs[2];
  const T* kbase = static_cast<const T*>(p.k) + b * p.ks[0] + h * p.ks[1];
  const T* vbase = static_cast<const T*>(p.v) + b * p.vs[0] + h * p.vs[1];
  const uint8_t* mrows = p.mask + b * p.ms[0] + h * p.ms[1] + static_cast<int64_t>(row0 + 4 * rg) * p.ms[2];

  const int32_t* fids = p.full_ids + b * p.fis[0] + h * p.fis[1] + static_cast<int64_t>(qblk) * p.fis[2];
  const int32_t* pids = p.part_ids + b * p.pis[0] + h * p.pis[1] + static_cast<int64_t>(qblk) * p.pis[2];
  // A caller-supplied length outside [0, nk] would walk the id list out of bounds: it is clamped
  // (as the tensor-core kernel does) and reported.
  const int nf_given = p.full_lens[b * p.fls[0] + h * p.fls[1] + static_cast<int64_t>(qblk) * p.fls[2]];   // line 107
  const int np_given = p.part_lens[b * p.pls[0] + h * p.pls[1] + static_cast<int64_t>(qblk) * p.pls[2]];   // line 127
  const int nf = min(max(nf_given, 0), nk), np = min(max(np_given, 0), nk);
  if ((nf != nf_given || np != np_given) && threadIdx.x == 0 && p.dev_status != nullptr)
    atomicMax(p.dev_status, SA_DEV_BAD_INDEX);
  const int total_units = (nf + np) * units;
  const int n_chunks = (total_units + 1) / 2;

  // unit u of the walk (full list first, then the partial one): the id of its block, asked for one chunk before it
  // is looked at
  auto fetch = [&](int u) -> int {
    if (u >= total_units) return -1;
    const int e = u / units;
    return e >= nf ? pids[(e - nf) * p.pis[3]] : fids[e * p.fis[3]];                        // line 33
  };
  // its first kv row, -1 for none
  auto unit_row = [&](int u, int id, bool& masked) -> int {
    masked = u / units >= nf;
    if (u >= total_units) return -1;
    if (id < 0 || id >= nk) {
      if (tid == 0 && p.dev_status != nullptr) atomicMax(p.dev_status, SA_DEV_BAD_INDEX);
      return -1;
    }
    return id * p.BK + (u % units) * 32;
  };
  // 32 rows of one unit -> dst (row pitch ld); zeros for a unit that does not exist (0 * P must stay 0)
  auto load_unit = [&](float* dst, int ld, const T* base, const int64_t* st, int kv0) {
    if (kv0 < 0) {
      for (int e = tid; e < 32 * D; e += kGroupThreads) dst[(e / D) * ld + e % D] = 0.f;
    } else if (std::is_same<T, float>::value && vec) {
      for (int e = tid; e < 32 * (D / 4); e += kGroupThreads) {
        const int c = e / (D / 4), d4 = e % (D / 4);
        simt_cp_async_16(dst + c * ld + 4 * d4, base + static_cast<int64_t>(kv0 + c) * st[2] + 4 * d4);
      }
    } else {
      for (int e = tid; e < 32 * D; e += kGroupThreads) {
        const int c = e / D, d = e % D;
        dst[c * ld + d] = to_f32<T>(base[static_cast<int64_t>(kv0 + c) * st[2] + d * st[3]]);
      }
    }
  };
  auto group_sync = [&] { ptx::named_bar_sync(1 + group, kGroupThreads); };

  int id[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) id[x] = fetch(2 * group + x);
  if (std::is_same<T, float>::value && vec) {                                               // lines 98-101
    for (int e = threadIdx.x; e < kRows * (D / 4); e += kGroups * kGroupThreads)
      simt_cp_async_16(Qs + (e / (D / 4)) * kLdK + 4 * (e % (D / 4)), q + static_cast<int64_t>(e / (D / 4)) * p.qs[2] + 4 * (e % (D / 4)));
  } else {
    for (int e = threadIdx.x; e < kRows * D; e += kGroups * kGroupThreads)
      Qs[(e / D) * kLdK + e % D] = to_f32<T>(q[static_cast<int64_t>(e / D) * p.qs[2] + (e % D) * p.qs[3]]);
  }

  float acc[4][kOC], m[4], l[4];                         // l: this thread's columns only
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY; l[i] = 0.f;                        // lines 103-104
#pragma unroll
    for (int j = 0; j < kOC; ++j) acc[i][j] = 0.f;       // line 105
  }

  int kv_row[2];
  bool masked[2];
  auto locate = [&](int chunk) {
#pragma unroll
    for (int x = 0; x < 2; ++x) kv_row[x] = unit_row(2 * chunk + x, id[x], masked[x]);
  };
  if (group < n_chunks) {
    locate(group);
#pragma unroll
    for (int x = 0; x < 2; ++x) load_unit(Ks + 32 * x * kLdK, kLdK, kbase, p.ks, kv_row[x]);
  }
  ptx::cp_async_commit();
  ptx::cp_async_wait<0>();
  __syncthreads();                                       // Q is in place
#pragma unroll 1
  for (int chunk = group; chunk < n_chunks; chunk += kGroups) {
    ptx::cp_async_wait<0>();
    group_sync();                                        // K has landed, everyone is done with the previous V
#pragma unroll
    for (int x = 0; x < 2; ++x) load_unit(Vs + 32 * x * D, D, vbase, p.vs, kv_row[x]);
    ptx::cp_async_commit();
#pragma unroll
    for (int x = 0; x < 2; ++x) id[x] = fetch(2 * (chunk + kGroups) + x);
    // attended columns of this thread, bit 4 i + x: row 4 rg + i, key cg + 16 x (a bit field: the loads fly over Q.K)
    uint32_t attend = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int kv0 = kv_row[x >> 1];
        bool on = kv0 >= 0;
        if (on && masked[x >> 1])                                                           // line 47
          on = mrows[i * p.ms[2] + static_cast<int64_t>(kv0 + cg + 16 * (x & 1)) * p.ms[3]] != 0;
        attend |= (on ? 1u : 0u) << (4 * i + x);
      }

    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int x = 0; x < 4; ++x) s[i][x] = 0.f;
#pragma unroll 2
    for (int d = 0; d < D; d += 4) {                                                        // line 40
      float4 a[4], kk[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(Qs + (4 * rg + i) * kLdK + d);
#pragma unroll
      for (int x = 0; x < 4; ++x) kk[x] = *reinterpret_cast<const float4*>(Ks + (cg + 16 * x) * kLdK + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          s[i][x] = fmaf(a[i].x, kk[x].x, s[i][x]);
          s[i][x] = fmaf(a[i].y, kk[x].y, s[i][x]);
          s[i][x] = fmaf(a[i].z, kk[x].z, s[i][x]);
          s[i][x] = fmaf(a[i].w, kk[x].w, s[i][x]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float top = -INFINITY;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        s[i][x] = (attend >> (4 * i + x)) & 1u ? s[i][x] * p.scale_log2 : -INFINITY;        // lines 47 / 51
        top = fmaxf(top, s[i][x]);
      }
#pragma unroll
      for (int w = 1; w < 16; w <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
      const float m_new = fmaxf(m[i], top);                                                 // lines 48 / 50
      const float ref = (m_new == -INFINITY) ? 0.f : m_new;        // guard the reference lacks (line 53)
      const float alpha = (m[i] == -INFINITY) ? 1.f : exp2f(m[i] - ref);                    // line 55
      float sum = 0.f;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float pe = exp2f(s[i][x] - ref);                                              // line 54
        sum += pe;
        Ps[(4 * rg + i) * kLdP + cg + 16 * x] = to_f32<T>(from_f32<T>(pe));                 // line 61 cast
      }
      l[i] = l[i] * alpha + sum;                                                            // line 57
      m[i] = m_new;                                                                         // line 56
#pragma unroll
      for (int j = 0; j < kOC; ++j) acc[i][j] *= alpha;                                     // line 58
    }
    ptx::cp_async_wait<0>();
    group_sync();                                        // V has landed, everyone is done with K (and P is written)
    if (chunk + kGroups < n_chunks) {
      locate(chunk + kGroups);
#pragma unroll
      for (int x = 0; x < 2; ++x) load_unit(Ks + 32 * x * kLdK, kLdK, kbase, p.ks, kv_row[x]);
      ptx::cp_async_commit();
    }
#pragma unroll 2
    for (int c = 0; c < kKeys; c += 4) {                                                    // line 61
      float4 pr[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) pr[i] = *reinterpret_cast<const float4*>(Ps + (4 * rg + i) * kLdP + c);
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        float vv[kOC];
        if constexpr (kOC >= 4) {
#pragma unroll
          for (int j = 0; j < kOC / 4; ++j)
            *reinterpret_cast<float4*>(vv + 4 * j) = *reinterpret_cast<const float4*>(Vs + (c + y) * D + 64 * j + 4 * cg);
        } else {
#pragma unroll
          for (int j = 0; j < kOC; ++j) vv[j] = Vs[(c + y) * D + kOC * cg + j];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float pe = y == 0 ? pr[i].x : y == 1 ? pr[i].y : y == 2 ? pr[i].z : pr[i].w;
#pragma unroll
          for (int j = 0; j < kOC; ++j) acc[i][j] = fmaf(pe, vv[j], acc[i][j]);
        }
      }
    }
  }

#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int w = 1; w < 16; w <<= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], w);
  // the groups' results meet in shared memory, over their K and V
  __syncthreads();
  float* mine = Ks;
  constexpr int kAcc0 = 3 * kRows;                       // max, sum, weight, then the accumulator (row pitch kLdK)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 4 * rg + i;
    if (cg == 0) { mine[r] = m[i]; mine[kRows + r] = l[i]; }
#pragma unroll
    for (int j = 0; j < kOC; ++j) {
      const int col = kOC >= 4 ? 64 * (j / 4) + 4 * cg + (j & 3) : kOC * cg + j;
      mine[kAcc0 + r * kLdK + col] = acc[i][j];
    }
  }
  __syncthreads();
  float* all = simt_smem + L::group0;
  if (threadIdx.x < kRows) {
    const int r = threadIdx.x;
    float top = -INFINITY, sum = 0.f, w[kGroups];
#pragma unroll
    for (int g = 0; g < kGroups; ++g) top = fmaxf(top, all[g * L::group_floats + r]);
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      const float mg = all[g * L::group_floats + r];
      w[g] = mg == -INFINITY ? 0.f : exp2f(mg - top);
      sum = fmaf(w[g], all[g * L::group_floats + kRows + r], sum);
    }
    const float inv = sum > 0.f ? 1.f / sum : 0.f;                                          // line 144
#pragma unroll
    for (int g = 0; g < kGroups; ++g) all[g * L::group_floats + 2 * kRows + r] = w[g] * inv;
    if (p.lse != nullptr)                          // m and l are in base 2 (scale folded, line 152)
      p.lse[(static_cast<int64_t>(b) * p.H + h) * p.Sq + row0 + r] =
          sum > 0.f ? (top + log2f(sum)) * 0.6931471805599453f : -INFINITY;
  }
  __syncthreads();
  T* o = static_cast<T*>(p.o) + b * p.os[0] + h * p.os[1] + static_cast<int64_t>(row0) * p.os[2];
  for (int e = threadIdx.x; e < kRows * D; e += kGroups * kGroupThreads) {
    const int r = e / D, col = e % D;
    float x = 0.f;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      const float* from = all + g * L::group_floats;
      x = fmaf(from[2 * kRows + r], from[kAcc0 + r * kLdK + col], x);
    }
    o[static_cast<int64_t>(r) * p.os[2] + static_cast<int64_t>(col) * p.os[3]] = from_f32<T>(x);   // line 146
  }
}

template <typename T, int D>
cudaError_t launch_simt_inst(const AttnParams& p, int vec, unsigned ctas, cudaStream_t stream) {
  using L = SimtSmem<D>;
  const DeviceInfo* info = current_device_info();
  if (info == nullptr) return cudaErrorInvalidDevice;
  static std::once_flag once[kMaxDevices];
  static cudaError_t attr[kMaxDevices];
  std::call_once(once[info->ordinal], [&] {
    attr[info->ordinal] = cudaFuncSetAttribute(attn_simt_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(L::bytes));
  });
  if (attr[info->ordinal] != cudaSuccess) return attr[info->ordinal];
  attn_simt_kernel<T, D><<<ctas, L::kGroups * kGroupThreads, L::bytes, stream>>>(p, vec);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_for_dtype(const AttnParams& p, cudaStream_t stream) {
  const long long ctas = static_cast<long long>(p.Sq / kRows) * p.B * p.H;
  if (ctas <= 0 || ctas > 0x7fffffffLL) return cudaErrorInvalidValue;
  const unsigned grid = static_cast<unsigned>(ctas);
  // 16-byte copies of Q, K and V rows (fp32): aligned bases, unit stride along d, the other strides multiples of four
  auto rows_ok = [](const void* base, const int64_t* st) {
    return reinterpret_cast<uintptr_t>(base) % 16 == 0 && st[3] == 1 && st[2] % 4 == 0 && st[1] % 4 == 0 && st[0] % 4 == 0;
  };
  const int vec = rows_ok(p.q, p.qs) && rows_ok(p.k, p.ks) && rows_ok(p.v, p.vs);
  switch (p.D) {
    case 16:  return launch_simt_inst<T, 16>(p, vec, grid, stream);
    case 32:  return launch_simt_inst<T, 32>(p, vec, grid, stream);
    case 64:  return launch_simt_inst<T, 64>(p, vec, grid, stream);
    case 128: return launch_simt_inst<T, 128>(p, vec, grid, stream);
    default:  return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_attn_simt(const AttnParams& p, cudaStream_t stream) {
  switch (p.dtype) {
    case SA_DTYPE_F32:  return launch_for_dtype<float>(p, stream);
    case SA_DTYPE_F16:  return launch_for_dtype<__half>(p, stream);
    case SA_DTYPE_BF16: return launch_for_dtype<__nv_bfloat16>(p, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sa
