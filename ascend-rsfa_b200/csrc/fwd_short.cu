// FlashAttention-2 forward for B200 (sm_100a), sequences of one key tile: "short" kernel.
//
// The counterpart of the reference's single-tile kernels _attn_fwd_small and _attn_fwd_small_causal
// (ascend_rsfa/flash_attention_forward.py:26-159): the whole row of scores is in registers, so there is no
// online recurrence - one maximum, one pass of exponentials, one division.
//
// What bounds it: HBM, and behind that the latency of a warp's own chain of products and exponentials.  A head
// of S <= 128 rows is 4 * S * D * 2 bytes for at most S / 2 FLOP per byte, so the kernel is built around keeping
// loads in flight.  Heads are independent and small, which is why the tensor path is warp-level mma.sync here:
// a warp owns 16 query rows from the first load to the last store, and nothing in the loop waits for more than
// the warps that share one head.  (A tcgen05 tile has 128 rows: the persistent kernels spend 3.4 us per head on
// the hand-overs between their roles whatever its length.)
//   team    = the ceil(S / 16) warps that work on one head, one strip of 16 query rows each
//   CTA     = as many teams as fit in eight warps and 96 KB of ring; two CTAs per SM (128 registers: three CTAs
//             with 80 spill and are 15-50 % slower, one with 255 has too few warps: 25-40 % slower)
//   ring    = `stages` slots per team, each one head's Q, K and V, filled by TMA (swizzled by the row length,
//             rows past S read as zeros)
// A slot is refilled by the last warp of the team that is done with it (a counter in shared memory tells
// which one that is), so no warp ever waits for a slot to become free and there is no producer warp.  O leaves
// through the warp's own rows of the Q tile, which only this warp read, as whole 16-byte pieces.
// Heads go to teams by a fixed stride: they all take equally long.  The loops over keys take 32 at a time so
// that the fragment loads of a step are issued together, ahead of its products.
// Measured on 4096 heads (us per launch from a graph of launches, inputs rotated; before = the kernel that had
// the size: fwd_generic at S <= 64, D <= 64 and D = 16, the tcgen05 kernels otherwise; floor = bytes at the
// measured copy rate, 6.55 TB/s):
//   S = 64 D = 64     72.3 -> 23.3 (floor 20.5)     S = 64 D = 128        95.5 -> 49.0 (floor 41.0)
//   S = 100 D = 32    84.0 -> 40.2 (floor 16.0)     the same, causal      84.0 -> 32.5
//   S = 128 D = 64    72.5 -> 67.0 (floor 41.0)     the same, causal      84.8 -> 51.5
//   S = 128 D = 16    57.3 -> 31.6 (floor 10.2)     S = 30 D = 64 (x 2)  109.9 -> 22.6 (floor 19.2)
// and at 2 heads, where latency is all there is: S = 128 D = 64 5.2 -> 4.3, S = 64 D = 128 6.2 -> 3.2.  At S = 128 D = 64
// without the mask a launch whose heads leave the last wave of two per SM thin is up to 4 % slower than on the tcgen05
// kernel (300 heads 10.9 -> 11.3, 600 15.4 -> 15.9, 1000 21.7 -> 22.4), one of full waves 4 to 8 % faster.
#include "../../include/rsfa.h"
#include "tcgen05_common.cuh"

namespace rsfa {
namespace {

constexpr int kMaxWarpsShort = 8;
constexpr int kMaxStagesShort = 8;
constexpr int kCtasPerSmShort = 2;            // 128 registers per thread
constexpr int kRingBytesShort = 96 * 1024;    // per CTA

struct ShortMaps {
  CUtensorMap q, k, v;
};

struct ShortPlan {
  int heads;       // B * H
  int first_loads; // heads whose loads a ring may start with: all, but for the test of a wait that runs out
  int strips;      // warps per team = ceil(S / 16)
  int teams;       // teams per CTA
  int stages;      // ring slots per team
  int tile_bytes;  // one of Q, K, V of one head: S rounded up to 32 rows
  // head / H as one multiplication: x / H = (x * div_mul) >> div_shift for 0 <= x < 2^31 (round-up
  // method of Granlund and Montgomery: div_mul = ceil(2^div_shift / H), div_shift = 31 + ceil(log2 H))
  unsigned long long div_mul;
  int div_shift;
};

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool kBf16>
__device__ __forceinline__ void mma_16x8x16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

// The same with C = 0: the first product of a sum needs no cleared registers.
template <bool kBf16>
__device__ __forceinline__ void mma_16x8x16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  }
}

// Byte offset of the 16-byte chunk `chunk` of row `row` in a TMA box of min(D, 64) columns: rows of up to 128
// bytes with the swizzle of that width, which spreads eight consecutive rows over all the banks.
template <int D>
__device__ __forceinline__ uint32_t box_offset(int row, int chunk) {
  constexpr int kRowBytes = 2 * (D < 64 ? D : 64);
  const int swizzle = (D >= 64) ? (row & 7) : (D == 32) ? ((row >> 1) & 3) : ((row >> 2) & 1);
  return static_cast<uint32_t>(row * kRowBytes + ((chunk ^ swizzle) << 4));
}

// kKeys: the key capacity of a warp's score registers (32, 64, 96 or 128), S <= kKeys.  kAll: no causal mask, and
// kKeys is S rounded up to 32: every row sees every step of 32 keys.
template <int D, int kKeys, bool kBf16, bool kAll>
__global__ void __launch_bounds__(32 * kMaxWarpsShort, kCtasPerSmShort)
fwd_short_kernel(const __grid_constant__ ShortMaps maps, const FwdParams p, const ShortPlan plan) {
  constexpr int kSteps = kKeys / 32;               // steps of 32 keys
  constexpr int kBoxes = D <= 64 ? 1 : D / 64;     // TMA boxes of 64 columns per row
  constexpr int kBoxCols = D / kBoxes;
  constexpr int kSlices = D / 16;                  // slices of 16 columns
  constexpr int kBoxSlices = kSlices / kBoxes;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kMaxWarpsShort * kMaxStagesShort];
  __shared__ int readers[kMaxWarpsShort * kMaxStagesShort];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int team = warp / plan.strips;
  int strip = warp - team * plan.strips;
  const int slots = plan.teams * plan.stages;
  for (int i = threadIdx.x; i < slots; i += blockDim.x) {
    mbar_init(smem_u32(&full_bar[i]), 1);
    readers[i] = 0;
  }
  if (threadIdx.x == 0) {
    abort_word = 0;
    tma_prefetch_desc(&maps.q);
    tma_prefetch_desc(&maps.k);
    tma_prefetch_desc(&maps.v);
  }
  fence_barrier_init();
  fence_proxy_async();
  __syncthreads();
  // Only this CTA's shared memory so far; global memory waits for the kernel in front on the stream.
  griddep_wait();

  const int S = p.S;
  const int first = blockIdx.x * plan.teams + team;
  const int stride = gridDim.x * plan.teams;
  const uint32_t slot_bytes = 3u * plan.tile_bytes;
  const uint32_t box_bytes = static_cast<uint32_t>(plan.tile_bytes) / kBoxes;
  const uint32_t ring = smem_base + static_cast<uint32_t>(team * plan.stages) * slot_bytes;

  auto batch_of = [&](int bh) {
    return static_cast<int>((static_cast<unsigned long long>(static_cast<unsigned int>(bh)) * plan.div_mul) >> plan.div_shift);
  };
  // one lane: Q, K and V of head `bh` into a slot of this team
  auto load_head = [&](int bh, int slot) {
    const uint32_t bar = smem_u32(&full_bar[team * plan.stages + slot]);
    const uint32_t dst = ring + slot * slot_bytes;
    const int b = batch_of(bh), h = bh - b * p.H;
    mbar_arrive_expect_tx(bar, slot_bytes);
#pragma unroll
    for (int bx = 0; bx < kBoxes; ++bx) {
      tma_load_4d(dst + bx * box_bytes, &maps.q, bar, bx * kBoxCols, 0, h, b);
      tma_load_4d(dst + plan.tile_bytes + bx * box_bytes, &maps.k, bar, bx * kBoxCols, 0, h, b);
      tma_load_4d(dst + 2 * plan.tile_bytes + bx * box_bytes, &maps.v, bar, bx * kBoxCols, 0, h, b);
    }
  };
  if (strip == 0 && lane == 0) {
    for (int s = 0; s < plan.stages; ++s)
      if (first + s * stride < plan.first_loads) load_head(first + s * stride, s);
  }
  __syncwarp();

  const float scale_log2 = p.sm_scale * kLog2e;
  // Fragment addresses inside a box, for its first 16 rows: blocks of 16 rows and boxes are a constant apart.
  constexpr uint32_t kBlockBytes = 16 * 2 * kBoxCols;
  uint32_t off_a[kBoxSlices], off_k[kBoxSlices];   // A fragments of Q and B fragments of V; B fragments of K
#pragma unroll
  for (int kk = 0; kk < kBoxSlices; ++kk) {
    off_a[kk] = box_offset<D>(lane & 15, kk * 2 + (lane >> 4));
    off_k[kk] = box_offset<D>((lane & 7) + ((lane >> 4) << 3), kk * 2 + ((lane >> 3) & 1));
  }

  int slot = 0;
  uint32_t phase = 0;
  bool ok = true;
  for (int bh = first; bh < plan.heads; bh += stride) {
    ok = mbar_wait_warp(smem_u32(&full_bar[team * plan.stages + slot]), phase, abort_flag, p.wait_limit_ns, kTagKvFull);
    if (!ok) break;
    const uint32_t sQ = ring + slot * slot_bytes + strip * kBlockBytes;   // this warp's rows
    const uint32_t sK = ring + slot * slot_bytes + plan.tile_bytes;
    const uint32_t sV = sK + plan.tile_bytes;
    const int r0 = strip * 16;                                     // rows r0 .. r0 + 15
    const int row_lo = r0 + (lane >> 2), row_hi = row_lo + 8;
    const int last_key = p.causal ? min(S - 1, r0 + 15) : S - 1;   // of any row of the strip
    const int n_steps = (last_key >> 5) + 1;
    const int lim_lo = p.causal ? min(S - 1, row_lo) : S - 1;      // last visible key of a row
    const int lim_hi = p.causal ? min(S - 1, row_hi) : S - 1;
    const int lim_all = p.causal ? r0 : S - 1;                     // keys up to here are visible to every row

    // ---- scores of 16 rows x 32 * n_steps keys
    uint32_t qf[kSlices][4];
#pragma unroll
    for (int kk = 0; kk < kSlices; ++kk) ldsm_x4(qf[kk], sQ + (kk / kBoxSlices) * box_bytes + off_a[kk % kBoxSlices]);
    float s[kSteps][4][4];
#pragma unroll
    for (int st = 0; st < kSteps; ++st) {
      if (kAll || st == 0 || st < n_steps) {
        // K fragments of up to four slices at a time: their loads go out together
#pragma unroll
        for (int bx = 0; bx < kBoxes; ++bx) {
          uint32_t kf[2][kBoxSlices][4];
#pragma unroll
          for (int i = 0; i < 2 * kBoxSlices; ++i)
            ldsm_x4(kf[i & 1][i >> 1], sK + bx * box_bytes + off_k[i >> 1] + (2 * st + (i & 1)) * kBlockBytes);
#pragma unroll
          for (int kk = 0; kk < kBoxSlices; ++kk) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (bx == 0 && kk == 0)
                mma_16x8x16_first<kBf16>(s[st][i], qf[kk], kf[i >> 1][kk][2 * (i & 1)], kf[i >> 1][kk][2 * (i & 1) + 1]);
              else
                mma_16x8x16<kBf16>(s[st][i], qf[bx * kBoxSlices + kk], kf[i >> 1][kk][2 * (i & 1)],
                                   kf[i >> 1][kk][2 * (i & 1) + 1]);
            }
          }
        }
      }
    }

    // ---- mask, row maximum (a row is spread over the four lanes of a quad)
    float m_lo = -INFINITY, m_hi = -INFINITY;
#pragma unroll
    for (int st = 0; st < kSteps; ++st) {
      if (kAll || st == 0 || st < n_steps) {
        if ((!kAll || st == kSteps - 1) && st * 32 + 31 > lim_all) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int col = st * 32 + i * 8 + (lane & 3) * 2 + (e & 1);
              if (col > ((e & 2) ? lim_hi : lim_lo)) s[st][i][e] = -INFINITY;
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          m_lo = max3(m_lo, s[st][i][0], s[st][i][1]);
          m_hi = max3(m_hi, s[st][i][2], s[st][i][3]);
        }
      }
    }
    m_lo = fmaxf(m_lo, __shfl_xor_sync(0xffffffffu, m_lo, 1));
    m_hi = fmaxf(m_hi, __shfl_xor_sync(0xffffffffu, m_hi, 1));
    m_lo = fmaxf(m_lo, __shfl_xor_sync(0xffffffffu, m_lo, 2));
    m_hi = fmaxf(m_hi, __shfl_xor_sync(0xffffffffu, m_hi, 2));

    // The maximum comes off before the scale goes on: exact where it counts, whatever the scores' size.  With s * scale -
    // (m * scale) in one operation every P of the row is off by a factor 2^e, e the rounding error of m * scale; the
    // division takes it out again, but from products of 2^28 (fp16) and 2^31 (fp32) on P does not hold it: rows whose
    // keys a program hides with the type's lowest value came out as NaN.  The second operation costs 0 to 3 %, 5 % at most
    // (4096 heads, us: S = 64 D = 64 23.3 -> 23.4, S = 100 D = 32 causal 31.8 -> 32.5, S = 128 D = 64 66.2 -> 67.7, S = 128
    // D = 16 30.7 -> 31.6, S = 112 D = 16 30.0 -> 31.5); a branch for large rows only costs as much or more (S = 64 D = 128 7 %).
    // A row of nothing but -inf has the sum 0.
    const float ref_lo = m_lo == -INFINITY ? 0.f : m_lo, ref_hi = m_hi == -INFINITY ? 0.f : m_hi;

    // ---- P = exp2((s - m) * scale), row sums, O += P V, step by step
    const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2);
    const uint64_t neg_lo2 = pack_f32x2(-ref_lo, -ref_lo);
    const uint64_t neg_hi2 = pack_f32x2(-ref_hi, -ref_hi);
    uint64_t sum_lo2 = pack_f32x2(0.f, 0.f), sum_hi2 = sum_lo2;
    float acc[D / 8][4];
#pragma unroll
    for (int st = 0; st < kSteps; ++st) {
      if (kAll || st == 0 || st < n_steps) {
        uint32_t pf[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float x0, x1, x2, x3;
          unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(s[st][i][0], s[st][i][1]), neg_lo2), scale2), x0, x1);
          unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(s[st][i][2], s[st][i][3]), neg_hi2), scale2), x2, x3);
          const float e0 = ex2(x0), e1 = ex2(x1), e2 = ex2(x2), e3 = ex2(x3);
          sum_lo2 = add_f32x2(sum_lo2, pack_f32x2(e0, e1));
          sum_hi2 = add_f32x2(sum_hi2, pack_f32x2(e2, e3));
          pf[i >> 1][2 * (i & 1)] = pack2<kBf16>(e0, e1);
          pf[i >> 1][2 * (i & 1) + 1] = pack2<kBf16>(e2, e3);
        }
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
          for (int bx = 0; bx < kBoxes; ++bx) {
            uint32_t vf[kBoxSlices][4];
#pragma unroll
            for (int dt = 0; dt < kBoxSlices; ++dt)
              ldsm_x4_trans(vf[dt], sV + bx * box_bytes + off_a[dt] + (2 * st + kb) * kBlockBytes);
#pragma unroll
            for (int dt = 0; dt < 2 * kBoxSlices; ++dt) {
              float (&o)[4] = acc[bx * 2 * kBoxSlices + dt];
              if (st == 0 && kb == 0)
                mma_16x8x16_first<kBf16>(o, pf[kb], vf[dt >> 1][2 * (dt & 1)], vf[dt >> 1][2 * (dt & 1) + 1]);
              else
                mma_16x8x16<kBf16>(o, pf[kb], vf[dt >> 1][2 * (dt & 1)], vf[dt >> 1][2 * (dt & 1) + 1]);
            }
          }
        }
      }
    }
    float l_lo, l_hi, l_odd;
    unpack_f32x2(sum_lo2, l_lo, l_odd);
    l_lo += l_odd;
    unpack_f32x2(sum_hi2, l_hi, l_odd);
    l_hi += l_odd;
    l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1);
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1);
    l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);
    const float inv_lo = 1.f / l_lo, inv_hi = 1.f / l_hi;

    // ---- O through this warp's rows of the Q tile: written as fragments, read back as 16-byte pieces
    __syncwarp();
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      constexpr int kBoxChunks = kBoxCols / 8;
      const uint32_t at = sQ + (i / kBoxChunks) * box_bytes + (lane & 3) * 4;
      st_shared_b32(at + box_offset<D>(lane >> 2, i % kBoxChunks), pack2<kBf16>(acc[i][0] * inv_lo, acc[i][1] * inv_lo));
      st_shared_b32(at + box_offset<D>((lane >> 2) + 8, i % kBoxChunks), pack2<kBf16>(acc[i][2] * inv_hi, acc[i][3] * inv_hi));
    }
    __syncwarp();
    uint4 out[kSlices];
    constexpr int kChunks = D / 8;   // 16-byte pieces of a row
#pragma unroll
    for (int i = 0; i < kSlices; ++i) {
      const int row = (i * 32 + lane) / kChunks, chunk = (i * 32 + lane) % kChunks;
      out[i] = ld_shared_v4(sQ + (chunk / (kBoxCols / 8)) * box_bytes + box_offset<D>(row, chunk % (kBoxCols / 8)));
    }
    // ---- the slot: the last warp of the team to get here fills it again
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      int* counter = &readers[team * plan.stages + slot];
      if (atomicAdd(counter, 1) == plan.strips - 1) {
        *counter = 0;
        __threadfence_block();
        fence_proxy_async();
        const int next = bh + plan.stages * stride;
        if (next < plan.heads) load_head(next, slot);
      }
    }
    __syncwarp();

    const int b = batch_of(bh), h = bh - b * p.H;
    uint16_t* go = reinterpret_cast<uint16_t*>(p.o) + b * p.o_stride[0] + h * p.o_stride[1];
#pragma unroll
    for (int i = 0; i < kSlices; ++i) {
      const int idx = i * 32 + lane;
      const int row = r0 + idx / kChunks;
      if (row < S) *reinterpret_cast<uint4*>(go + row * p.o_stride[2] + (idx % kChunks) * 8) = out[i];
    }
    if (p.lse != nullptr && (lane & 3) == 0) {
      float* lse = p.lse + static_cast<int64_t>(bh) * S;
      if (row_lo < S) lse[row_lo] = m_lo * p.sm_scale + logf(l_lo);
      if (row_hi < S) lse[row_hi] = m_hi * p.sm_scale + logf(l_hi);
    }
    if (++slot == plan.stages) {
      slot = 0;
      phase ^= 1u;
    }
    // With the causal mask a strip's work grows with its number: warps swap strips, first with last, from
    // head to head, so that each has the same work over two heads (the ring lets them drift that far apart).
    if (p.causal) strip = plan.strips - 1 - strip;
  }
  griddep_launch_dependents();
  if (!ok && lane == 0) {
    // Give loads still in flight time to land before shared memory goes away, then say what ran out.
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    atomicCAS(p.status, 0, *abort_flag);
  }
}

// [B, H, S, D] tensor as a 4-D map with boxes of min(D, 64) columns x `box_rows` and the swizzle of that row length.
bool make_short_map(CUtensorMap* map, const void* base, const FwdParams& p, const int64_t* st, int box_rows) {
  return make_map_boxed(map, base, p, st, p.D < 64 ? p.D : 64, box_rows,
                        p.D >= 64 ? CU_TENSOR_MAP_SWIZZLE_128B : p.D == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

template <int D, int kKeys, bool kBf16, bool kAll>
cudaError_t launch_short_one(const FwdParams& p, int sm_count, cudaStream_t stream, long long* launches) {
  ShortPlan plan;
  plan.heads = p.B * p.H;
  plan.first_loads = (p.test_drop_load >= 0 && p.test_drop_load < plan.heads) ? p.test_drop_load : plan.heads;
  plan.strips = (p.S + 15) / 16;
  const int rows = (p.S + 31) / 32 * 32;   // keys are taken 32 at a time; rows past S read as zeros
  plan.tile_bytes = rows * D * 2;
  // Teams per CTA: eight warps' worth, as far as the ring holds a slot for each, and no more than it takes
  // to give every SM work.
  plan.teams = kMaxWarpsShort / plan.strips;
  if (plan.teams > kRingBytesShort / (3 * plan.tile_bytes)) plan.teams = kRingBytesShort / (3 * plan.tile_bytes);
  const int spread = (plan.heads + sm_count - 1) / sm_count;
  if (plan.teams > spread) plan.teams = spread;
  plan.div_shift = 31;
  while ((1ll << (plan.div_shift - 31)) < p.H) ++plan.div_shift;
  plan.div_mul = ((1ull << plan.div_shift) + p.H - 1) / p.H;
  ShortMaps maps;
  if (!make_short_map(&maps.q, p.q, p, p.q_stride, rows) ||
      !make_short_map(&maps.k, p.k, p, p.k_stride, rows) ||
      !make_short_map(&maps.v, p.v, p, p.v_stride, rows))
    return cudaErrorInvalidValue;
  if (plan.teams < 1) return cudaErrorInvalidValue;   // a head larger than the ring: short_fits() lets none through
  const int stage_set = plan.teams * 3 * plan.tile_bytes;
  plan.stages = kRingBytesShort / stage_set;
  if (plan.stages > kMaxStagesShort) plan.stages = kMaxStagesShort;
  const long long per_cta = kCtasPerSmShort;
  long long grid = (plan.heads + plan.teams - 1) / plan.teams;
  if (grid > per_cta * sm_count) grid = per_cta * sm_count;
  const long long rounds = (plan.heads + grid * plan.teams - 1) / (grid * plan.teams);
  if (plan.stages > rounds) plan.stages = static_cast<int>(rounds);
  const int smem = plan.stages * stage_set + 1024;
  auto kern = fwd_short_kernel<D, kKeys, kBf16, kAll>;
  static std::atomic<unsigned long long> smem_done{0};   // per kernel instantiation, bit per device
  cudaError_t e = set_dynamic_smem_once(smem_done, reinterpret_cast<const void*>(kern), kRingBytesShort + 1024);
  if (e != cudaSuccess) return e;
  e = launch_persistent(kern, static_cast<int>(grid), 32 * plan.teams * plan.strips, smem, stream, p.pdl != 0, maps, p, plan);
  if (e == cudaSuccess) *launches += 1;
  return e;
}

// Without the mask every row sees all steps: the loops over them have no branches then, and the score registers are
// as many as the length needs, in steps of 32 keys (4096 heads, us: S = 100 D = 32 42.1 -> 40.1, S = 112 D = 16 33.4 ->
// 29.5, S = 90 D = 64 46.1 -> 42.3, S = 20 D = 32, 8192 heads, 12.6 -> 11.9).  Not at D = 64 with 128 keys, where the
// straight line spills (64.9 -> 66.8), and not with fewer than 64 keys' registers for causal rows of D >= 64 (S = 30
// 21.9 -> 22.4).  These figures are from before the maximum came off the scores in an operation of its own.
template <int D, int kKeys>
cudaError_t launch_short_keys(const FwdParams& p, int sm_count, cudaStream_t stream, long long* launches) {
  if constexpr (D < 64 || kKeys < 128) {
    if (!p.causal)
      return p.bf16 ? launch_short_one<D, kKeys, true, true>(p, sm_count, stream, launches)
                    : launch_short_one<D, kKeys, false, true>(p, sm_count, stream, launches);
  }
  return p.bf16 ? launch_short_one<D, kKeys, true, false>(p, sm_count, stream, launches)
                : launch_short_one<D, kKeys, false, false>(p, sm_count, stream, launches);
}

template <int D>
cudaError_t launch_short_dim(const FwdParams& p, int sm_count, cudaStream_t stream, long long* launches) {
  if (p.S <= 32 && (D < 64 || !p.causal)) return launch_short_keys<D, 32>(p, sm_count, stream, launches);
  if (p.S <= 64) return launch_short_keys<D, 64>(p, sm_count, stream, launches);
  if constexpr (D <= 64) {
    if (p.S <= 96) return launch_short_keys<D, 96>(p, sm_count, stream, launches);
    return launch_short_keys<D, 128>(p, sm_count, stream, launches);
  } else {
    return cudaErrorInvalidValue;
  }
}

}  // namespace

// Sizes the kernel takes.  Measured against what had them before (see the table above); D = 128 with more than
// 64 keys would need 96 KB per head and both score and output registers of 64 per thread.
bool short_fits(int S, int D, float sm_scale) { return S >= 1 && (D <= 64 ? S <= 128 : D == 128 && S <= 64) && sm_scale > 0.f; }

cudaError_t launch_fwd_short(const FwdParams& p, int sm_count, cudaStream_t stream, long long* launches) {
  switch (p.D) {
    case 16: return launch_short_dim<16>(p, sm_count, stream, launches);
    case 32: return launch_short_dim<32>(p, sm_count, stream, launches);
    case 64: return launch_short_dim<64>(p, sm_count, stream, launches);
    case 128: return launch_short_dim<128>(p, sm_count, stream, launches);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace rsfa
