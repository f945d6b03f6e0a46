// tc_mlp.cuh — the proposer's MLP on the 5th-generation tensor cores (tcgen05.mma, accumulators in
// tensor memory), over 128-row tiles.
//
// Layout.  Operands are BF16 in shared memory in the K-major canonical layout without swizzle:
// 8x8-element core matrices of 128 contiguous bytes (8 rows x 16 bytes); core matrix (row group g,
// K chunk c) of an A tile sits at c * LBO + g * 128 (SBO = 128), so within one K chunk the 128 rows
// are contiguous 16-byte rows: the layer-1 tile is the stored features as they are (K chunk 0)
// followed by a zero chunk (K padded from 8 to 16).  A weight image (64 output rows) has
// LBO = 1024.  One tcgen05.mma (M = 128, N = 64, K = 16, kind::f16, BF16 x BF16 -> FP32) covers
// two K chunks: one per tile for layer 1, four for layers 2 and 3.  Accumulators are 64 TMEM columns,
// lane = row, so after each layer each of the 128 threads of a tile reads its own row back with
// tcgen05.ld.32x32b (a warp reads the 32 lanes of its quarter), applies bias + ReLU, rounds to
// BF16 and writes the next layer's A row.
//
// A tile is a chain of three MMA round trips, so what counts is the number of tiles in flight and the
// instructions of the epilogue.  A CTA holds the weights once for four groups of 128 threads, each
// with a tile, an mbarrier and 64 TMEM columns of its own: with two CTAs an SM has eight tiles in
// flight (one-tile CTAs, each with its 18 KB of weights, fitted five).  The epilogue adds the bias two
// columns at a time (add.rn.f32x2) and applies ReLU in the conversion to BF16.
//
// Synchronisation.  One thread of a group issues the MMAs and commits them to the group's mbarrier;
// every thread of the group waits on it with an iteration limit, and one named barrier per layer
// joins the group.  That barrier also reduces the threads' verdicts on their wait, so that a wait that
// runs out in any of them stops the whole group after the same layer (a flag in shared memory would
// not do: a thread that is through the barrier could set it for the next layer before another has read
// it for this one, and the two would part).  The status is set then; TMEM is always freed.  A CTA
// allocates 256 TMEM columns and its shared memory keeps at most two on an SM: allocation never has
// to wait.
#ifndef PLIS_TC_MLP_CUH_
#define PLIS_TC_MLP_CUH_

#include <cuda_bf16.h>
#include <stdint.h>

namespace plis {
namespace tc {

constexpr uint32_t kA1Bytes = 2 * 2048;        // A tile of layer 1: 128 rows x K 16
constexpr uint32_t kABytes = 8 * 2048;         // A tile of layers 2, 3: 128 rows x K 64
constexpr uint32_t kW1Bytes = 2 * 1024;        // W1^T: 64 x 16
constexpr uint32_t kWBytes = 8 * 1024;         // W2^T, W3^T: 64 x 64
constexpr uint32_t kWImageBytes = kW1Bytes + 2 * kWBytes;  // 18 KB, the packed weight image
constexpr uint32_t kWaitLimit = 1u << 22;

// instruction descriptor: D F32, A BF16, B BF16, both K-major, N = 64, M = 128
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, no swizzle (start, leading and stride byte offsets >> 4, version 1)
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(kIdesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void ld16(uint32_t taddr, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// two binary32 sums at once, and two values to BF16 (lo in the low half) with negative ones to zero
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
  return (uint64_t)__float_as_uint(hi) << 32 | __float_as_uint(lo);
}
__device__ __forceinline__ uint32_t relu_bf16x2(uint64_t v) {
  uint32_t r;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;"
      : "=r"(r)
      : "f"(__uint_as_float((uint32_t)(v >> 32))), "f"(__uint_as_float((uint32_t)v)));
  return r;
}

// byte offset of element (row, k) in a K-major canonical tile whose K chunks are `chunk` bytes apart
__device__ __forceinline__ uint32_t canon(uint32_t row, uint32_t k, uint32_t chunk) {
  return (k >> 3) * chunk + (row >> 3) * 128u + (row & 7u) * 16u + (k & 7u) * 2u;
}

// wait for the mbarrier phase `parity`; false when the limit ran out
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i)
    if (try_wait(bar, parity)) return true;
  return false;
}

struct Params {
  const uint4* wimg;   // packed weight image (kWImageBytes), global
  const float* b1;
  const float* b2;
  const float* b3;
  const float* w4;
  float b4;
};

// Persistent tile kernel: shared memory of one CTA, kGroups groups of 128 threads with a tile each
constexpr uint32_t kGroups = 4;
constexpr uint32_t kThreads = kGroups * 128;
constexpr uint32_t kPOffW = 0;
constexpr uint32_t kPOffA = kPOffW + kWImageBytes;            // A tiles of layers 2, 3, one per group
constexpr uint32_t kPOffA1 = kPOffA + kGroups * kABytes;      // features: K chunk 0 of the layer-1 A tiles
constexpr uint32_t kPOffZero = kPOffA1 + kGroups * 2048;      // K chunk 1: zeros (the padding of K 8 -> 16)
constexpr uint32_t kPOffVec = kPOffZero + 2048;
constexpr uint32_t kPOffBar = kPOffVec + 4 * 64 * 4;          // an mbarrier per group, then the TMEM address
constexpr uint32_t kPSmemBytes = kPOffBar + kGroups * 8 + 16;
constexpr uint32_t kPTmemCols = kGroups * 64;
static_assert(kPSmemBytes * 3 > 228 * 1024 && kPTmemCols * 2 <= 512, "two CTAs per SM, and TMEM for both");

__device__ __forceinline__ void group_sync(uint32_t group) { asm volatile("bar.sync %0, 128;" ::"r"(group + 1u) : "memory"); }
// the same barrier; true in all 128 threads when `v` is true in any of them
__device__ __forceinline__ bool group_any(uint32_t group, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tbar.red.or.pred q, %1, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(group + 1u), "r"(v ? 1u : 0u)
      : "memory");
  return r != 0;
}

// The MLP on tcgen05 for the rows of `feats` (normalised BF16 features, 16 bytes per row, rows
// 0 .. 128 * ntiles - 1 readable), tiles taken round robin by the groups of the grid.
// sink.begin(row) is called when a tile's rows are known (to start loads), sink.end(row, y) with its
// result, by the thread that owns the row.  A wait that runs out sets *status and its group stops.
template <class Sink>
static __device__ __forceinline__ void mlp_tiles(const Params& P, const uint4* __restrict__ feats, uint32_t ntiles,
                                                 uint8_t* smem, int* status, uint32_t wait_limit, Sink& sink) {
  if (wait_limit == 0) wait_limit = kWaitLimit;
  const uint32_t tid = threadIdx.x;  // blockDim.x == kThreads
  const uint32_t group = tid >> 7, t = tid & 127u;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar = sbase + kPOffBar + 8u * group;
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + kPOffBar + kGroups * 8);
  float* vec = reinterpret_cast<float*>(smem + kPOffVec);
  {
    uint4* dst = reinterpret_cast<uint4*>(smem + kPOffW);
    for (uint32_t i = tid; i < kWImageBytes / 16; i += kThreads) dst[i] = __ldg(&P.wimg[i]);
    if (tid < 128) reinterpret_cast<uint4*>(smem + kPOffZero)[tid] = make_uint4(0u, 0u, 0u, 0u);
    if (tid < 64) {
      vec[tid] = __ldg(&P.b1[tid]);
      vec[64 + tid] = __ldg(&P.b2[tid]);
      vec[128 + tid] = __ldg(&P.b3[tid]);
      vec[192 + tid] = __ldg(&P.w4[tid]);
    }
    if (t == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    if (tid < 32) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                   "r"(kPTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  fence_before();
  fence_async_smem();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *slot + 64u * group;
  const uint32_t my_cols = tmem + ((t & 96u) << 16);  // lanes 32 * (warp of the group)
  uint8_t* a1 = smem + kPOffA1 + 2048u * group;
  uint8_t* a = smem + kPOffA + kABytes * group;
  const uint32_t sa1 = sbase + kPOffA1 + 2048u * group, sa = sbase + kPOffA + kABytes * group;
  uint32_t phase = 0;
  const uint32_t first = blockIdx.x * kGroups + group, step = gridDim.x * kGroups;
  uint4 next = first < ntiles ? feats[first * 128u + t] : make_uint4(0u, 0u, 0u, 0u);
  bool ok = true;
  for (uint32_t tile = first; tile < ntiles && ok; tile += step) {
    const uint32_t row = tile * 128u + t;
    // row t of chunk 0 of the layer-1 A tile sits at t * 16: the features as they are stored
    reinterpret_cast<uint4*>(a1)[t] = next;
    sink.begin(row);
    if (tile + step < ntiles) next = feats[(tile + step) * 128u + t];
    fence_before();
    fence_async_smem();
    group_sync(group);
    float out = 0.f;
#pragma unroll
    for (int layer = 0; layer < 3; ++layer) {
      if (t == 0) {
        fence_after();
        if (layer == 0) {
          mma(tmem, sdesc(sa1, sbase + kPOffZero - sa1, 128), sdesc(sbase + kPOffW, 1024, 128), 0u);
        } else {
          const uint32_t w = sbase + kPOffW + kW1Bytes + (layer == 1 ? 0u : kWBytes);
          for (uint32_t ks = 0; ks < 4; ++ks)
            mma(tmem, sdesc(sa + ks * 2u * 2048u, 2048, 128), sdesc(w + ks * 2u * 1024u, 1024, 128), ks > 0 ? 1u : 0u);
        }
        commit(bar);
      }
      const bool got = wait_phase(bar, phase & 1u, wait_limit);
      phase += 1;
      fence_after();
      __syncwarp();
      if (__all_sync(0xffffffffu, got)) {
        if (layer < 2) {
          const ulonglong2* b = reinterpret_cast<const ulonglong2*>(vec + 64 * layer);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float v[16];
            ld16(my_cols + 16u * c, v);
            uint32_t p[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const ulonglong2 bb = b[4 * c + i];
              p[2 * i] = relu_bf16x2(add2(pair(v[4 * i], v[4 * i + 1]), bb.x));
              p[2 * i + 1] = relu_bf16x2(add2(pair(v[4 * i + 2], v[4 * i + 3]), bb.y));
            }
            *reinterpret_cast<uint4*>(a + canon(t, 16u * c, 2048)) = make_uint4(p[0], p[1], p[2], p[3]);
            *reinterpret_cast<uint4*>(a + canon(t, 16u * c + 8u, 2048)) = make_uint4(p[4], p[5], p[6], p[7]);
          }
        } else {
          const float4* b = reinterpret_cast<const float4*>(vec + 128);
          const float4* w = reinterpret_cast<const float4*>(vec + 192);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float v[16];
            ld16(my_cols + 16u * c, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 bb = b[4 * c + i], ww = w[4 * c + i];
              out = out + fmaxf(v[4 * i] + bb.x, 0.f) * ww.x;
              out = out + fmaxf(v[4 * i + 1] + bb.y, 0.f) * ww.y;
              out = out + fmaxf(v[4 * i + 2] + bb.z, 0.f) * ww.z;
              out = out + fmaxf(v[4 * i + 3] + bb.w, 0.f) * ww.w;
            }
          }
          out = out + P.b4;
        }
      }
      fence_before();
      fence_async_smem();
      if (group_any(group, !got)) {
        ok = false;
        break;
      }
    }
    if (ok) sink.end(row, out);
  }
  if (!ok) wait_phase(bar, (phase - 1u) & 1u, kWaitLimit);  // the MMAs in flight finish before their TMEM is freed
  fence_before();
  __syncthreads();
  fence_after();
  if (tid < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*slot), "r"(kPTmemCols) : "memory");
  if (t == 0 && !ok) atomicExch(status, 6 /* PLIS_ERR_TIMEOUT */);
}

}  // namespace tc
}  // namespace plis

#endif
