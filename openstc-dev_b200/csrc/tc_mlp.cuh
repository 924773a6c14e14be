// tc_mlp.cuh — the surrogate network's forward pass on the 5th-generation
// tensor cores (tcgen05), transposed: the weights are the A operand and 64
// states at a time the B operand, so that every weight stays on the SM.
//
// One CTA of 512 threads owns one SM: W2 (128 KB), W1 and W4 in shared memory,
// W3 in half of tensor memory (an A operand may be read from there). Two groups
// of 8 warps walk tiles of 64 states, each with its own activations (in place:
// a layer's products are done before its epilogue writes) and its own 128
// accumulator columns, so that the products of one group run under the
// epilogue of the other. Per tile:
//   L1  D[256x64]  = W1[256x16]  X0^T     2 MMAs (two halves of 128 features)
//   L2  D          = W2[256x256] A1^T    32 MMAs (W2 from shared memory)
//   L3  D          = W3[256x256] A2^T    32 MMAs (W3 from tensor memory)
//   L4  D4[64x16]  = A3[64x256]  W4^T    16 MMAs (M = 128: the upper 64 rows read
//                                        whatever follows the activations and
//                                        are not used)
// Epilogue: thread (warp, lane) holds one feature of all 64 states: bias, SiLU,
// BF16 pairs of neighbouring features exchanged with the neighbouring lane, 4-byte
// stores into the next layer's operand.
//
// Bound by the chain of a tile: three epilogues of 2400 cycles (the special-function
// unit's share, 768 SiLUs a state at one exponential each and one reciprocal for two, is
// 1536) and products of 2100 cycles a layer (66 cycles for each M = 128, N = 64, the rate of
// N = 128), the two groups mostly in step. With 128-state tiles as the A operand, one in
// flight per SM and W2 / W3 streamed from L2 for every tile, 1.5 million states took
// 1718 us; now 1042.
//
// One thread of a group issues its MMAs and commits them to the group's mbarrier,
// which the group waits on for at most WAIT_NS of the global timer. When a wait
// runs out anywhere in a group, the group stops walking tiles: it sets the error
// word, commits once more so that the barrier tracks every MMA it issued, waits
// for that (bounded again) and for its own asynchronous copies; the CTA frees its
// tensor memory when both groups are done.
#pragma once
#include <cuda_bf16.h>

#include "mlp.cuh"

namespace ostc {
namespace tc {

using mlp::KIN;
using mlp::NH;
using mlp::NOUTP;

constexpr int ROWS = 64;  // states per tile
constexpr int THREADS = 512, GROUPS = 2, GTHREADS = THREADS / GROUPS;
// activations of a tile as a K-major operand whose K-adjacent core matrices lie
// 144 bytes apart: a warp's epilogue stores go to four of them at once, which at
// the dense 128 bytes would share their banks
constexpr unsigned ACT_LBO = 144, ACT_SBO = NH / 8 * ACT_LBO;
constexpr unsigned ACT_BYTES = ROWS / 8 * ACT_SBO;
// shared memory map (bytes); what follows the second activations is readable (layer 4)
constexpr unsigned SM_ACT = 0;                                // 2 x 64 x 256 bf16
constexpr unsigned SM_W2 = SM_ACT + GROUPS * ACT_BYTES;       // 256 x 256 bf16
constexpr unsigned SM_W1 = SM_W2 + NH * NH * 2;               // 256 x 16 bf16
constexpr unsigned SM_W4 = SM_W1 + NH * KIN * 2;              // 16 x 256 bf16
constexpr unsigned SM_X0 = SM_W4 + NOUTP * NH * 2;            // 2 x 64 x 16 bf16
constexpr unsigned SM_BAR = SM_X0 + GROUPS * ROWS * KIN * 2;  // one mbarrier (8 B) per group
constexpr unsigned SM_TMEM = SM_BAR + 8 * GROUPS;             // allocated tensor-memory base (4 B)
constexpr unsigned SM_BYTES = SM_TMEM + 8;
static_assert(SM_BYTES <= 227 * 1024, "one CTA's shared memory");
static_assert(SM_ACT + (GROUPS - 1) * ACT_BYTES + 128 / 8 * ACT_SBO <= SM_BYTES, "layer 4 reads 128 rows");
// tensor memory: group g's accumulators in columns 128 g .. 128 g + 127 (64 per half
// of the features), W3 in columns 256 .. 511 (128 per half)
constexpr unsigned TMEM_COLS = 512, TM_W3 = 256;
constexpr unsigned long long WAIT_NS = 1000000000ull;  // 1 s of the global timer per mbarrier wait

// byte offset of element (r, k) of an R x K operand in the canonical K-major
// no-swizzle layout: 8 x 16-byte core matrices, K-adjacent cores 128 B apart
// (leading byte offset), 8-row groups K/8 * 128 B apart (stride byte offset)
__device__ __forceinline__ unsigned core_off(int r, int k, int K) {
  return (unsigned)(((r >> 3) * (K >> 3) + (k >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// shared-memory matrix descriptor (tcgen05): start, LBO, SBO in 16-byte
// units, descriptor version 1, no swizzle
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr, unsigned lbo, unsigned sbo) {
  return (unsigned long long)((addr >> 4) & 0x3FFF) | ((unsigned long long)((lbo >> 4) & 0x3FFF) << 16) |
         ((unsigned long long)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// instruction descriptor: BF16 x BF16 -> F32, both K-major, M = 128, N
__host__ __device__ constexpr unsigned idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
}

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mma_issue(unsigned tmem_d, unsigned long long a, unsigned long long b, unsigned idesc,
                                          unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// bounded wait for the mbarrier phase `parity`; false when WAIT_NS ran out. The
// timer is read only once a first round of tries has failed: the read is slow
// against the products that most waits are for.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) {
  for (unsigned it = 0; it < 32; ++it)
    if (bar_try(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (unsigned it = 0;; ++it) {
    if (bar_try(bar, parity)) return true;
    if ((it & 31) == 31 && global_ns() - t0 > WAIT_NS) return false;
  }
}

// 32 consecutive FP32 columns of this thread's lane (no wait: tmem_wait_ld)
__device__ __forceinline__ void tmem_ld32_async(unsigned taddr, unsigned *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 consecutive FP32 columns of this thread's lane
__device__ __forceinline__ void tmem_ld32(unsigned taddr, float *v) {
  unsigned r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(unsigned taddr, float *v) {
  unsigned r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *(const unsigned *)&h;
}

__device__ __forceinline__ void cp_async16(unsigned dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_prior1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// copy a row-major global N x K bf16 matrix into the canonical layout; each
// CTA starts at its own offset, so the SMs that stream the same weights at
// the same time spread over the L2 slices instead of queueing on one line
__device__ __forceinline__ void load_weights(unsigned char *smem, unsigned off, const __nv_bfloat16 *w, int N, int K) {
  const int chunks = N * K / 8;
  const int rot = (int)((blockIdx.x * 613u) % (unsigned)chunks);
  for (int i = threadIdx.x; i < chunks; i += THREADS) {
    const int c = i + rot < chunks ? i + rot : i + rot - chunks;
    const int n = c / (K / 8), kc = c % (K / 8);
    cp_async16(smem_u32(smem + off + core_off(n, kc * 8, K)), w + (long long)n * K + kc * 8);
  }
}

// one MMA with the A operand in tensor memory
__device__ __forceinline__ void mma_issue_ta(unsigned tmem_d, unsigned tmem_a, unsigned long long b, unsigned idesc,
                                             unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(b), "r"(idesc), "r"(accumulate));
}

// 32 consecutive columns of this thread's lane, written (no wait: tmem_wait_st)
__device__ __forceinline__ void tmem_st32(unsigned taddr, const unsigned *r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// the barrier of one group's threads, and the same with an OR over them
__device__ __forceinline__ void group_sync(int g) {
  asm volatile("barrier.cta.sync %0, %1;" ::"r"(1 + g), "r"(GTHREADS) : "memory");
}
__device__ __forceinline__ bool group_or(int g, bool v) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"((unsigned)v), "r"(1 + g), "r"(GTHREADS)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// z / (1 + exp(-z)) of two values with one reciprocal; the exponentials are held
// below 2^62, so that the product of the denominators stays finite (SiLU is below
// 1e-16 there)
__device__ __forceinline__ void silu2(float &a, float &b) {
  constexpr float log2e = 1.4426950408889634f;
  const float da = 1.f + ex2(fminf(-log2e * a, 62.f)), db = 1.f + ex2(fminf(-log2e * b, 62.f));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(da * db));
  a *= r * db;
  b *= r * da;
}

// The network core. `Io` supplies, per tile of 64 rows and for the group's threads
// (t = 0 .. 255),
//   void stage(int tile, unsigned char *x0, int t)    the tile's rows as standardised
//                                              BF16 in the operand layout, by plain
//                                              stores or cp.async
//   void store(int tile, int row, const float *y10)   standardised outputs
// Returns nothing; errors go to *err (1 = a wait ran out).
template <typename Io>
__device__ void mlp_tiles(const mlp::Net &net, int n_tiles, Io &io, int *err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = tid / GTHREADS, t = tid % GTHREADS;  // group, thread of the group
  const int half = (warp >> 2) & 1;                  // features 128 half .. 128 half + 127
  const int f = half * 128 + (warp & 3) * 32 + lane;  // this thread's feature
  const unsigned bar = smem_u32(smem + SM_BAR + 8 * g);
  unsigned *tmem_slot = (unsigned *)(smem + SM_TMEM);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // resident weights; each thread keeps its feature's biases
  load_weights(smem, SM_W1, net.w1(), NH, KIN);
  load_weights(smem, SM_W2, net.w2(), NH, NH);
  load_weights(smem, SM_W4, net.w4(), NOUTP, NH);
  const float bias1 = net.b1()[f], bias2 = net.b2()[f], bias3 = net.b3()[f];
  fence_before();
  __syncthreads();
  fence_after();
  const unsigned tmem = *tmem_slot;
  const unsigned lane_addr = (unsigned)((warp & 3) * 32) << 16;
  if (g == 0) {  // W3: row f into lane f % 128, two values of K per column
    const uint4 *w = (const uint4 *)(net.w3() + (long long)f * NH);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      unsigned r[32];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint4 v = __ldg(w + c * 8 + e);
        r[4 * e] = v.x, r[4 * e + 1] = v.y, r[4 * e + 2] = v.z, r[4 * e + 3] = v.w;
      }
      tmem_st32(tmem + lane_addr + TM_W3 + half * 128 + c * 32, r);
    }
    tmem_wait_st();
  }
  cp_async_wait_all();
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();

  unsigned char *act = smem + SM_ACT + g * ACT_BYTES, *x0 = smem + SM_X0 + g * ROWS * KIN * 2;
  const unsigned act0 = smem_u32(act), d0 = tmem + 128 * g;
  // where this thread's stores go: even lanes hold the even states of a pair of
  // features, odd lanes the odd ones
  unsigned char *out = act + (f >> 3) * ACT_LBO + (f & 6) * 2 + (lane & 1) * 16;
  unsigned parity = 0;
  bool timed_out = false;  // group-uniform: a bounded wait ran out somewhere in the group
  const int stride = GROUPS * gridDim.x;
  int tile = blockIdx.x * GROUPS + g;
  if (tile < n_tiles) io.stage(tile, x0, t);
  for (; tile < n_tiles; tile += stride) {
    cp_async_wait_all();
    fence_async_smem();
    fence_before();
    group_sync(g);
    fence_after();
    if (t == 0) {
      const unsigned long long b = smem_desc(smem_u32(x0), 128, 2 * 128);
      for (int h = 0; h < 2; ++h)
        mma_issue(d0 + 64 * h, smem_desc(smem_u32(smem + SM_W1) + h * 128 * KIN * 2, 128, 2 * 128), b, idesc_bf16(ROWS),
                  0);
      // net.withhold_commit (a diagnostic of the timeout path): no completion
      // signal for this product, so the wait below runs out
      if (!net.withhold_commit) mma_commit(bar);
    }
    for (int layer = 0; layer < 3; ++layer) {
      if (group_or(g, !bar_wait(bar, parity))) {
        timed_out = true;
        break;
      }
      parity ^= 1;
      fence_after();
      // the next tile's rows load under this tile's layers (layer 1 has read its own)
      if (layer == 0 && tile + stride < n_tiles) io.stage(tile + stride, x0, t);
      // epilogue: bias + SiLU -> BF16 activations (the next layer's operand)
      const float b = layer == 0 ? bias1 : (layer == 1 ? bias2 : bias3);
      unsigned acc[ROWS];
      tmem_ld32_async(d0 + lane_addr + 64 * half, acc);
      tmem_ld32_async(d0 + lane_addr + 64 * half + 32, acc + 32);
      tmem_wait_ld();
#pragma unroll
      for (int n = 0; n < ROWS; n += 2) {
        float a0 = __uint_as_float(acc[n]) + b, a1 = __uint_as_float(acc[n + 1]) + b;
        silu2(a0, a1);
        const unsigned own = pack_bf16(a0, a1);  // states n, n + 1 of this feature
        const unsigned oth = __shfl_xor_sync(0xffffffffu, own, 1);
        // even lane: state n of features f, f + 1; odd lane: state n + 1 of f - 1, f
        const unsigned w = lane & 1 ? __byte_perm(oth, own, 0x7632) : __byte_perm(own, oth, 0x5410);
        *(unsigned *)(out + (n >> 3) * ACT_SBO + (n & 7) * 16) = w;
      }
      fence_async_smem();
      fence_before();
      group_sync(g);
      fence_after();
      if (t == 0) {
        // unrolled, so that each product costs its one thread an addition per descriptor
        const unsigned long long ad = smem_desc(act0, ACT_LBO, ACT_SBO);
        constexpr unsigned id = idesc_bf16(ROWS);
        if (layer == 0) {
          const unsigned long long wd = smem_desc(smem_u32(smem + SM_W2), 128, NH * 16);
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int s = 0; s < NH / 16; ++s)
              mma_issue(d0 + 64 * h, wd + (h * 128 * NH * 2 + s * 256) / 16, ad + s * 2 * ACT_LBO / 16, id, s > 0);
        } else if (layer == 1) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int s = 0; s < NH / 16; ++s)
              mma_issue_ta(d0 + 64 * h, tmem + TM_W3 + h * 128 + s * 8, ad + s * 2 * ACT_LBO / 16, id, s > 0);
        } else {
          const unsigned long long wd = smem_desc(smem_u32(smem + SM_W4), 128, NH * 16);
#pragma unroll
          for (int s = 0; s < NH / 16; ++s)
            mma_issue(d0, ad + s * 2 * ACT_LBO / 16, wd + s * 256 / 16, idesc_bf16(NOUTP), s > 0);
        }
        mma_commit(bar);
      }
    }
    if (timed_out || group_or(g, !bar_wait(bar, parity))) {
      timed_out = true;
      break;
    }
    parity ^= 1;
    fence_after();
    if (t < ROWS) {
      float v[16], y[10];
      tmem_ld16(d0 + lane_addr, v);
#pragma unroll
      for (int i = 0; i < 10; ++i) y[i] = v[i] + net.b4()[i];
      io.store(tile, t, y);
    }
  }
  if (timed_out) {
    // drain: one more commit tracks every MMA this group issued; wait for it
    // (bounded) before the memory goes
    if (t == 0) {
      mma_commit(bar);
      if (err) atomicExch(err, 1);
    }
    bar_wait(bar, parity);
  }
  cp_async_wait_all();
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

// rows of 16 standardised BF16 features (12 and 4 zeros, 32 bytes, the
// operand's K) in; rows of 10 FP32 outputs out
struct PackedIo {
  const __nv_bfloat16 *x;
  float *y;
  int n;
  __device__ void stage(int tile, unsigned char *x0, int t) const {
    if (t >= 2 * ROWS) return;
    const int row = t >> 1, half = t & 1;
    const long long q = (long long)tile * ROWS + row;
    unsigned char *dst = x0 + core_off(row, half * 8, KIN);
    if (q < n)
      cp_async16(smem_u32(dst), x + q * KIN + half * 8);
    else
      *(uint4 *)dst = make_uint4(0, 0, 0, 0);
  }
  __device__ void store(int tile, int row, const float *o) const {
    const long long q = (long long)tile * ROWS + row;
    if (q >= n) return;
    float2 *d = (float2 *)(y + q * mlp::NOUT);
#pragma unroll
    for (int i = 0; i < mlp::NOUT / 2; ++i) d[i] = make_float2(o[2 * i], o[2 * i + 1]);
  }
};

}  // namespace tc
}  // namespace ostc
