// gm_mlp.cu -- the learned initial guess on the fifth-generation tensor
// cores: inference and training kernels and their host-side drivers.
//
// Every product is D[128 x N] = A[128 x K] B[N x K]^T with A and B in BF16,
// D in FP32 tensor memory: tcgen05.mma (kind::f16, one CTA, M = 128) issued
// by one thread, its operands in shared memory in the 128-byte-swizzled
// layout that TMA writes (rows of 64 BF16 elements; a K-major atom is 128
// rows x 128 bytes), completion signalled through an mbarrier by
// tcgen05.commit, the accumulator read back with tcgen05.ld (thread t of
// warp w reads row 32 w + t).  Weights come from BF16 copies in global
// memory (L2 resident) by 2-D TMA loads into a two-stage ring, so the load
// of the next weight block overlaps the current product and epilogue.
// Activations are written into the operand tile by the epilogue threads
// themselves (the swizzle computed in place), so a tile's three layers run
// back to back without leaving the SM.  Inference keeps two tiles in
// flight per CTA, each with eight epilogue warps, and a producer warp.
//
// Training runs per batch: (1) one fused kernel per 128-pixel tile for the
// forward pass, the loss, and the backward pass through the activations
// (dH2 = dOut W3, dZ2 = dH2 * GELU'(Z2), dH1 = dZ2 W2, dZ1 = dH1 * GELU'(Z1)),
// whose operands and gradients it stores row-major (TMA stores of the
// operand tiles) for (2) the weight-gradient kernel, dW = G^T A over the
// batch, with both operands MN-major; (3) the bias gradients; (4) Adam on the
// FP32 parameters, which also rewrites the BF16 copies.
//
// Waits are bounded: a wait that runs past 2 s sets an error flag that the
// host reads, and the kernel then stops issuing work, waits (bounded) for
// its copies in flight, frees its tensor memory and returns.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>

#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "gm_mlp.cuh"

namespace gm {
namespace mlp {
namespace {

// Inference kernel: 8 epilogue warps a tile, two tiles' worth, and a producer
// warp; training kernel: 16 epilogue warps.  Warp w reads rows
// 32 (w % 4) .. + 31 of the accumulator, and a tile's warpgroups split each
// epilogue's columns in equal parts.  The weight-gradient
// kernel: 4 warps, one row each.
constexpr int kThreads = 512;
constexpr int kWThreads = 128;
constexpr uint64_t kWaitNs = 2000000000ull;   // a wait gives up after 2 s

// error codes written to the kernel's error word
enum : int { kErrNone = 0, kErrWaitLoad = 1, kErrWaitMma = 2, kErrWaitStage = 3 };

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for the phase of barrier b with the given parity.  Returns false when
// it gave up: after kWaitNs (it then records `code` in *err and raises the
// block's abort flag) or as soon as another thread has raised the flag.
__device__ __noinline__ bool mbar_wait_slow(uint64_t* b, uint32_t parity, volatile int* abort, int* err, int code,
                                            bool stop_on_abort) {
  const uint64_t t0 = now_ns();
  while (!mbar_test(b, parity)) {
    if (stop_on_abort && *abort) return false;
    if (now_ns() - t0 > kWaitNs) {
      *abort = 1;
      atomicCAS(err, kErrNone, code);
      return false;
    }
  }
  return true;
}
// The phase is usually complete by the time a thread asks (a weight block
// loaded during the previous products, the products during the epilogue):
// one test inline, the bounded loop out of line.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort, int* err, int code,
                                          bool stop_on_abort = true) {
  if (mbar_test(b, parity)) return true;
  return mbar_wait_slow(b, parity, abort, err, code, stop_on_abort);
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 2-D TMA: box at (x = inner coordinate, y = row) into / out of shared memory
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(saddr(bar))
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x),
               "r"(y), "r"(src)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// tensor memory: allocation by one warp, fences around thread syncs
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(dst)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor of a 128-byte-swizzled operand.  K-major:
// 8-row groups 1024 bytes apart (SBO); MN-major: 8-row (K) groups SBO apart
// and 64-element MN blocks LBO apart.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;   // descriptor version of this architecture
  d |= (uint64_t)2 << 61;   // 128-byte swizzle
  return d;
}
// Instruction descriptor: BF16 x BF16 -> FP32, M x N, K-major (0) or
// MN-major (1) operands.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
               : "memory");
}
// 32 columns of this warp's 32 lanes: the load is asynchronous; its
// registers are valid after tmem_wait32 on the same array, whose asm takes
// them as operands so that no read of them is placed before the wait.
__device__ __forceinline__ void tmem_issue32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait32(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  tmem_issue32(taddr, r);
  tmem_wait32(r);
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15])
               :
               : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 16-byte chunk j (elements 8j..8j+7 of its 64-element row) of row r of the
// K-major swizzled atom at `atom` (shared-memory address).
__device__ __forceinline__ void st_chunk(uint32_t atom, int r, int j, const uint32_t (&w)[4]) {
  const uint32_t a = atom + (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((j ^ (r & 7)) << 4));
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
               : "memory");
}

// GELU in its tanh form (Hendrycks & Gimpel, 2016): z (1 + tanh u) / 2 with
// u = sqrt(2 / pi) (z + 0.044715 z^3), written as z s, s = 1 / (1 + exp(-2 u))
// -- one exponential and one reciprocal on the special-function unit -- and
// its derivative s + z s (1 - s) d(2u)/dz.
__device__ __forceinline__ float gelu_s(float z, float* du2) {
  const float z2 = z * z;
  const float u2 = 1.5957691216057308f * z * (1.f + 0.044715f * z2);
  if (du2) *du2 = 1.5957691216057308f * (1.f + 0.134145f * z2);
  // exp(80) keeps the denominator inside the fast reciprocal's range
  return __fdividef(1.f, 1.f + __expf(fminf(-u2, 80.f)));
}
__device__ __forceinline__ float gelu(float z) { return z * gelu_s(z, nullptr); }
__device__ __forceinline__ float gelu_grad(float z) {
  float du2;
  const float s = gelu_s(z, &du2);
  return s + z * s * (1.f - s) * du2;
}


// ---------------------------------------------------------------- kernel layout
// Shared memory (offsets from a 1024-byte aligned base).
constexpr uint32_t kSA = 0;            // activation operand: 4 K-atoms x [128 rows x 128 B]
constexpr uint32_t kSW = 65536;        // weight ring: 2 stages x 64 KB
constexpr uint32_t kStage = 65536;
constexpr uint32_t kSD = 196608;       // output-gradient operand: 1 atom [128 x 64]
constexpr uint32_t kSBar = 212992;     // barriers, tensor-memory address, abort flag
constexpr uint32_t kSPar = kSBar + 128; // b1, b2, in_mean, in_scale (floats), read by every tile
constexpr int kParFloats = 256 + 256 + 128 + 128;
constexpr size_t kSmemBytes = kSPar + 4 * kParFloats + 1024;

struct NetMaps {
  CUtensorMap m[5];                    // w1b, w2b, w3b, w2tb, w3tb
};
enum { kMapW1 = 0, kMapW2, kMapW3, kMapW2t, kMapW3t };

// One weight block of a layer: `natoms` K-atoms (64 K each) of a weight copy
// with `rows` rows (N), multiplied with A-operand atoms a_first.. (of the
// activation tile, or of the output-gradient tile when a_sd), into tensor
// columns tcol.., accumulating onto what is there when acc, ending its layer
// (the epilogue waits for it) when end.  The weight block's K offset is
// that of its A atoms.
struct Job {
  uint8_t map, natoms, a_first, a_sd;
  uint16_t rows, tcol;
  uint8_t acc, end;
};
constexpr int kTrainJobs = 7;
__constant__ Job c_jobs[kTrainJobs] = {
    {kMapW1, 2, 0, 0, 256, 0, 0, 1},      // Z1 = X W1^T
    {kMapW2, 2, 0, 0, 256, 256, 0, 0},    // Z2 = H1 W2^T (K 0..127)
    {kMapW2, 2, 2, 0, 256, 256, 1, 1},    //            (K 128..255)
    {kMapW3, 4, 0, 0, 16, 0, 0, 1},       // out = H2 W3^T
    {kMapW3t, 1, 0, 1, 256, 0, 0, 1},     // dH2 = dOut W3
    {kMapW2t, 2, 0, 0, 256, 256, 0, 0},   // dH1 = dZ2 W2 (K 0..127)
    {kMapW2t, 2, 2, 0, 256, 256, 1, 1},   //            (K 128..255)
};
// weight blocks of layer L: [first, last)
__device__ __forceinline__ int layer_first(int L) { return L == 0 ? 0 : (L == 1 ? 1 : L + 1); }
__device__ __forceinline__ int layer_last(int L) { return L == 0 ? 1 : (L == 1 ? 3 : (L == 4 ? 7 : L + 2)); }

struct Bars {
  uint64_t full[2], mma;
  uint32_t tmem;
  int abort;
};

// Producer (thread 0): the TMA loads of one weight block into a stage.
__device__ __forceinline__ void load_job(const Job& j, const NetMaps& nm, uint32_t stage, uint64_t* full) {
  const uint32_t atom = (uint32_t)j.rows * 128u;
  mbar_expect_tx(full, atom * j.natoms);
  for (int a = 0; a < j.natoms; ++a) tma_load_2d(stage + a * atom, &nm.m[j.map], 64 * (j.a_first + a), 0, full);
}

// Issuer (thread 0): the products of one weight block, K in steps of 16
// (32 bytes along a swizzled 128-byte row).
__device__ __forceinline__ void mma_job(const Job& j, uint32_t tmem, uint32_t tcol, uint32_t sA, uint32_t sD,
                                        uint32_t stage) {
  const uint32_t idesc = idesc_bf16(128, j.rows, 0, 0);
  const uint32_t abase = j.a_sd ? sD : sA + j.a_first * 16384u;
  const uint32_t batom = (uint32_t)j.rows * 128u;
  for (int k = 0; k < j.natoms * 4; ++k) {
    const int a = k >> 2, kk = k & 3;
    const uint64_t ad = sw128_desc(abase + a * 16384u + kk * 32u, 16, 1024);
    const uint64_t bd = sw128_desc(stage + a * batom + kk * 32u, 16, 1024);
    mma_bf16(tmem + tcol, ad, bd, idesc, (k > 0 || j.acc) ? 1u : 0u);
  }
}

// Producer / issuer state (thread 0), and the epilogue barrier's parity
// (all threads).  Weight blocks run in the order of c_jobs, tile after tile,
// through the two stages in turn.
struct Pipe {
  uint32_t fph[2] = {0, 0};                     // next parity to wait for
  bool inflight[2] = {false, false};            // a load into stage s not yet waited for
  uint32_t mph = 0;
  int64_t g = 0, loaded = 0;                    // weight blocks run and loads started so far
};

// Thread 0, with the products of every block run so far complete: start the
// loads of the next two blocks of `total` that are not on their way yet.
__device__ __forceinline__ void load_ahead(int64_t total, const NetMaps& nm, Bars* B, uint32_t base, Pipe& p) {
  while (p.loaded < total && p.loaded < p.g + 2) {
    const int s = (int)(p.loaded & 1);
    load_job(c_jobs[p.loaded % kTrainJobs], nm, base + kSW + s * kStage, &B->full[s]);
    p.inflight[s] = true;
    ++p.loaded;
  }
}

// Thread 0: run the next weight block: wait for its weights, issue its
// products, signal the epilogue at the end of a layer.  Returns false on abort.
__device__ bool run_job(const Job& j, Bars* B, uint32_t base, Pipe& p, int* err) {
  const int s = (int)(p.g & 1);
  if (!mbar_wait(&B->full[s], p.fph[s], &B->abort, err, kErrWaitLoad)) return false;
  p.fph[s] ^= 1u;
  p.inflight[s] = false;
  tc_fence_after();
  mma_job(j, B->tmem, j.tcol, base + kSA, base + kSD, base + kSW + s * kStage);
  if (j.end) mma_commit(&B->mma);
  ++p.g;
  return true;
}

// Load a tile's inputs (batch rows row0..,  pixel idx[row] or the row itself)
// standardised and rounded to BF16 into the activation atoms 0-1.  Warp w of
// the NW that share the work takes the rows 128 / NW w .., a row at a time:
// lane f holds features 4 f .. 4 f + 3, so a row is one coalesced read (a row
// per lane instead touched 32 lines an instruction and took 10 k cycles a
// tile) and the lane's standardisation stays in registers.  Rows of 4 nl
// floats start on 16-byte boundaries and the feature count is a multiple of
// 4, so every 4-feature group is read whole or not at all.
template <int NW>
__device__ __forceinline__ void load_x(const float* spar, const float* __restrict__ iquv,
                                       const uint32_t* __restrict__ idx, int64_t row0, int64_t n, int nl,
                                       uint32_t sA, int w) {
  constexpr int R = kTile / NW, U = 8;   // rows of this warp, reads in flight
  static_assert(R % U == 0 && R <= 32, "a warp's rows");
  const int f = threadIdx.x & 31;
  const uint32_t mine = idx && f < R && row0 + w * R + f < n ? __ldg(idx + row0 + w * R + f) : 0u;
  const float4 mu = reinterpret_cast<const float4*>(spar + 512)[f];
  const float4 sc = reinterpret_cast<const float4*>(spar + 640)[f];
  const uint32_t atom = sA + (uint32_t)(f >> 4) * 16384u;
#pragma unroll 1
  for (int r0 = w * R; r0 < w * R + R; r0 += U) {
    float4 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t b = row0 + r0 + u;
      const int64_t p = idx ? (int64_t)__shfl_sync(0xffffffffu, mine, r0 + u - w * R) : b;
      if (b < n && f < nl)
        x[u] = __ldg(reinterpret_cast<const float4*>(iquv + p * (4 * nl)) + f);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u;
      uint32_t lo = 0u, hi = 0u;
      if (row0 + r < n && f < nl) {
        lo = pack_bf16((x[u].x - mu.x) * sc.x, (x[u].y - mu.y) * sc.y);
        hi = pack_bf16((x[u].z - mu.z) * sc.z, (x[u].w - mu.w) * sc.w);
      }
      const uint32_t a = atom + (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((((f >> 1) & 7) ^ (r & 7)) << 4) +
                                           8 * (f & 1));
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(lo), "r"(hi) : "memory");
    }
  }
}

// Ask for the lines of a tile's inputs in L2 (thread i of the 256 that share it).
__device__ __forceinline__ void prefetch_x(const float* __restrict__ iquv, int64_t row0, int64_t n, int nl, int i) {
  const int64_t rows = n - row0 < kTile ? n - row0 : kTile;
  const char* p = reinterpret_cast<const char*>(iquv + row0 * (4 * nl));
  for (int64_t o = 128 * (int64_t)i; o < rows * (16 * nl); o += 128 * 256)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
}

// Epilogue of a hidden layer over the accumulator at tensor column zcol:
// h = GELU(z + bias) into the activation atoms (K = feature); with zspill,
// z + bias also to zspill[128 c] (columns 4 c .. 4 c + 3 of this row: a warp's
// rows are neighbours there).  This thread: row r, part `part` of PARTS of
// the 256 columns, 32 at a time, the next 32 columns' tensor-memory load in
// flight while these are processed.  bias: 256 floats in shared memory.
__device__ __forceinline__ void hidden_chunk(const uint32_t (&zr)[32], int q, const float* bias, uint32_t sA,
                                             int r, float4* zspill) {
  float z[32];
  const float4* b4 = reinterpret_cast<const float4*>(bias + 32 * q);
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const float4 bv = b4[u];
    z[4 * u] = __uint_as_float(zr[4 * u]) + bv.x;
    z[4 * u + 1] = __uint_as_float(zr[4 * u + 1]) + bv.y;
    z[4 * u + 2] = __uint_as_float(zr[4 * u + 2]) + bv.z;
    z[4 * u + 3] = __uint_as_float(zr[4 * u + 3]) + bv.w;
  }
  if (zspill) {
#pragma unroll
    for (int u = 0; u < 8; ++u)
      zspill[(8 * q + u) * kTile] = make_float4(z[4 * u], z[4 * u + 1], z[4 * u + 2], z[4 * u + 3]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    uint32_t w[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) w[h] = pack_bf16(gelu(z[8 * u + 2 * h]), gelu(z[8 * u + 2 * h + 1]));
    st_chunk(sA + (q >> 1) * 16384u, r, (q & 1) * 4 + u, w);
  }
}

template <int PARTS>
__device__ __forceinline__ void hidden_epilogue(uint32_t tmem_row, uint32_t zcol, const float* bias, uint32_t sA,
                                                int r, int part, float4* zspill) {
  constexpr int N = 8 / PARTS;   // chunks of 32 columns
  const int q0 = N * part;
  const uint32_t t0 = tmem_row + zcol + 32 * q0;
  uint32_t za[32], zb[32];
  tmem_issue32(t0, za);
#pragma unroll
  for (int j = 0; j < N; j += 2) {
    tmem_wait32(za);
    tmem_issue32(t0 + 32 * (j + 1), zb);
    hidden_chunk(za, q0 + j, bias, sA, r, zspill);
    tmem_wait32(zb);
    if (j + 2 < N) tmem_issue32(t0 + 32 * (j + 2), za);
    hidden_chunk(zb, q0 + j + 1, bias, sA, r, zspill);
  }
}

// The parameters every tile reads (b1, b2, in_mean, in_scale) into the
// shared-memory block at spar, once per launch.
__device__ __forceinline__ void stage_params(const gm_mlp* __restrict__ P, float* spar) {
  for (int i = threadIdx.x; i < kParFloats; i += blockDim.x)
    spar[i] = i < 256 ? P->b1[i] : (i < 512 ? P->b2[i - 256] : (i < 640 ? P->in_mean[i - 512] : P->in_scale[i - 640]));
}

// Outputs (de-standardised) -> start model (Init_Model layout) within the
// reference's ranges (check, milosUtils.cu:160-238); fixed parameters and
// v_mac / filling factor from the guess model.
__device__ __forceinline__ void outputs_to_model(const float (&y)[kOut], const double* guess, const int* fix,
                                                 double* m) {
  const double bl = y[6], bq = y[7], bu = y[8];
  const double bt = sqrt(bq * bq + bu * bu);
  const double B = sqrt(bl * bl + bt * bt);
  const double gam = atan2(bt, bl) * (180.0 / 3.14159265358979323846);
  double phi = 0.5 * atan2(bu, bq) * (180.0 / 3.14159265358979323846);
  if (phi < 0) phi += 180.0;
  double v[11];
  v[0] = fmin(fmax((double)y[0], 1.0), 2500.0);
  v[1] = fmin(B, 5000.0);
  v[2] = fmin(fmax((double)y[1], -20.0), 20.0);
  v[3] = fmin(fmax((double)y[2], 1e-4), 0.6);
  v[4] = fmin(fmax((double)y[3], 1e-4), 10.0);
  v[5] = gam;
  v[6] = phi;
  v[7] = fmin(fmax((double)y[4], 1e-4), 2.0);
  v[8] = fmin(fmax((double)y[5], 1e-4), 2.0);
  v[9] = guess[9];
  v[10] = guess[10];
#pragma unroll
  for (int i = 0; i < 11; ++i) m[i] = (i < 9 && fix[i] && isfinite(v[i])) ? v[i] : guess[i];
}

struct InferArgs {
  const gm_mlp* p;
  const float* iquv;
  int64_t n;
  int nl;
  double guess[11];
  int fix[11];
  double* models;
  int* err;
};

struct TrainKArgs {
  const gm_mlp* p;
  const float* iquv;
  const float* y16;        // [pixels][16] standardised targets
  const uint32_t* idx;     // batch row -> pixel
  int64_t n;               // rows of this batch (a multiple of 128)
  int nl;
  float gscale;            // d loss / d output per unit of error: 2 / (rows x 9)
  float* zspill;           // [tiles][64][128][4] pre-activations of layer 1 (4-column group, row)
  float* loss;             // sum of squared errors (atomic)
  int* err;
};

struct ActMaps {
  // row-major BF16 [rows][128 | 256 | 256 | 64 | 256 | 256], boxes of 64 x 128
  CUtensorMap x, h1, h2, g3, g2, g1;
};

__device__ __forceinline__ void setup(Bars* B, uint32_t ncols) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(&B->full[0], 1);
    mbar_init(&B->full[1], 1);
    mbar_init(&B->mma, 1);
    B->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if ((tid >> 5) == 0) tmem_alloc(&B->tmem, ncols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}

// End of a kernel (every thread): thread 0 waits, bounded, for the weight
// loads still in flight (there are none unless the kernel aborted), for its
// products (a last commit) and for its stores; then the tensor memory is
// freed.
__device__ __forceinline__ void teardown(Bars* B, Pipe& p, uint32_t ncols, int* err) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s)
      if (p.inflight[s]) mbar_wait(&B->full[s], p.fph[s], &B->abort, err, kErrWaitLoad, false);
    mma_commit(&B->mma);
    mbar_wait(&B->mma, p.mph, &B->abort, err, kErrWaitMma, false);
    tma_store_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == 0) tmem_dealloc(B->tmem, ncols);
}

}  // namespace

// ---------------------------------------------------------------- inference
// Persistent and warp-specialised, two 128-pixel tiles in flight per CTA
// (slots 0 and 1: each its own activation tile in shared memory, 256
// tensor-memory columns and eight epilogue warps).  Warps 8 s .. 8 s + 7 load
// slot s's inputs, and after each of its products turn the accumulator into
// the next operand (GELU) or the start models; warp 16's first thread streams
// the weights through two 32 KB stages by TMA and issues the products.  Per
// pair of tiles (A in slot 0, B in slot 1) the products run L0(A) L0(B) L1(A)
// L1(B) L2(A) L2(B); each waits for the epilogue that wrote its operand
// (hready, the slot's 256 threads arrive) and each epilogue for its product
// (zready, a commit), so the slots' epilogues overlap each other and the
// products of the other slot.
//
// Bound by the epilogues: 512 GELUs a pixel, two special-function operations
// each, 60 us of that unit for 2^18 pixels, and about as many issue slots.
// Eight warps serving both slots in turn, each thread reading a row of inputs
// (10 k of a tile's 42 k cycles), took 197 us; sixteen, each pair of
// warpgroups on its own slot, rows read coalesced from lines asked for a
// tile ahead, and one warpgroup loading the next tile while the other forms
// the start models: 163 us (that unit 43 % active; a slot still waits 9 k of
// 36 k cycles for its products).
constexpr int kIEpi = 256;                     // epilogue threads of a slot
constexpr int kIThreads = 2 * kIEpi + 32;      // and the producer warp
constexpr uint32_t kIAct = 65536;              // one slot's activation tile (4 K-atoms)
constexpr uint32_t kIW = 2 * kIAct;            // weight stages
constexpr uint32_t kIStage = 32768;            // one K-atom of a 256-row weight
constexpr uint32_t kIBar = kIW + 2 * kIStage;
constexpr uint32_t kIPar = kIBar + 128;
constexpr size_t kISmemBytes = kIPar + 4 * kParFloats + 1024;

struct IBars {
  uint64_t full[2], empty[2];   // weight stages: loaded / free again
  uint64_t zready[2];           // slot's accumulator written (product committed)
  uint64_t hready[2];           // slot's operand tile written (256 epilogue threads)
  uint64_t fin;
  uint32_t tmem;
  int abort;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
}

// Producer state (warp 16, lane 0)
struct Prod {
  uint32_t fph[2] = {0, 0}, eph[2] = {0, 0}, hph[2] = {0, 0};
  bool pend[2] = {false, false}, inflight[2] = {false, false};
};

// Load `natoms` K-atoms (from atom k0) of a weight into stage st, once the
// products that last read the stage are done.
__device__ __forceinline__ bool p_load(Prod& P, IBars* B, uint32_t wbase, int st, const CUtensorMap* map, int k0,
                                       int natoms, uint32_t atom_bytes, int* err) {
  if (P.pend[st]) {
    if (!mbar_wait(&B->empty[st], P.eph[st], &B->abort, err, kErrWaitStage)) return false;
    P.eph[st] ^= 1u;
    P.pend[st] = false;
  }
  mbar_expect_tx(&B->full[st], atom_bytes * natoms);
  for (int a = 0; a < natoms; ++a) tma_load_2d(wbase + st * kIStage + a * atom_bytes, map, 64 * (k0 + a), 0, &B->full[st]);
  P.inflight[st] = true;
  return true;
}
__device__ __forceinline__ bool p_wait(Prod& P, IBars* B, int st, int* err) {
  if (!mbar_wait(&B->full[st], P.fph[st], &B->abort, err, kErrWaitLoad)) return false;
  P.fph[st] ^= 1u;
  P.inflight[st] = false;
  tc_fence_after();
  return true;
}
__device__ __forceinline__ void p_release(Prod& P, IBars* B, int st) {
  mma_commit(&B->empty[st]);
  P.pend[st] = true;
}
__device__ __forceinline__ bool p_wait_operand(Prod& P, IBars* B, int slot, int* err) {
  if (!mbar_wait(&B->hready[slot], P.hph[slot], &B->abort, err, kErrWaitMma)) return false;
  P.hph[slot] ^= 1u;
  tc_fence_after();
  return true;
}
// The products of `natoms` K-atoms: A from the slot's tile (atoms a0..),
// B from a stage (atoms b_atom_bytes apart), N = rows, into tensor column
// tcol; the first accumulates onto what is there when acc.
__device__ __forceinline__ void mma_atoms(uint32_t tcol, uint32_t sa, int a0, uint32_t sb, uint32_t b_atom_bytes,
                                          int natoms, int rows, bool acc) {
  const uint32_t idesc = idesc_bf16(128, rows, 0, 0);
  for (int a = 0; a < natoms; ++a)
    for (int kk = 0; kk < 4; ++kk) {
      const uint64_t ad = sw128_desc(sa + (a0 + a) * 16384u + kk * 32u, 16, 1024);
      const uint64_t bd = sw128_desc(sb + a * b_atom_bytes + kk * 32u, 16, 1024);
      mma_bf16(tcol, ad, bd, idesc, (acc || a > 0 || kk > 0) ? 1u : 0u);
    }
}

// Epilogue thread: this thread's shared-memory writes and tensor-memory
// reads of the slot are done; the producer may go on with it.
__device__ __forceinline__ void epi_arrive(uint64_t* bar) {
  fence_proxy_async();
  tc_fence_before();
  mbar_arrive(bar);
}

__global__ void __launch_bounds__(kIThreads, 1)
mlp_infer_kernel(const __grid_constant__ NetMaps nm, const InferArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t base = (saddr(smem_raw) + 1023u) & ~1023u;
  unsigned char* gbase = smem_raw + (base - saddr(smem_raw));
  IBars* B = reinterpret_cast<IBars*>(gbase + kIBar);
  float* spar = reinterpret_cast<float*>(gbase + kIPar);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int64_t tiles = (a.n + kTile - 1) / kTile;
  const int64_t G = gridDim.x;
  stage_params(a.p, spar);
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&B->full[i], 1);
      mbar_init(&B->empty[i], 1);
      mbar_init(&B->zready[i], 1);
      mbar_init(&B->hready[i], 256);
    }
    mbar_init(&B->fin, 1);
    B->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&B->tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t wbase = base + kIW;
  if (warp == 2 * kIEpi / 32) {
    // ---- producer: weights and products
    Prod P;
    bool ok = true;
    if ((tid & 31) == 0) {
      const CUtensorMap* w1 = &nm.m[kMapW1];
      const CUtensorMap* w2 = &nm.m[kMapW2];
      const CUtensorMap* w3 = &nm.m[kMapW3];
      for (int64_t tA = blockIdx.x; tA < tiles && ok; tA += 2 * G) {
        const bool hasB = tA + G < tiles;
        const int nslot = hasB ? 2 : 1;
        // L0: both K-atoms of W1 resident, the products of both slots
        ok = p_load(P, B, wbase, 0, w1, 0, 1, kIStage, a.err) && p_load(P, B, wbase, 1, w1, 1, 1, kIStage, a.err);
        ok = ok && p_wait(P, B, 0, a.err) && p_wait(P, B, 1, a.err);
        for (int sl = 0; sl < nslot && ok; ++sl) {
          ok = p_wait_operand(P, B, sl, a.err);
          if (!ok) break;
          const uint32_t tcol = B->tmem + 256u * sl, sa = base + sl * kIAct;
          mma_atoms(tcol, sa, 0, wbase, 0, 1, 256, false);
          mma_atoms(tcol, sa, 1, wbase + kIStage, 0, 1, 256, true);
          mma_commit(&B->zready[sl]);
        }
        if (!ok) break;
        p_release(P, B, 0);
        p_release(P, B, 1);
        // L1: the four K-atoms of W2 streamed through the stages, per slot
        for (int sl = 0; sl < nslot && ok; ++sl) {
          const uint32_t tcol = B->tmem + 256u * sl, sa = base + sl * kIAct;
          ok = p_load(P, B, wbase, 0, w2, 0, 1, kIStage, a.err) && p_load(P, B, wbase, 1, w2, 1, 1, kIStage, a.err);
          ok = ok && p_wait_operand(P, B, sl, a.err);
          for (int h = 0; h < 2 && ok; ++h) {
            if (h == 1)
              ok = p_load(P, B, wbase, 0, w2, 2, 1, kIStage, a.err) && p_load(P, B, wbase, 1, w2, 3, 1, kIStage, a.err);
            for (int st = 0; st < 2 && ok; ++st) {
              ok = p_wait(P, B, st, a.err);
              if (!ok) break;
              mma_atoms(tcol, sa, 2 * h + st, wbase + st * kIStage, 0, 1, 256, h + st > 0);
              p_release(P, B, st);
            }
          }
          if (ok) mma_commit(&B->zready[sl]);
        }
        if (!ok) break;
        // L2: W3 (16 rows, 4 K-atoms of 2 KB) in stage 0 for both slots
        ok = p_load(P, B, wbase, 0, w3, 0, 4, 16u * 128u, a.err) && p_wait(P, B, 0, a.err);
        for (int sl = 0; sl < nslot && ok; ++sl) {
          ok = p_wait_operand(P, B, sl, a.err);
          if (!ok) break;
          mma_atoms(B->tmem + 256u * sl, base + sl * kIAct, 0, wbase, 16u * 128u, 4, 16, false);
          mma_commit(&B->zready[sl]);
        }
        if (ok) p_release(P, B, 0);
      }
      if (!ok) atomicCAS(a.err, kErrNone, kErrWaitMma);
      // end: loads still in flight (only after an abort), then every product
      for (int st = 0; st < 2; ++st)
        if (P.inflight[st]) mbar_wait(&B->full[st], P.fph[st], &B->abort, a.err, kErrWaitLoad, false);
      mma_commit(&B->fin);
      mbar_wait(&B->fin, 0, &B->abort, a.err, kErrWaitMma, false);
    }
  } else {
    // ---- epilogue warps of slot sl: accumulator row, column half
    const int sl = tid / kIEpi, row = tid & (kTile - 1), half = (tid / kTile) & 1;
    const uint32_t trow = B->tmem + 256u * sl + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t act = base + sl * kIAct;
    uint32_t zph = 0;
    bool ok = true;
    auto zwait = [&] {
      ok = mbar_wait(&B->zready[sl], zph, &B->abort, a.err, kErrWaitMma);
      zph ^= 1u;
      tc_fence_after();
      return ok;
    };
    int64_t t = blockIdx.x + sl * G;
    if (t < tiles) {
      load_x<8>(spar, a.iquv, nullptr, t * kTile, a.n, a.nl, act, warp & 7);
      epi_arrive(&B->hready[sl]);
    }
    for (; t < tiles && ok; t += 2 * G) {
      const int64_t tn = t + 2 * G;   // this slot's next tile
      if (tn < tiles) prefetch_x(a.iquv, tn * kTile, a.n, a.nl, tid & (kIEpi - 1));
#pragma unroll 1
      for (int L = 0; L < 2; ++L) {
        if (!zwait()) break;
        hidden_epilogue<2>(trow, 0, spar + 256 * L, act, row, half, nullptr);
        epi_arrive(&B->hready[sl]);
      }
      if (!ok || !zwait()) break;
      // one warpgroup reads the outputs while the other loads the next tile
      float o[16];
      if (half == 0) tmem_ld16(trow, o);
      else if (tn < tiles) load_x<4>(spar, a.iquv, nullptr, tn * kTile, a.n, a.nl, act, warp & 3);
      if (tn < tiles) epi_arrive(&B->hready[sl]);
      const int64_t b = t * kTile + row;
      if (half == 0 && b < a.n) {
        float y[kOut];
#pragma unroll
        for (int j = 0; j < kOut; ++j) y[j] = (o[j] + a.p->b3[j]) * a.p->out_scale[j] + a.p->out_mean[j];
        double m[11];
        outputs_to_model(y, a.guess, a.fix, m);
#pragma unroll
        for (int i = 0; i < 11; ++i) a.models[b * 11 + i] = m[i];
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(B->tmem, 512);
}

// ---------------------------------------------------------------- training: forward + activation backward
// Per tile of the batch: X -> Z1 -> H1 -> Z2 -> H2 -> out, the loss and
// dOut = 2 (out - y) / (rows x 9), then dH2 = dOut W3, dZ2 = dH2 GELU'(Z2),
// dH1 = dZ2 W2, dZ1 = dH1 GELU'(Z1).  Tensor columns: Z1 0..255 (kept in
// zspill), Z2 256..511 (kept until dZ2), out 0..15, dH2 0..255, dH1
// 256..511.  X, H1, H2, dOut, dZ2, dZ1 go row-major to global memory (TMA
// stores of the operand tiles) for the weight gradients.
//
// Bound by one tile's chain of phases (a batch of 8192 has 64 tiles on 148
// SMs), so each is cut: 16 warps share the epilogues, the next two weight
// blocks load while an epilogue runs, Z1's spill is laid out by column group so
// that a warp's rows are neighbours, and a warp reads its rows of X in one
// batch.  65 -> 43.5 us for 8192 rows (8 warps; the spill a row per thread,
// 14 k of 96 k cycles each way; the second half of W2 loaded after the first
// half's products; X in two batches behind their indices, 19 k cycles).
__global__ void __launch_bounds__(kThreads, 1)
mlp_train_kernel(const __grid_constant__ NetMaps nm, const __grid_constant__ ActMaps am, const TrainKArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t base = (saddr(smem_raw) + 1023u) & ~1023u;
  Bars* B = reinterpret_cast<Bars*>(smem_raw + (base - saddr(smem_raw)) + kSBar);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = tid & (kTile - 1), part = tid / kTile;   // accumulator row, column quarter
  float* spar = reinterpret_cast<float*>(smem_raw + (base - saddr(smem_raw)) + kSPar);
  stage_params(a.p, spar);
  setup(B, 512);
  const uint32_t trow = B->tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const uint32_t sA = base + kSA, sD = base + kSD;
  const int64_t tiles = a.n / kTile;
  Pipe p;
  bool ok = true;
  // weight blocks of this CTA's tiles
  const int64_t blocks = (int64_t)blockIdx.x < tiles ? (tiles - 1 - blockIdx.x) / gridDim.x * kTrainJobs + kTrainJobs : 0;
  if (tid == 0) load_ahead(blocks, nm, B, base, p);
  for (int64_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
    const int64_t b = t * kTile + row;   // this thread's batch row
    float4* zrow = reinterpret_cast<float4*>(a.zspill) + t * (kTile * kHid / 4) + row;
    // the previous tile's stores must have read the operand tiles
    if (tid == 0) tma_store_wait_read();
    __syncthreads();
    load_x<16>(spar, a.iquv, a.idx, t * kTile, a.n, a.nl, sA, warp);
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      tma_store_2d(&am.x, 0, (int)(t * kTile), sA);
      tma_store_2d(&am.x, 64, (int)(t * kTile), sA + 16384u);
      tma_store_commit();
    }
    // five layers: 0 Z1, 1 Z2, 2 out, 3 dH2, 4 dH1
    for (int L = 0; L < 5 && ok; ++L) {
      if (tid == 0) {
        for (int j = layer_first(L); j < layer_last(L) && ok; ++j) ok = run_job(c_jobs[j], B, base, p, a.err);
      }
      ok = mbar_wait(&B->mma, p.mph, &B->abort, a.err, kErrWaitMma) && ok;
      p.mph ^= 1u;
      // both stages' products are done: the next loads run beside the epilogue;
      // an epilogue that overwrites the activation tile waits for its stores
      if (tid == 0 && ok) load_ahead(blocks, nm, B, base, p);
      if (tid == 0 && L != 2) tma_store_wait_read();
      __syncthreads();
      ok = ok && !B->abort;
      if (!ok) break;
      tc_fence_after();
      if (L == 0) {
        hidden_epilogue<4>(trow, 0, spar, sA, row, part, zrow);
      } else if (L == 1) {
        hidden_epilogue<4>(trow, 256, spar + 256, sA, row, part, nullptr);
      } else if (L == 2) {
        if (part == 0) {   // the 9 outputs: the first warpgroup
          float o[16];
          tmem_ld16(trow, o);
          const float* yt = a.y16 + (int64_t)a.idx[b] * 16;
          float sq = 0.f;
          float g[kOut];
#pragma unroll
          for (int j = 0; j < kOut; ++j) {
            const float d = o[j] + a.p->b3[j] - __ldg(yt + j);
            sq += d * d;
            g[j] = a.gscale * d;
          }
          uint32_t w[4] = {pack_bf16(g[0], g[1]), pack_bf16(g[2], g[3]), pack_bf16(g[4], g[5]),
                           pack_bf16(g[6], g[7])};
          st_chunk(sD, row, 0, w);
          w[0] = pack_bf16(g[8], 0.f);
          w[1] = w[2] = w[3] = 0u;
          st_chunk(sD, row, 1, w);
          w[0] = 0u;
#pragma unroll
          for (int j = 2; j < 8; ++j) st_chunk(sD, row, j, w);
#pragma unroll
          for (int o2 = 16; o2 > 0; o2 >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o2);
          if (lane == 0) atomicAdd(a.loss, sq);
        }
      } else {
        // dZ = dH GELU'(Z): L 3 -> dZ2 (dH2 at column 0, Z2 at 256);
        // L 4 -> dZ1 (dH1 at column 256, Z1 from the spill); this
        // warpgroup's quarter of the columns
#pragma unroll 1
        for (int q = 2 * part; q < 2 * part + 2; ++q) {
          float dh[32], z[32];
          if (L == 3) {
            tmem_ld32(trow + 32 * q, dh);
            tmem_ld32(trow + 256 + 32 * q, z);   // the product, without its bias
#pragma unroll
            for (int e = 0; e < 32; ++e) z[e] += spar[256 + 32 * q + e];
          } else {
            tmem_ld32(trow + 256 + 32 * q, dh);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const float4 v = zrow[(8 * q + u) * kTile];
              z[4 * u] = v.x;
              z[4 * u + 1] = v.y;
              z[4 * u + 2] = v.z;
              z[4 * u + 3] = v.w;
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t w[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int e = 8 * u + 2 * h;
              w[h] = pack_bf16(dh[e] * gelu_grad(z[e]), dh[e + 1] * gelu_grad(z[e + 1]));
            }
            st_chunk(sA + (q >> 1) * 16384u, row, (q & 1) * 4 + u, w);
          }
        }
      }
      fence_proxy_async();
      tc_fence_before();
      __syncthreads();
      tc_fence_after();
      // row-major copies for the weight gradients
      if (tid == 0) {
        const int y = (int)(t * kTile);
        const CUtensorMap* m = L == 0 ? &am.h1 : L == 1 ? &am.h2 : L == 2 ? &am.g3 : L == 3 ? &am.g2 : &am.g1;
        const uint32_t src = L == 2 ? sD : sA;
        const int natoms = L == 2 ? 1 : 4;
        for (int k = 0; k < natoms; ++k) tma_store_2d(m, 64 * k, y, src + 16384u * k);
        tma_store_commit();
      }
    }
  }
  teardown(B, p, 512, a.err);
}

// ---------------------------------------------------------------- training: weight and bias gradients
// The FP32 parameters of a gm_mlp in one flat index: w1, b1, w2, b2, w3, b3.
constexpr int kNW1 = kHid * kIn, kNW2 = kHid * kHid, kNW3 = kOut * kHid;
constexpr int kParams = kNW1 + kHid + kNW2 + kHid + kNW3 + kOut;
constexpr int kOffB1 = kNW1, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kNW2, kOffW3 = kOffB2 + kHid,
              kOffB3 = kOffW3 + kNW3;
constexpr int kPartStride = (kParams + 31) & ~31;   // a partial gradient; 16-byte stores into each
static_assert(kOffW2 % 4 == 0 && kPartStride % 4 == 0, "aligned blocks of the weights");

// One launch.  dW[m][n] = sum over a slice of the batch of A[b][m] Bm[b][n]
// for one 128 x 64 block; both operands row-major in global memory, MN-major
// in the product (8-row K groups 1024 bytes apart, 64-element M blocks 8 KB
// apart), 4-stage TMA ring.  Products: 0 dW1 = G1^T X (4 blocks), 1 dW2 =
// G2^T H1 (8 blocks), 2 dW3^T = H2^T dOut (2 blocks, stored transposed).  A
// slice's blocks fill one partial gradient, which the optimiser sums in
// order: the same gradient every time, where atomic additions into one
// differed from run to run.  Two warps of one block per M range add up the
// columns of its gradient operand as the stages pass, the bias gradients: a
// kernel of its own read the gradients again and took as long as this one
// (14.7 us a batch of 8192 rows).
struct WgradArgs {
  float* part;          // [kslices][kPartStride]
  int64_t rows;         // batch rows (a multiple of 64)
  int kslices;          // batch slices per block
  int* err;
};
struct WgradMaps {
  CUtensorMap a[3], b[3];   // boxes of 64 x 64 elements
};
constexpr int kWStages = 4;
constexpr uint32_t kWStageBytes = 16384 + 8192;   // A: 2 boxes (m 0..127), B: 1 box (n 0..63)
constexpr int kWBlocks = 14;
constexpr size_t kWgradSmem = kWStages * kWStageBytes + 256 + 1024;

__global__ void __launch_bounds__(kWThreads, 1)
mlp_wgrad_kernel(const __grid_constant__ WgradMaps wm, const WgradArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t base = (saddr(smem_raw) + 1023u) & ~1023u;
  struct WB {
    uint64_t full[kWStages], empty[kWStages], done;
    uint32_t tmem;
    int abort;
  };
  WB* B = reinterpret_cast<WB*>(smem_raw + (base - saddr(smem_raw)) + kWStages * kWStageBytes);
  const int tid = threadIdx.x, warp = tid >> 5;
  int blk = blockIdx.x;
  const int slice = blk % a.kslices;
  blk /= a.kslices;
  int g, mb, nb;
  if (blk < 4) {
    g = 0; mb = blk >> 1; nb = blk & 1;
  } else if (blk < 12) {
    g = 1; mb = (blk - 4) >> 2; nb = (blk - 4) & 3;
  } else {
    g = 2; mb = blk - 12; nb = 0;
  }
  // whose column sums this block forms: its A operand (G1, G2) or B (dOut)
  const bool bias = g < 2 ? nb == 0 : mb == 0;
  if (tid == 0) {
    for (int s = 0; s < kWStages; ++s) {
      mbar_init(&B->full[s], 1);
      mbar_init(&B->empty[s], bias ? 3 : 1);   // the products' commit and the two summing warps
    }
    mbar_init(&B->done, 1);
    B->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&B->tmem, 64);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const int64_t ksteps = a.rows / 64;
  const int64_t k0 = ksteps * slice / a.kslices, k1 = ksteps * (slice + 1) / a.kslices;
  const CUtensorMap* ma = &wm.a[g];
  const CUtensorMap* mbm = &wm.b[g];
  bool inflight[kWStages] = {false, false, false, false};
  uint32_t fph[kWStages] = {0, 0, 0, 0};
  if (tid == 0) {
    const uint32_t idesc = idesc_bf16(128, 64, 1, 1);
    uint32_t eph[kWStages] = {0, 0, 0, 0};
    bool pend[kWStages] = {false, false, false, false};
    bool ok = true;
    auto issue = [&](int64_t k) -> bool {
      const int s = (int)((k - k0) % kWStages);
      const uint32_t st = base + s * kWStageBytes;
      if (pend[s]) {
        if (!mbar_wait(&B->empty[s], eph[s], &B->abort, a.err, kErrWaitStage)) return false;
        eph[s] ^= 1u;
        pend[s] = false;
      }
      mbar_expect_tx(&B->full[s], kWStageBytes);
      tma_load_2d(st, ma, mb * 128, (int)(k * 64), &B->full[s]);
      tma_load_2d(st + 8192u, ma, mb * 128 + 64, (int)(k * 64), &B->full[s]);
      tma_load_2d(st + 16384u, mbm, nb * 64, (int)(k * 64), &B->full[s]);
      inflight[s] = true;
      return true;
    };
    for (int64_t k = k0; k < k1 && k < k0 + kWStages - 1 && ok; ++k) ok = issue(k);
    for (int64_t k = k0; k < k1 && ok; ++k) {
      const int s = (int)((k - k0) % kWStages);
      const uint32_t st = base + s * kWStageBytes;
      if (!mbar_wait(&B->full[s], fph[s], &B->abort, a.err, kErrWaitLoad)) {
        ok = false;
        break;
      }
      fph[s] ^= 1u;
      inflight[s] = false;
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        // 16 batch rows = two 8-row groups of 1024 bytes
        const uint64_t ad = sw128_desc(st + kk * 2048u, 8192, 1024);
        const uint64_t bd = sw128_desc(st + 16384u + kk * 2048u, 8192, 1024);
        mma_bf16(B->tmem, ad, bd, idesc, (k > k0 || kk > 0) ? 1u : 0u);
      }
      mma_commit(&B->empty[s]);
      pend[s] = true;
      if (k + kWStages - 1 < k1) ok = issue(k + kWStages - 1);
    }
    // the last commit covers every product issued (also after an abort)
    mma_commit(&B->done);
  } else if (bias && (warp == 1 || warp == 2)) {
    // two columns a thread, as 4 bytes of each swizzled 128-byte row
    const int u = tid - 32;
    const bool mine = g < 2 || u < kOut16 / 2;
    const uint32_t col = (g < 2 ? (uint32_t)(u >> 5) * 8192u : 16384u) + 4u * (u & 3);
    const uint32_t chunk = (uint32_t)(u & 31) >> 2;
    float s0 = 0.f, s1 = 0.f;
    for (int64_t k = k0; k < k1; ++k) {
      const int s = (int)((k - k0) % kWStages);
      if (!mbar_wait(&B->full[s], (uint32_t)((k - k0) / kWStages) & 1u, &B->abort, a.err, kErrWaitLoad)) break;
      if (mine) {
        const uint32_t st = base + s * kWStageBytes + col;
#pragma unroll 16
        for (uint32_t r = 0; r < 64; ++r) {
          uint32_t v;
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(st + r * 128u + ((chunk ^ (r & 7u)) << 4)));
          s0 += __uint_as_float(v << 16);
          s1 += __uint_as_float(v & 0xffff0000u);
        }
      }
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(&B->empty[s]);
    }
    const int c = g == 0 ? kOffB1 + mb * 128 + 2 * u : (g == 1 ? kOffB2 + mb * 128 + 2 * u : kOffB3 + 2 * u);
    float* part = a.part + (size_t)slice * kPartStride;
    if (mine && c < kParams) part[c] = s0;
    if (mine && c + 1 < kParams) part[c + 1] = s1;
  }
  __syncthreads();
  const bool ran = k1 > k0;
  bool ok = mbar_wait(&B->done, 0, &B->abort, a.err, kErrWaitMma, false) && ran;
  __syncthreads();
  ok = ok && !B->abort;
  if (ok) {
    tc_fence_after();
    const uint32_t trow = B->tmem + ((uint32_t)(warp * 32) << 16);
    const int m = mb * 128 + tid;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      float v[32];
      tmem_ld32(trow + 32 * h, v);
      float* part = a.part + (size_t)slice * kPartStride;
      if (g < 2) {
        // this thread's 32 columns are contiguous in its row of dW1 / dW2
        float4* dst = reinterpret_cast<float4*>(part + (g == 0 ? m * kIn : kOffW2 + m * kHid) + nb * 64 + 32 * h);
#pragma unroll
        for (int e = 0; e < 32; e += 4) dst[e / 4] = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
      } else if (h == 0) {
#pragma unroll
        for (int n = 0; n < kOut; ++n) part[kOffW3 + n * kHid + m] = v[n];
      }
    }
  }
  if (tid == 0)
    for (int s = 0; s < kWStages; ++s)
      if (inflight[s]) mbar_wait(&B->full[s], fph[s], &B->abort, a.err, kErrWaitLoad, false);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(B->tmem, 64);
}

// ---------------------------------------------------------------- parameters
__device__ __forceinline__ float* param_at(gm_mlp* p, int i, bool* bias) {
  *bias = false;
  if (i < kNW1) return &p->w1[0][0] + i;
  i -= kNW1;
  if (i < kHid) { *bias = true; return p->b1 + i; }
  i -= kHid;
  if (i < kNW2) return &p->w2[0][0] + i;
  i -= kNW2;
  if (i < kHid) { *bias = true; return p->b2 + i; }
  i -= kHid;
  if (i < kNW3) return &p->w3[0][0] + i;
  i -= kNW3;
  *bias = true;
  return p->b3 + i;
}

// The BF16 operand copies of parameter i (weights only); padding stays zero.
__device__ __forceinline__ void pack_one(const gm_mlp* p, uint16_t* pack, int i) {
  if (i < kNW1) {
    const int o = i / kIn, c = i % kIn;
    pack[kW1b + o * kIn + c] = __bfloat16_as_ushort(__float2bfloat16_rn(p->w1[o][c]));
    return;
  }
  i -= kNW1 + kHid;
  if (i >= 0 && i < kNW2) {
    const int o = i / kHid, c = i % kHid;
    const uint16_t v = __bfloat16_as_ushort(__float2bfloat16_rn(p->w2[o][c]));
    pack[kW2b + o * kHid + c] = v;
    pack[kW2tb + c * kHid + o] = v;
    return;
  }
  i -= kNW2 + kHid;
  if (i >= 0 && i < kNW3) {
    const int o = i / kHid, c = i % kHid;
    const uint16_t v = __bfloat16_as_ushort(__float2bfloat16_rn(p->w3[o][c]));
    pack[kW3b + o * kHid + c] = v;
    pack[kW3tb + c * kG + o] = v;
  }
}

__global__ void mlp_pack_kernel(const gm_mlp* p, uint16_t* pack) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x) pack_one(p, pack, i);
}

// Gradient of flat parameter i: the sum of its partials in order.
__device__ __forceinline__ float grad_at(const float* __restrict__ part, int slices, int i) {
  float g = 0.f;
#pragma unroll 8
  for (int k = 0; k < slices; ++k) g += __ldg(part + (size_t)k * kPartStride + i);
  return g;
}

// The gradient of a batch as a gm_mlp (checks).
__global__ void mlp_grad_kernel(const float* part, int slices, gm_mlp* grad) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x) {
    bool bias;
    float* g = param_at(grad, i, &bias);
    *g = grad_at(part, slices, i);
  }
}

// Adam with decoupled weight decay (weights only) on every parameter, its
// BF16 copy rewritten.  c1, c2: the bias corrections 1 / (1 - beta^t).
__global__ void mlp_adam_kernel(gm_mlp* p, const float* part, int slices, gm_mlp* m1, gm_mlp* m2,
                                uint16_t* pack, float lr, float wd, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x) {
    bool bias;
    float* w = param_at(p, i, &bias);
    float* ma = param_at(m1, i, &bias);
    float* mb = param_at(m2, i, &bias);
    const float gv = grad_at(part, slices, i);
    const float av = 0.9f * *ma + 0.1f * gv;
    const float bv = 0.999f * *mb + 0.001f * gv * gv;
    *ma = av;
    *mb = bv;
    *w -= lr * ((av * c1) / (sqrtf(bv * c2) + 1e-8f) + (bias ? 0.f : wd * *w));
    pack_one(p, pack, i);
  }
}

// The 9 outputs that stand for a model (Init_Model layout).
__device__ __forceinline__ void model_targets(const double* __restrict__ m, double (&v)[kOut]) {
  const double g = m[5] * (3.14159265358979323846 / 180.0);
  const double ph = 2.0 * m[6] * (3.14159265358979323846 / 180.0);
  v[0] = m[0];
  v[1] = m[2];
  v[2] = m[3];
  v[3] = m[4];
  v[4] = m[7];
  v[5] = m[8];
  v[6] = m[1] * cos(g);
  v[7] = m[1] * sin(g) * cos(ph);
  v[8] = m[1] * sin(g) * sin(ph);
}

// Standardised targets [n][16] of the models [n][11] (the 9 outputs, then
// zeros).
__global__ void mlp_targets_kernel(const double* __restrict__ truth, int64_t n, const gm_mlp* p, float* y16) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double v[kOut];
    model_targets(truth + i * 11, v);
    for (int j = 0; j < 16; ++j)
      y16[i * 16 + j] = j < kOut ? (float)((v[j] - p->out_mean[j]) / p->out_scale[j]) : 0.f;
  }
}

// Standardisation of inputs and targets from the first m pixels (at most
// 65 536): sums and sums of squares of every feature and target in double,
// per block (mlp_moments_kernel, thread f of a row group owns feature f, a
// row's features read together; the targets a pixel per thread), then the
// blocks' in order and the mean and scale into the network
// (mlp_standardise_kernel).  Bound by the read of the pixels (31 MB at 30
// samples); copied to the host and summed there they took about 28 of the
// 39 ms of a training call, here 0.05 ms.
constexpr int kMomBlocks = 148, kMomThreads = 256, kMom = kIn + kOut16;
__global__ void __launch_bounds__(kMomThreads)
mlp_moments_kernel(const float* __restrict__ iquv, const double* __restrict__ truth, int64_t m, int nl,
                   double2* __restrict__ part) {
  __shared__ double2 sh[kMomThreads / 32][kOut];
  __shared__ double2 sx[kIn];
  const int t = threadIdx.x, f = t & (kIn - 1), g = t / kIn, F = 4 * nl;
  constexpr int G = kMomThreads / kIn;
  double s = 0.0, ss = 0.0;
  if (f < F) {
#pragma unroll 4
    for (int64_t r = (int64_t)blockIdx.x * G + g; r < m; r += (int64_t)gridDim.x * G) {
      const double v = (double)__ldg(iquv + r * F + f);
      s += v;
      ss += v * v;
    }
  }
  if (g == 1) sx[f] = make_double2(s, ss);
  double ys[kOut] = {}, yss[kOut] = {};
  for (int64_t r = (int64_t)blockIdx.x * kMomThreads + t; r < m; r += (int64_t)gridDim.x * kMomThreads) {
    double v[kOut];
    model_targets(truth + r * 11, v);
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
      const double y = (double)(float)v[j];
      ys[j] += y;
      yss[j] += y * y;
    }
  }
#pragma unroll
  for (int j = 0; j < kOut; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ys[j] += __shfl_xor_sync(0xffffffffu, ys[j], o);
      yss[j] += __shfl_xor_sync(0xffffffffu, yss[j], o);
    }
    if ((t & 31) == 0) sh[t >> 5][j] = make_double2(ys[j], yss[j]);
  }
  __syncthreads();
  if (g == 0) part[(size_t)blockIdx.x * kMom + f] = make_double2(s + sx[f].x, ss + sx[f].y);
  if (t < kOut) {
    double2 a = sh[0][t];
    for (int w = 1; w < kMomThreads / 32; ++w) {
      a.x += sh[w][t].x;
      a.y += sh[w][t].y;
    }
    part[(size_t)blockIdx.x * kMom + kIn + t] = a;
  }
}
static_assert(kMomThreads == 2 * kIn, "two row groups a block");

__global__ void __launch_bounds__(kMom)
mlp_standardise_kernel(const double2* __restrict__ part, int blocks, int64_t m, int nl, gm_mlp* p) {
  const int f = threadIdx.x;
  double s = 0.0, ss = 0.0;
  const bool used = f < 4 * nl || (f >= kIn && f < kIn + kOut);
  if (used) {
#pragma unroll 8
    for (int b = 0; b < blocks; ++b) {
      const double2 v = part[(size_t)b * kMom + f];
      s += v.x;
      ss += v.y;
    }
  }
  const double mu = s / (double)m, d = __dsub_rn(ss / (double)m, __dmul_rn(mu, mu)), var = d < 0.0 ? 0.0 : d;
  if (f < kIn) {
    p->in_mean[f] = used ? (float)mu : 0.f;
    p->in_scale[f] = used && var > 1e-20 ? (float)(1.0 / sqrt(var)) : 0.f;
  } else {
    p->out_mean[f - kIn] = used ? (float)mu : 0.f;
    p->out_scale[f - kIn] = used && var > 1e-20 ? (float)sqrt(var) : 1.f;
  }
}

// An epoch's visiting order: a pseudo-random permutation of [0, n) drawn on
// the device, so that no host shuffle or copy sits between epochs.  A
// 4-round Feistel network on 2 hb bits (2^(2 hb) >= n), its round function
// the MurmurHash3 finaliser of (half ^ round key), restricted to [0, n) by
// cycle walking (Black & Rogaway, "Ciphers with arbitrary finite domains",
// 2002): re-applying the bijection until the value falls inside keeps the
// map one to one and ends within the cycle of i, fewer than 4 n steps
// (expected under 4).  hb = 0 writes the identity.
__device__ __forceinline__ uint32_t fmix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x85ebca6bu;
  x ^= x >> 13;
  x *= 0xc2b2ae35u;
  x ^= x >> 16;
  return x;
}

__global__ void mlp_order_kernel(uint32_t* __restrict__ idx, uint32_t n, int hb, uint64_t key) {
  const uint32_t mask = hb ? (1u << hb) - 1u : 0u;
  const uint64_t cap = 4ull * n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t x = i;
    if (hb) {
      uint64_t walk = 0;
      do {
        uint32_t l = x >> hb, r = x & mask;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t f = fmix32(r ^ (uint32_t)(key >> (16 * k)) ^ (0x9e3779b9u * (uint32_t)(k + 1))) & mask;
          const uint32_t t = l ^ f;
          l = r;
          r = t;
        }
        x = (l << hb) | r;
      } while (x >= n && ++walk < cap);
    }
    idx[i] = x;
  }
}

// ---------------------------------------------------------------- host
namespace {

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }
  return fn;
}

// 2-D BF16 map of a row-major [rows][cols] matrix, boxes of 64 columns x
// box_rows rows, 128-byte swizzle.
bool make_map(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint32_t box_rows) {
  auto enc = encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool net_maps(const uint16_t* pack, NetMaps* nm) {
  return make_map(&nm->m[kMapW1], pack + kW1b, kIn, kHid, 256) &&
         make_map(&nm->m[kMapW2], pack + kW2b, kHid, kHid, 256) &&
         make_map(&nm->m[kMapW3], pack + kW3b, kHid, kOut16, 16) &&
         make_map(&nm->m[kMapW2t], pack + kW2tb, kHid, kHid, 256) &&
         make_map(&nm->m[kMapW3t], pack + kW3tb, kG, kHid, 256);
}

int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 1;
}

// The buffers of a training call, carved from one block of device memory in
// 256-byte steps; without memory it only adds up what they need.
struct Carver {
  char* base;
  size_t used = 0;
  template <typename T>
  T* get(size_t count) {
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += (sizeof(T) * count + 255) & ~(size_t)255;
    return p;
  }
};

struct TrainBufs {
  gm_mlp *grad, *m1, *m2;
  uint16_t *x, *h1, *h2, *g1, *g2, *g3;
  float *z, *y16, *loss, *gpart;
  uint32_t* idx;
  double2* part;
  size_t bytes;
};
// one product block per SM; two (twice the slices) leave the products at
// 13.5 us and make the optimiser sum twice as many partials, 8.7 us for 6.6
int grad_slices(int64_t B, int sms) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(B / 64, sms / kWBlocks));
}
TrainBufs carve(void* base, int64_t n, int64_t B, int slices) {
  Carver c{static_cast<char*>(base)};
  TrainBufs b{};
  b.grad = c.get<gm_mlp>(1);
  b.m1 = c.get<gm_mlp>(1);
  b.m2 = c.get<gm_mlp>(1);
  b.x = c.get<uint16_t>((size_t)B * kIn);
  b.h1 = c.get<uint16_t>((size_t)B * kHid);
  b.h2 = c.get<uint16_t>((size_t)B * kHid);
  b.g1 = c.get<uint16_t>((size_t)B * kHid);
  b.g2 = c.get<uint16_t>((size_t)B * kHid);
  b.g3 = c.get<uint16_t>((size_t)B * kG);
  b.z = c.get<float>((size_t)B * kHid);
  b.y16 = c.get<float>((size_t)n * 16);
  b.idx = c.get<uint32_t>((size_t)n);
  b.loss = c.get<float>(1);
  b.part = c.get<double2>((size_t)kMomBlocks * kMom);
  b.gpart = c.get<float>((size_t)slices * kPartStride);
  b.bytes = c.used;
  return b;
}

}  // namespace

void init_net(gm_mlp* net, int nl, uint64_t seed) {
  std::memset(net, 0, sizeof(*net));
  net->abi_version = GM_ABI_VERSION;
  net->nl = nl;
  for (int f = 0; f < kIn; ++f) net->in_scale[f] = f < 4 * nl ? 1.f : 0.f;
  for (int j = 0; j < kOut16; ++j) net->out_scale[j] = 1.f;
  std::mt19937_64 rng(seed);
  auto fill = [&](float* w, int fan_out, int fan_in, int used_in, float gain) {
    const float a = gain * std::sqrt(6.f / (float)used_in);   // variance 2 / fan-in
    std::uniform_real_distribution<float> u(-a, a);
    for (int o = 0; o < fan_out; ++o)
      for (int i = 0; i < fan_in; ++i) w[o * fan_in + i] = i < used_in ? u(rng) : 0.f;
  };
  fill(&net->w1[0][0], kHid, kIn, 4 * nl, 1.f);
  fill(&net->w2[0][0], kHid, kHid, kHid, 1.f);
  fill(&net->w3[0][0], kOut, kHid, kHid, 0.1f);   // outputs start near the mean
}

cudaError_t devnet_load(DevNet* d, const gm_mlp* host, cudaStream_t s) {
  cudaError_t e = cudaMemcpyAsync(d->p, host, sizeof(gm_mlp), cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return e;
  mlp_pack_kernel<<<256, 256, 0, s>>>(d->p, d->pack);
  d->nl = host->nl;
  return cudaGetLastError();
}

cudaError_t devnet_create(DevNet* d, const gm_mlp* host, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  if (!d->p) {
    DevNet n;
    e = cudaMalloc(&n.p, sizeof(gm_mlp));
    if (e == cudaSuccess) e = cudaMalloc(&n.pack, sizeof(uint16_t) * kPackElems);
    // the copies' padding stays zero
    if (e == cudaSuccess) e = cudaMemsetAsync(n.pack, 0, sizeof(uint16_t) * kPackElems, s);
    NetMaps nm;
    if (e == cudaSuccess && !net_maps(n.pack, &nm)) e = cudaErrorInvalidValue;
    if (e != cudaSuccess) {
      devnet_destroy(&n);
      return e;
    }
    n.mw1 = nm.m[kMapW1];
    n.mw2 = nm.m[kMapW2];
    n.mw3 = nm.m[kMapW3];
    n.mw2t = nm.m[kMapW2t];
    n.mw3t = nm.m[kMapW3t];
    *d = n;
  }
  return devnet_load(d, host, s);
}

void devnet_destroy(DevNet* d) {
  if (d->p) cudaFree(d->p);
  if (d->pack) cudaFree(d->pack);
  *d = DevNet{};
}

cudaError_t predict(const DevNet& d, const float* iquv, int64_t n, int nl, const double* guess, const int* fix,
                    double* models, int* err, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (nl != d.nl || 4 * nl > kIn || !err) return cudaErrorInvalidValue;
  // the input tiles are read in 16-byte vectors
  if (reinterpret_cast<uintptr_t>(iquv) & 15u) return cudaErrorInvalidValue;
  NetMaps nm;
  nm.m[kMapW1] = d.mw1;
  nm.m[kMapW2] = d.mw2;
  nm.m[kMapW3] = d.mw3;
  nm.m[kMapW2t] = d.mw2t;
  nm.m[kMapW3t] = d.mw3t;
  InferArgs a{};
  a.p = d.p;
  a.iquv = iquv;
  a.n = n;
  a.nl = nl;
  for (int i = 0; i < 11; ++i) {
    a.guess[i] = guess[i];
    a.fix[i] = fix ? fix[i] : 1;
  }
  a.models = models;
  a.err = err;
  cudaError_t e =
      cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kISmemBytes);
  if (e != cudaSuccess) return e;
  const int64_t tiles = (n + kTile - 1) / kTile;
  const int grid = (int)std::min<int64_t>(tiles, sm_count());
  mlp_infer_kernel<<<grid, kIThreads, kISmemBytes, s>>>(nm, a);
  return cudaGetLastError();
}

size_t train_bytes(int64_t n, int64_t batch) {
  return carve(nullptr, n, batch, grad_slices(batch, sm_count())).bytes;
}

cudaError_t train(gm_mlp* net, const TrainArgs& a, DevNet& d, void* ws, size_t ws_bytes, float* loss_out,
                  gm_mlp* grads_out, int* err, cudaStream_t s, const char** why) {
  auto fail = [&](const char* w, cudaError_t e) {
    if (why) *why = w;
    return e;
  };
  const int64_t B = a.grads_only ? a.n : (int64_t)a.batch;
  if (B <= 0 || B % kTile || a.n < B || B > (int64_t)1 << 30)
    return fail("the batch must be a positive multiple of 128 and at most the pixel count", cudaErrorInvalidValue);
  if (a.n > (int64_t)1 << 31) return fail("at most 2^31 training pixels", cudaErrorInvalidValue);
  if (a.nl < 1 || 4 * a.nl > kIn || net->nl != a.nl) return fail("the network's grid differs", cudaErrorInvalidValue);
  if (!err) return fail("no error word", cudaErrorInvalidValue);
  if (reinterpret_cast<uintptr_t>(a.iquv) & 15u)
    return fail("the profiles must start on a 16-byte boundary", cudaErrorInvalidValue);
  const int64_t n = a.n;
  const int sms = sm_count();
  const int64_t tiles = B / kTile;
  const int tgrid = (int)std::min<int64_t>(tiles, sms);
  const int kslices = grad_slices(B, sms);
  const TrainBufs buf = carve(ws, n, B, kslices);
  if (!ws || ws_bytes < buf.bytes) return fail("no workspace", cudaErrorInvalidValue);
  gm_mlp *grad = buf.grad, *m1 = buf.m1, *m2 = buf.m2;
  uint16_t *x = buf.x, *h1 = buf.h1, *h2 = buf.h2, *g1 = buf.g1, *g2 = buf.g2, *g3 = buf.g3;
  float *z = buf.z, *y16 = buf.y16, *loss = buf.loss, *gpart = buf.gpart;
  uint32_t* idx = buf.idx;
  cudaError_t e = devnet_create(&d, net, s);
  if (e != cudaSuccess) return fail("network upload", e);
  cudaMemsetAsync(grad, 0, sizeof(gm_mlp), s);
  cudaMemsetAsync(m1, 0, sizeof(gm_mlp), s);
  cudaMemsetAsync(m2, 0, sizeof(gm_mlp), s);
  NetMaps nm;
  ActMaps am;
  WgradMaps wm;
  bool maps = net_maps(d.pack, &nm) && make_map(&am.x, x, kIn, B, 128) && make_map(&am.h1, h1, kHid, B, 128) &&
              make_map(&am.h2, h2, kHid, B, 128) && make_map(&am.g3, g3, kG, B, 128) &&
              make_map(&am.g2, g2, kHid, B, 128) && make_map(&am.g1, g1, kHid, B, 128) &&
              make_map(&wm.a[0], g1, kHid, B, 64) && make_map(&wm.b[0], x, kIn, B, 64) &&
              make_map(&wm.a[1], g2, kHid, B, 64) && make_map(&wm.b[1], h1, kHid, B, 64) &&
              make_map(&wm.a[2], h2, kHid, B, 64) && make_map(&wm.b[2], g3, kG, B, 64);
  if (!maps) return fail("tensor-map encoding", cudaErrorInvalidValue);
  if (net->steps == 0 && !a.grads_only) {
    const int64_t m = std::min<int64_t>(n, 65536);
    mlp_moments_kernel<<<kMomBlocks, kMomThreads, 0, s>>>(a.iquv, a.truth, m, a.nl, buf.part);
    mlp_standardise_kernel<<<1, kMom, 0, s>>>(buf.part, kMomBlocks, m, a.nl, d.p);
  }
  mlp_targets_kernel<<<1024, 256, 0, s>>>(a.truth, n, d.p, y16);
  e = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(mlp_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgradSmem);
  if (e != cudaSuccess) return fail("kernel attributes", e);
  const int epochs = a.grads_only ? 1 : std::max(1, a.epochs);
  const int64_t steps_per_epoch = n / B;
  const int64_t total = steps_per_epoch * epochs;
  // visiting order: the identity for a gradient check, else a fresh
  // permutation per epoch keyed by the seed
  int hb = 0;
  if (!a.grads_only)
    while ((uint64_t)1 << (2 * hb) < (uint64_t)n) ++hb;
  std::mt19937_64 rng(a.seed);
  const int order_blocks = (int)std::min<int64_t>((n + 255) / 256, 4 * (int64_t)sm_count());
  int64_t step = 0;
  int64_t t_adam = net->steps;
  for (int ep = 0; ep < epochs && e == cudaSuccess; ++ep) {
    mlp_order_kernel<<<order_blocks, 256, 0, s>>>(idx, (uint32_t)n, hb, rng());
    e = cudaMemsetAsync(loss, 0, sizeof(float), s);
    for (int64_t st = 0; st < steps_per_epoch && e == cudaSuccess; ++st, ++step) {
      TrainKArgs ka{};
      ka.p = d.p;
      ka.iquv = a.iquv;
      ka.y16 = y16;
      ka.idx = idx + st * B;
      ka.n = B;
      ka.nl = a.nl;
      ka.gscale = 2.f / (float)(B * kOut);
      ka.zspill = z;
      ka.loss = loss;
      ka.err = err;
      mlp_train_kernel<<<tgrid, kThreads, kSmemBytes, s>>>(nm, am, ka);
      WgradArgs wa{};
      wa.part = gpart;
      wa.rows = B;
      wa.kslices = kslices;
      wa.err = err;
      mlp_wgrad_kernel<<<kWBlocks * kslices, kWThreads, kWgradSmem, s>>>(wm, wa);
      if (!a.grads_only) {
        ++t_adam;
        const double lr = a.lr * 0.5 * (1.0 + std::cos(M_PI * (double)step / (double)std::max<int64_t>(1, total)));
        const float c1 = (float)(1.0 / (1.0 - std::pow(0.9, (double)t_adam)));
        const float c2 = (float)(1.0 / (1.0 - std::pow(0.999, (double)t_adam)));
        mlp_adam_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(d.p, gpart, kslices, m1, m2, d.pack, (float)lr,
                                                              a.weight_decay, c1, c2);
      }
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && loss_out) {
      float sum = 0.f;
      e = cudaMemcpyAsync(&sum, loss, sizeof(float), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      loss_out[ep] = sum / (float)((double)steps_per_epoch * B * kOut);
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  int code = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&code, err, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && code != 0) e = cudaErrorLaunchTimeout;
  if (e == cudaSuccess) {
    const int64_t steps0 = net->steps;
    if (a.grads_only) {
      if (grads_out) {
        mlp_grad_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(gpart, kslices, grad);
        e = cudaMemcpyAsync(grads_out, grad, sizeof(gm_mlp), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      }
    } else {
      e = cudaMemcpy(net, d.p, sizeof(gm_mlp), cudaMemcpyDeviceToHost);
      net->steps = steps0 + total;
    }
  }
  return e == cudaSuccess ? e : fail(code ? "a training kernel gave up waiting" : "training", e);
}

}  // namespace mlp
}  // namespace gm
