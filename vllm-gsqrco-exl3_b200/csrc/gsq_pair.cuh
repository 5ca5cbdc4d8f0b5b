// What the GEMMs on pairs of CTAs share (gsq_gemm4.cu, gsq_gemm6.cu): ring positions, bounded waits, arrivals on the other
// CTA's barriers, operand descriptors of the layout in gsq_planes.cuh, tensor-memory loads.
#pragma once
#include "gsq_tc.cuh"

namespace gsq {
namespace pl {

using namespace tc;

constexpr int SMEM_MAX = 227 * 1024;
constexpr int G_THREADS = 384;
constexpr int CONS_WARP0 = 4, CONS_WARPS = 8;
constexpr int IDLE_REGS = 40, CONS_REGS = 232;   // 128 x 40 + 256 x 232 = the 384 x 168 the block is launched with
constexpr int MAX_STAGES = 8;
constexpr int G_TMEM = 512;
constexpr int SMEM_HEAD = 1024;                  // barriers; the stages start 1024-byte aligned
constexpr int ROW_GROUP = 8;                     // row tiles of a rasterisation group

static __device__ int pair_error = 0;            // sticky, one per translation unit: a wait gave up

struct Cursor {
  uint32_t i, ph;
  __device__ __forceinline__ void next(uint32_t n) {
    if (++i == n) { i = 0; ph ^= 1u; }
  }
};

// Bounded: gives up about a second after the first failed try (SM clocks; the global timer takes about a microsecond to
// read), or when another thread of the CTA has. The hardware suspends a waiting thread inside try_wait.
__device__ __forceinline__ bool try_bar(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (try_bar(bar, parity)) return true;
  const long long t0 = clock64();
  for (int spin = 1; spin < (1 << 28); ++spin) {
    if (try_bar(bar, parity)) return true;
    if ((spin & 15) == 0 && (*abort_flag || clock64() - t0 > 2000000000ll)) break;
  }
  if (!*abort_flag) {
    *abort_flag = 1;
    atomicExch(&pair_error, 1);
  }
  return false;
}

// Arrival on a barrier of the other CTA. No cluster-scope release: it would wait for every outstanding store of the SM
// (about 1000 cycles under this kernel's traffic, on every stage), and nothing here is handed over through ordinary
// stores -- what the waiting side uses are bytes that bulk copies have landed and tensor-memory reads that have completed.
__device__ __forceinline__ void arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// K-major tile of 8-row groups of 1024 bytes under the 128-byte swizzle; one MMA (K = 16) takes 32 bytes of a row, the
// next one starts 32 bytes further
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
  uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xFFFFFFFF;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0;
}
// the MMAs issued so far have completed -> one arrival on the barrier at this offset in each CTA of the pair
__device__ __forceinline__ void commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, "
      "%28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
        "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
        "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
// what follows may not use the loaded registers before this point (the wait above it)
__device__ __forceinline__ void pin32(uint32_t* v) {
#pragma unroll
  for (int i = 0; i < 32; i += 8)
    asm volatile("" : "+r"(v[i]), "+r"(v[i + 1]), "+r"(v[i + 2]), "+r"(v[i + 3]), "+r"(v[i + 4]), "+r"(v[i + 5]), "+r"(v[i + 6]), "+r"(v[i + 7]));
}

// Item -> pair of row tiles, token block and superblocks [sb0, sb1): groups of ROW_GROUP row tiles, token blocks inside; the
// parts of K of a tile run side by side.
__device__ __forceinline__ void place_item(int item, int splits, int nsb, int n_tb, int n_rp, int& rp, int& tb, int& sb0, int& sb1) {
  const int split = splits > 1 ? item % splits : 0;
  if (splits > 1) item /= splits;
  sb0 = split * nsb / splits;
  sb1 = (split + 1) * nsb / splits;
  const int per = ROW_GROUP * n_tb, grp = item / per, rem = item - grp * per;
  const int in_grp = min(ROW_GROUP, n_rp - grp * ROW_GROUP);
  tb = rem / in_grp;
  rp = grp * ROW_GROUP + rem - tb * in_grp;
}

// One persistent pair per item, at most as many as the device runs at once (max_pairs: kept per device and kernel).
template <typename G>
static int launch_pairs(void (*kern)(G), int threads, const G& g, std::atomic<int> (&max_pairs)[64], int64_t items, int smem, int sm_count, cudaStream_t st) {
  int dev = 0;
  GSQ_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return GSQ_ERR_UNSUPPORTED;
  if (items > INT32_MAX) return GSQ_ERR_TOO_LARGE;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = st;
  if (!max_pairs[dev]) {
    GSQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
    // (an SM without a free neighbour in its GPC stays out)
    cudaLaunchAttribute ca;
    ca.id = cudaLaunchAttributeClusterDimension;
    ca.val.clusterDim.x = 2;
    ca.val.clusterDim.y = 1;
    ca.val.clusterDim.z = 1;
    cfg.gridDim = dim3(2u * (unsigned)sm_count);
    cfg.dynamicSmemBytes = SMEM_MAX;
    cfg.attrs = &ca;
    cfg.numAttrs = 1;
    int n = 0;
    GSQ_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
    if (n < 1) return GSQ_ERR_UNSUPPORTED;
    max_pairs[dev] = n;
  }
  const int most = max_pairs[dev];
  cfg.gridDim = dim3(2u * (unsigned)(items < most ? items : most));
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, g));
  return GSQ_OK;
}

}  // namespace pl
}  // namespace gsq
