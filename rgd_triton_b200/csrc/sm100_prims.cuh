// Blackwell (sm_100a) primitives used by the tensor-memory attention kernels:
// mbarriers with BOUNDED waits, TMA tiled loads, tcgen05 tensor-memory
// allocation, MMA issue / commit, tensor-memory loads and stores, and the
// shared-memory / instruction descriptors the MMA consumes.  Inline PTX only.
#pragma once

#include <cuda.h>   // CUtensorMap (types only; the encoder is fetched at run time)

#include "common.cuh"

namespace rgd {
namespace sm100 {

// ---------------------------------------------------------------------------
// Device status word.  Any bounded wait that runs out stores a non-zero code
// here and every other wait in flight sees it and gives up too, so a kernel
// whose pipeline broke ends in bounded time with its tensor memory released.
// ---------------------------------------------------------------------------
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;   // 2 s per wait

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Wait for the phase with the given parity to complete.  Returns false when
// the wait was abandoned (time limit, or another thread already flagged an
// error in *status); `code` identifies the waiting site.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *status, int code,
                                          unsigned long long limit_ns = WAIT_LIMIT_NS) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = globaltimer_ns();
    for (uint32_t i = 1;; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 0u) {
            if (*reinterpret_cast<volatile int *>(status) != 0) return false;
            if (globaltimer_ns() - t0 > limit_ns) {
                atomicCAS(status, 0, code);
                return false;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Order in which a 1-D grid walks the (batch, head) x tile-block pairs.  Without a causal mask the
// blocks of one head run next to each other (they share its K and V in L2).  Under a causal mask the
// work per block differs, and the blocks of `group` heads are interleaved by rank, heaviest rank
// first, so that the last CTAs to start are the lightest ones.  A group has as many heads as 48 MB hold
// the shared operands of, rounded so that all groups are about equal (a last group of a few heads is a
// tail of its own).  Forward / forward + backward in us, measured in turns:
//                            one head   12 MB       24 MB       48 MB       96 MB    48 MB, ragged last group
//   [2, 3001, 16, 128]       117 / 453  101 / 418   97 / 416    97 / 417    97 / 417    97 / 417
//   [2, 4608, 24, 64]        271 / 901  252 / 850   238 / 833   237 / 830   236 / 832   268 / 876
//   [2, 2600, 20, 128]       121 / 456  113 / 434   110 / 431   103 / 424   100 / 424   123 / 465
//   [2, 4096, 24, 128]       278 / 1138 261 / 1097  248 / 1088  247 / 1081  248 / 1099  242 / 1080
// ---------------------------------------------------------------------------
struct TileOrder {
    int nblk, group, BH;
};
__device__ __forceinline__ void tile_of(const TileOrder &o, int &rank, int &bh) {
    const int per = o.nblk * o.group;
    const int g = (int)blockIdx.x / per, rem = (int)blockIdx.x - g * per;
    const int heads = min(o.group, o.BH - g * o.group);
    rank = rem / heads;
    bh = g * o.group + rem - rank * heads;
}
inline TileOrder make_tile_order(int nblk, int BH, bool causal, int64_t bytes_per_head) {
    if (!causal || BH <= 0) return {nblk, 1, BH};
    const int64_t fit = (48ll << 20) / (bytes_per_head > 0 ? bytes_per_head : 1);
    const int most = (int)(fit < 1 ? 1 : fit > BH ? BH : fit), groups = (BH - 1) / most + 1;
    return {nblk, (BH - 1) / groups + 1, BH};
}

// Programmatic dependent launch: a kernel launched with launch_pdl may start while its predecessor in
// the stream still runs; grid_wait() returns once the predecessor has completed and its writes are
// visible, grid_trigger() (every CTA) allows the successor to start.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... Params, typename... Args>
inline int launch_pdl_cluster(void (*kernel)(Params...), dim3 grid, int cluster_x, int threads, size_t smem, cudaStream_t st,
                              Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attrs[2]{};
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = cluster_x;
    attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = cluster_x > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
    count_launch();
    return cuda_status(e);
}
template <typename... Params, typename... Args>
inline int launch_pdl(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    return launch_pdl_cluster(kernel, grid, 1, threads, smem, st, args...);
}

// ---------------------------------------------------------------------------
// TMA: tiled 4-D load global -> shared, completion on an mbarrier.  No
// multicast: every CTA fetches its own tiles from this GPU's memory.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_4d(void *smem_dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1,
                                            int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
// Untiled bulk copy global -> shared; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_load_1d(void *smem_dst, const void *gsrc, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---------------------------------------------------------------------------
// Tensor memory (TMEM)
// ---------------------------------------------------------------------------
// Warp-collective.  ncols: power of two in [32, 512].  The base address is
// written to *smem_result.
__device__ __forceinline__ void tmem_alloc(uint32_t *smem_result, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp gets columns
// [col, col+32) of TMEM lane (32 * (warp % 4) + i).  Warp-collective.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
          "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]),
          "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// ---------------------------------------------------------------------------
// MMA descriptors
// ---------------------------------------------------------------------------
// Instruction descriptor for kind::f16 (fp16 / bf16 operands, fp32 accumulate):
// bits [4,6) accumulator format (1 = f32), [7,10) A format, [10,13) B format
// (0 = f16, 1 = bf16), bit 15 / 16 A / B major (0 = K-major, 1 = MN-major),
// [17,23) N >> 3, [24,29) M >> 4.
__host__ __device__ constexpr uint32_t make_idesc(bool bf16, int M, int N, bool a_mn_major, bool b_mn_major) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
           ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Shared-memory matrix descriptor, 128-byte swizzle.  Fields (16-byte units):
// [0,14) start address, [16,30) leading-dimension byte offset, [32,46) stride
// byte offset, [46,48) version = 1, [61,64) layout type (2 = SWIZZLE_128B).
//   K-major operand (rows of 64 16-bit elements = one 128-byte swizzle row):
//     LBO = 1 (unused), SBO = 1024 bytes between groups of 8 rows.
//   MN-major operand (64 MN elements contiguous, one 128-byte row per K index):
//     LBO = bytes between 64-element MN blocks, SBO = 1024 bytes between groups
//     of 8 K rows.
__device__ __forceinline__ uint64_t make_sdesc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3fffu);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3fffu) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}

// Makes shared-memory writes of this thread (generic proxy) visible to the async proxy, through
// which MMAs and bulk copies read shared memory.
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// The same descriptor `bytes` further into shared memory.  The start-address field is the
// low 14 bits in 16-byte units and shared memory ends below 2^18 bytes, so the sum never
// carries into the next field: one add instead of re-encoding the descriptor per MMA (the
// issuing thread's instruction count is what bounds the MMA rate of small tiles).
__device__ __forceinline__ uint64_t sdesc_advance(uint64_t desc, uint32_t bytes) {
    return desc + (uint64_t)(bytes >> 4);
}

// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; A holds 16-bit pairs packed in 32-bit columns.
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                        bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
// Make `bar` complete one arrival once every MMA issued so far by this thread
// has finished (implies tcgen05.fence::before_thread_sync).
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// ---------------------------------------------------------------------------
// Clusters: barrier and distributed shared memory
// ---------------------------------------------------------------------------
// shared::cluster address of the object at this shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(const void *p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}

// All threads of all CTAs of the cluster.
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// ---------------------------------------------------------------------------
// Host: tensor maps
// ---------------------------------------------------------------------------
// Encode a 4-D tiled tensor map over a (B, H, T, d) view of 16-bit elements
// with 128-byte swizzle: dimensions (innermost first) d, T, H, B; box
// [box_d, box_t, 1, 1].  Returns RGD_OK or a status code.
int encode_heads_map(CUtensorMap *out, const void *base, int64_t B, int64_t H, int64_t T, int64_t d,
                     int64_t stride_b, int64_t stride_h, int64_t stride_n, int box_d, int box_t, bool bf16);
// Whether encode_heads_map accepts this view: 16-byte aligned base, and for every dimension of
// extent > 1 a positive stride that is a multiple of 16 bytes and below the descriptor's limit.
bool heads_map_encodable(const void *base, int64_t B, int64_t H, int64_t T, int64_t stride_b, int64_t stride_h,
                         int64_t stride_n);
// The same through a launch-plan cache (rgd_cache, may be null): a descriptor already encoded
// for exactly these arguments is copied out of the cache instead of being re-encoded.
int encode_heads_map_cached(rgd_cache *cache, CUtensorMap *out, const void *base, int64_t B, int64_t H, int64_t T,
                            int64_t d, int64_t stride_b, int64_t stride_h, int64_t stride_n, int box_d, int box_t,
                            bool bf16);

}  // namespace sm100
}  // namespace rgd
