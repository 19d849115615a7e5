// Attention forward for few queries (at most 16 per head): decoding steps, pooled or resampled
// cross-attention.  K and V are read once and dominate everything else, so the kernel is a stream over
// the keys: every warp walks its own 16-key tiles with a ring of cp.async stages that no other warp
// waits for, and the keys of one head are split over the warps of a CTA and the CTAs of a cluster, so
// that few heads still fill the chip.  The tensor-memory kernel gives a head one CTA whose single query
// tile runs scores -> softmax -> P V one after the other (1.8 us per 128 keys whatever the query count):
// [4, 1, 16, 128] against 4096 keys took 57.5 us there.
//
// One m16n8k16 MMA row tile holds all queries (rows past Tq are zeros).  The partial results of the
// warps (unnormalised O, row maximum, row sum) meet in shared memory and are combined through the
// cluster's distributed shared memory, each CTA taking a share of the output: no workspace, no second
// launch.
#include <math.h>

#include "attn_mma.cuh"
#include "sm100_prims.cuh"

namespace rgd {
namespace attn {

using namespace rgd::sm100;

constexpr int FEW_WARPS = 4;
constexpr int FEW_QUERIES = 16;
constexpr int FEW_KEYS = 16;                // keys per tile
constexpr int FEW_CLUSTER = 8;              // largest portable cluster

struct FewParams {
    AttnParams a;
    float scale_log2;
    int ntiles;
};

__device__ __forceinline__ void few_cp16(void *dst, const void *src, bool valid) {
    // not valid: nothing is read, 16 zero bytes are written
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ float few_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// STAGES of K and V tiles per warp, rows padded by 16 bytes (conflict-free ldmatrix).  Three stages of
// head_dim 128 let two CTAs share an SM.  The warp's partial O goes over its own ring afterwards.
template <typename T, int D>
struct FewSmem {
    static constexpr int STAGES = D == 128 ? 3 : 4;
    static constexpr int LD = D + PAD;
    struct alignas(16) Warp {
        union {
            T kv[STAGES][2][FEW_KEYS * LD];
            float o[FEW_QUERIES * D];
        };
    };
    Warp w[FEW_WARPS];
    float m[FEW_WARPS][FEW_QUERIES], l[FEW_WARPS][FEW_QUERIES];
};

template <typename T, int D, bool BIAS>
__global__ void __launch_bounds__(FEW_WARPS * 32) attn_few_kernel(const __grid_constant__ FewParams fp) {
    using Smem = FewSmem<T, D>;
    constexpr int STAGES = Smem::STAGES, LD = Smem::LD, CPR = D / 8;
    const AttnParams &p = fp.a;
    extern __shared__ __align__(16) unsigned char few_smem[];
    Smem &sm = *reinterpret_cast<Smem *>(few_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
    const int crank = blockIdx.x, csize = gridDim.x;        // the cluster spans the x dimension
    const int bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H;
    const T *kg = reinterpret_cast<const T *>(p.k) + (int64_t)b * p.k_sb + (int64_t)h * p.k_sh;
    const T *vg = reinterpret_cast<const T *>(p.v) + (int64_t)b * p.v_sb + (int64_t)h * p.v_sh;
    const T *qg = reinterpret_cast<const T *>(p.q) + (int64_t)b * p.q_sb + (int64_t)h * p.q_sh;
    const int first = crank * FEW_WARPS + warp, step = csize * FEW_WARPS;
    const int n = first < fp.ntiles ? (fp.ntiles - first + step - 1) / step : 0;
    typename Smem::Warp &ws = sm.w[warp];

    auto load_tile_async = [&](int i) {
        if (i < n) {
            const int key0 = (first + i * step) * FEW_KEYS;
            T *kd = ws.kv[i % STAGES][0], *vd = ws.kv[i % STAGES][1];
#pragma unroll
            for (int j = 0; j < FEW_KEYS * CPR / 32; ++j) {
                const int idx = j * 32 + lane, r = idx / CPR, c = (idx - r * CPR) * 8;
                const bool valid = key0 + r < p.Tk && c < p.d;
                const int64_t row = valid ? key0 + r : 0;
                const int ch = valid ? c : 0;
                few_cp16(kd + r * LD + c, kg + row * p.k_sn + ch, valid);
                few_cp16(vd + r * LD + c, vg + row * p.v_sn + ch, valid);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) load_tile_async(i);

    // Q as A fragments, rows past Tq and channels past d as zeros
    uint32_t aq[D / 16][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = gq + (e & 1) * 8, c = kk * 16 + (e >> 1) * 8 + tq * 2;
            aq[kk][e] = (r < p.Tq && c < p.d) ? *reinterpret_cast<const uint32_t *>(qg + (int64_t)r * p.q_sn + c) : 0u;
        }
    const char *bias_bh = nullptr;
    if constexpr (BIAS)
        bias_bh = reinterpret_cast<const char *>(p.bias) + ((int64_t)b * p.b_sb + (int64_t)h * p.b_sh) * (p.bias_f32 ? 4 : 2);

    float o[D / 8][4];
#pragma unroll
    for (int i = 0; i < D / 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
    float m_ref[2] = {-INFINITY, -INFINITY}, l_sum[2] = {0.f, 0.f};      // rows gq and gq + 8
    const int mi = lane >> 3, mr = lane & 7;

    for (int i = 0; i < n; ++i) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncwarp();
        load_tile_async(i + STAGES - 1);        // into the stage that was consumed one tile ago
        const T *ks = ws.kv[i % STAGES][0], *vs = ws.kv[i % STAGES][1];
        const int key0 = (first + i * step) * FEW_KEYS;
        float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            uint32_t bf[4];
            ldmatrix_x4(bf, ks + (mr + (mi >> 1) * 8) * LD + kk * 16 + (mi & 1) * 8);
            Mma<T>::mma(s[0], aq[kk], bf[0], bf[1]);
            Mma<T>::mma(s[1], aq[kk], bf[2], bf[3]);
        }
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = key0 + t * 8 + tq * 2 + (e & 1), r = gq + (e >> 1) * 8;
                float x = s[t][e] * fp.scale_log2;
                if constexpr (BIAS)
                    if (key < p.Tk && r < p.Tq) {
                        const float bv = bias_at_t<T>(p, bias_bh, r, key);
                        x += p.bias_f32 ? bias_log2<float>(bv) : bias_log2<T>(bv);
                    }
                if (key >= p.Tk) x = -INFINITY;
                s[t][e] = x;
                mx[e >> 1] = fmaxf(mx[e >> 1], x);
            }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
        }
        // The reference follows the maximum, so that the largest probability of a warp's keys is exactly 1 and
        // not rounded to 16 bits (a reference that lags by up to 2^8 put up to 10 % on the output's error against
        // 64 bits); a new maximum gets rare along the keys, and the loop is bound by its loads anyway.
        bool want[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) want[r] = mx[r] > m_ref[r];
        if (__any_sync(0xffffffffu, want[0] || want[1])) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float alpha = !want[r] ? 1.f : (m_ref[r] == -INFINITY ? 0.f : few_ex2(m_ref[r] - mx[r]));
                if (want[r]) m_ref[r] = mx[r];
                l_sum[r] *= alpha;
#pragma unroll
                for (int j = 0; j < D / 8; ++j) {
                    o[j][2 * r] *= alpha;
                    o[j][2 * r + 1] *= alpha;
                }
            }
        }
        uint32_t pk[4];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float mu = m_ref[r] == -INFINITY ? 0.f : m_ref[r];
                const float p0 = few_ex2(s[t][2 * r] - mu), p1 = few_ex2(s[t][2 * r + 1] - mu);
                l_sum[r] += p0 + p1;
                pk[t * 2 + r] = Mma<T>::pack(p0, p1);
            }
#pragma unroll
        for (int nn = 0; nn < D / 16; ++nn) {
            uint32_t bf[4];
            ldmatrix_x4_trans(bf, vs + (mr + (mi & 1) * 8) * LD + nn * 16 + (mi >> 1) * 8);
            Mma<T>::mma(o[2 * nn], pk, bf[0], bf[1]);
            Mma<T>::mma(o[2 * nn + 1], pk, bf[2], bf[3]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();

    // this warp's partial result over its own ring
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l_sum[r] += __shfl_xor_sync(0xffffffffu, l_sum[r], 1);
        l_sum[r] += __shfl_xor_sync(0xffffffffu, l_sum[r], 2);
        const int row = gq + r * 8;
        if (row < p.Tq) {
            if (tq == 0) {
                sm.m[warp][row] = m_ref[r];
                sm.l[warp][row] = l_sum[r];
            }
#pragma unroll
            for (int j = 0; j < D / 8; ++j)
                *reinterpret_cast<float2 *>(&ws.o[row * D + j * 8 + tq * 2]) = make_float2(o[j][2 * r], o[j][2 * r + 1]);
        }
    }
    cluster_sync_all();

    // combine: this CTA's share of the Tq x d / 4 output quads
    const int quads = p.d >> 2;
    T *og = reinterpret_cast<T *>(p.out_o) + (int64_t)b * p.o_sb + (int64_t)h * p.o_sh;
    for (int e = crank * FEW_WARPS * 32 + (int)threadIdx.x; e < p.Tq * quads; e += csize * FEW_WARPS * 32) {
        const int row = e / quads, c = (e - row * quads) * 4;
        float M = -INFINITY;
        for (int cr = 0; cr < csize; ++cr)
#pragma unroll
            for (int w = 0; w < FEW_WARPS; ++w) M = fmaxf(M, ld_cluster_f32(cluster_addr(&sm.m[w][row], cr)));
        const float mu = M == -INFINITY ? 0.f : M;
        float L = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int cr = 0; cr < csize; ++cr)
#pragma unroll
            for (int w = 0; w < FEW_WARPS; ++w) {
                const float f = few_ex2(ld_cluster_f32(cluster_addr(&sm.m[w][row], cr)) - mu);
                const float4 v = ld_cluster_f32x4(cluster_addr(&sm.w[w].o[row * D + c], cr));
                L = fmaf(ld_cluster_f32(cluster_addr(&sm.l[w][row], cr)), f, L);
                acc.x = fmaf(v.x, f, acc.x); acc.y = fmaf(v.y, f, acc.y);
                acc.z = fmaf(v.z, f, acc.z); acc.w = fmaf(v.w, f, acc.w);
            }
        const float inv = L > 0.f ? 1.f / L : 0.f;
        uint2 out;
        out.x = Mma<T>::pack(acc.x * inv, acc.y * inv);
        out.y = Mma<T>::pack(acc.z * inv, acc.w * inv);
        *reinterpret_cast<uint2 *>(og + (int64_t)row * p.o_sn + c) = out;
        if (c == 0) p.lse[(int64_t)bh * p.Tq_rounded + row] = L > 0.f ? (M + log2f(L)) * 0.6931471805599453f : -INFINITY;
    }
    // rows of the log-sum-exp past the queries
    if (crank == 0)
        for (int row = p.Tq + (int)threadIdx.x; row < p.Tq_rounded; row += FEW_WARPS * 32)
            p.lse[(int64_t)bh * p.Tq_rounded + row] = INFINITY;
    cluster_sync_all();                         // no CTA leaves while another still reads its shared memory
}

bool few_fwd_eligible(const AttnParams &p) {
    return p.Tq >= 1 && p.Tq <= FEW_QUERIES && p.Tk >= 1 && !p.causal && p.d >= 8 && p.d <= 128 && p.d % 8 == 0 && p.vec_q &&
           p.vec_k && p.vec_v && p.vec_o && (int64_t)p.B * p.H <= 65535;
}

template <typename T, int D>
static int launch_few(const FewParams &fp, cudaStream_t st) {
    const AttnParams &p = fp.a;
    const int BH = p.B * p.H;
    // Splits of a head's keys: as many CTAs as the chip holds at once (two per SM), at least one tile per warp.
    // More heads than half of that fill the chip unsplit at head dims above 64, and below in halves (three CTAs share
    // an SM there); quarters and eighths only add combining.  8 queries of 192 heads, us at 1 / 2 / 4 / 8 splits:
    //   head_dim 128: 512 keys 14.9 / 18.7 / 24.9 / 45.5, 4096 keys 75.2 / 82.3 / 74.9 / 94.5
    //   head_dim 64:  512 keys 12.6 / 10.9 / 16.8 / 32.8, 4096 keys 49.1 / 42.4 / 43.6 / 58.7
    // and of 96 heads, head_dim 128: 512 keys 12.7 / 11.4 / 16.9 / 25.0, 4096 keys 47.6 / 41.5 / 48.7 / 51.5.
    const int room = 2 * num_sms();
    const bool many = BH > room / 2;
    int split = 1;
    while (split < (many ? (D > 64 ? 1 : 2) : FEW_CLUSTER) && split * 2 * FEW_WARPS <= fp.ntiles && (many || split * 2 * BH <= room))
        split *= 2;
    const size_t smem = sizeof(FewSmem<T, D>);
    auto kernel = p.bias_kind == RGD_BIAS_NONE ? attn_few_kernel<T, D, false> : attn_few_kernel<T, D, true>;
    if (int e = ensure_dyn_smem(reinterpret_cast<const void *>(kernel), smem)) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(split, BH);
    cfg.blockDim = dim3(FEW_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = split;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, fp);
    count_launch();
    return cuda_status(e);
}

int few_fwd(const AttnParams &p, int dtype, cudaStream_t st) {
    FewParams fp{};
    fp.a = p;
    fp.scale_log2 = p.scale * LOG2E;
    fp.ntiles = (p.Tk + FEW_KEYS - 1) / FEW_KEYS;
    if (p.d > 64) return dtype == RGD_BF16 ? launch_few<__nv_bfloat16, 128>(fp, st) : launch_few<__half, 128>(fp, st);
    return dtype == RGD_BF16 ? launch_few<__nv_bfloat16, 64>(fp, st) : launch_few<__half, 64>(fp, st);
}

}  // namespace attn
}  // namespace rgd
