// cluster_trunk.cu -- the 128-wide tensor-core trunk for small batches: a
// cluster of four CTAs keeps one board's activations in shared memory.
//
// The persistent trunk (tc_conv.cu) hands every layer over through global
// memory: stores, flags, polls and window loads are 6 to 7k of the ~15k cycles
// a layer takes when each SM has at most one item.  Here a CTA holds five of
// the board's 19 rows (the last four) for the whole net; a layer's output goes
// straight into the other of its two row buffers, and one board row to each
// neighbour by a shared-memory-to-shared-memory bulk copy that completes on the
// neighbour's barrier.
//
//   * rows: pitch 24 (19 points + 5 zero columns), so that a board row is
//     three 8-row swizzle groups: a halo copy keeps every byte's place in the
//     128-byte swizzle, and buffers start on group boundaries.  Own rows are
//     0..119, the neighbours' at -24..-1 and 120..143; zeros off the board.
//   * the MMA: M = 128 output channels (the weight stage), N = 128 rows, K
//     order as in the trunk (64-channel half, tap, 16 channels), so every
//     accumulator is the same sum: the results are bit for bit the trunk's.
//   * first layer: the expanded L5 rows (pitch 19) are loaded a board row at a
//     time into rows of pitch 24, two more on each side.
//   * weights: 16 KB stages (a tap x 64 channels) through a ring of 7; they do
//     not depend on the layers, so the next layer's first seven arrive while a
//     layer is handed over.
//
// What bounds it: shared memory in the MMAs (8 KB of operands for 64 cycles and
// a weight stage written every four: ~6.7k cycles a layer), then the hand-over
// (~2k).  24 positions, policy + value: 150 us against 223 on the trunk's
// 64-row items.
//
// Warps: 0 weights (and the first layer's rows), 1 MMA issuer and TMEM owner,
// 2..17 epilogue (a TMEM lane quarter x 32 rows each).
//
// A neighbour's copy into a row buffer follows, through the layer in between,
// this CTA's last MMA that read the buffer; a CTA leaves only when the whole
// cluster has finished.  Every wait is bounded (the limit is a launch
// parameter), whole warps decide together; after one that ran out the CTA stops
// issuing, waits (bounded) for copies in flight, and leaves through the same
// cluster barrier.
#include "lg_kernels.h"

#include <cstring>

namespace lg {

using namespace ptx;

namespace {

constexpr int kClSize = 4;
constexpr int kClPitch = 24;
constexpr int kClRows = 5;                         // board rows of a CTA
constexpr int kClOwn = kClRows * kClPitch;         // 120
constexpr int kClN = 128;                          // rows of an MMA
constexpr int kClPre = 32, kClPre5 = 48;           // buffer rows before the own ones
constexpr int kClBufRows = kClPre + kClN + 32;     // 192
constexpr int kClBuf5Rows = kClPre5 + kClN + 48;   // 224
constexpr int kClHalf = kClBufRows * 128, kClHalf5 = kClBuf5Rows * 128;
constexpr int kClStage = 128 * 128;
constexpr int kClStages = 7;
constexpr int kClHalo = kClPitch * 128;            // bytes of a board row, one half
constexpr int kClEpiWarps = 16;
constexpr int kClThreads = 64 + kClEpiWarps * 32;
constexpr uint32_t kClWait = 1u << 21;             // default limit of a wait, in polls
// buffer 0: layer inputs of odd index (layer 0's output); buffer 1: the first
// layer's rows, then layer inputs of even index
constexpr int kClOff1 = 2 * kClHalf, kClOffW = kClOff1 + 2 * kClHalf5;
constexpr int kClOffCtl = kClOffW + kClStages * kClStage;

struct ClCtl {
    uint64_t w_full[kClStages], w_empty[kClStages];
    uint64_t in_full, acc_full, act_ready, halo_full[2], row_done[2], mma_done;
    uint32_t tmem_base;
    int abort_flag;
};
constexpr int kClSmem = kClOffCtl + (int)sizeof(ClCtl) + 1024;
static_assert(kClHalf % 1024 == 0 && kClHalf5 % 1024 == 0 && kClSmem <= 227 * 1024, "shared memory");

struct ClParams {
    const float *bias, *scale;    // [nl][128], the 3x3 layers (scale may be null)
    const float *bias0, *scale0;  // [128], the first layer
    const float *head_w;          // [128]
    float *parts;                 // [4][part_stride]
    size_t part_stride;
    int nl;
    int *err;
    uint32_t wait_limit;
    int stall;                    // test hook: the first CTA's second layer waits for what comes only later
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared memory of this CTA -> shared memory of a CTA of the cluster,
// completing `bytes` on that CTA's barrier
__device__ __forceinline__ void copy_to_cta(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void cl_ffma2(float &d0, float &d1, float a0, float a1, float b, float c) {
    asm("{\n.reg .b64 ra, rb, rc, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %4};\n"
        "mov.b64 rc, {%5, %5};\nfma.rn.f32x2 rd, ra, rb, rc;\nmov.b64 {%0, %1}, rd;\n}"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
template <bool F16>
__device__ __forceinline__ uint32_t cl_pack_relu(float lo, float hi) {
    uint32_t d;
    if (F16)
        asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    else
        asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// 32 values per lane -> lane L holds the sum over the warp of value L, in the
// trunk's order.
__device__ __forceinline__ float cl_transpose_sum(float (&a)[32], int lane) {
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
        const bool upper = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const float keep = upper ? a[i + w] : a[i], send = upper ? a[i] : a[i + w];
            a[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
    }
    return a[0];
}

// The MMAs of a layer: per 64-channel half and tap one weight stage against
// the buffer's rows at the tap's offset.  Called by a converged warp; false if
// a stage did not arrive.
template <bool FIRST, bool F16>
__device__ __forceinline__ bool cl_layer(ClCtl &ctl, uint32_t tmem, uint64_t w_desc, uint64_t x_desc, uint32_t &g,
                                         uint32_t limit) {
    constexpr int NT = FIRST ? 5 : 9, HALF = FIRST ? kClHalf5 : kClHalf, PRE = FIRST ? kClPre5 : kClPre;
    constexpr uint32_t idesc = idesc_16(128, kClN, F16);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int t = 0; t < NT; ++t, ++g) {
            const uint32_t s = g % kClStages;
            if (!mbar_wait_warp(&ctl.w_full[s], (g / kClStages) & 1, limit)) return false;
            tc_fence_after();
            const int shift = FIRST ? (t - 2) * kClPitch : (t / 3 - 1) * kClPitch + t % 3 - 1;
            const uint64_t a = w_desc + (uint64_t)(s * (uint32_t)(kClStage >> 4));
            const uint64_t b = x_desc + (uint64_t)(h * (HALF >> 4) + (PRE + shift) * 8);
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    mma_bf16(tmem, a + 2 * kk, b + 2 * kk, idesc, (h == 0 && t == 0 && kk == 0) ? 0u : 1u);
                mma_commit(&ctl.w_empty[s]);
                if (h == 1 && t == NT - 1) mma_commit(&ctl.acc_full);
            }
            __syncwarp();
        }
    return true;
}

}  // namespace

template <bool F16>
__global__ void __launch_bounds__(kClThreads, 1) __cluster_dims__(kClSize, 1, 1)
    cluster_trunk_kernel(const __grid_constant__ CUtensorMap in5, const __grid_constant__ CUtensorMap w0_map,
                         const __grid_constant__ CUtensorMap w_map, const ClParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *const buf0 = smem, *const buf1 = smem + kClOff1, *const wst = smem + kClOffW;
    ClCtl &ctl = *reinterpret_cast<ClCtl *>(smem + kClOffCtl);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid / 32, 0), lane = tid % 32;
    const int rank = (int)cluster_rank(), board = blockIdx.x / kClSize;
    const int y0 = rank * kClRows, ny = min(kClRows, kBoard - y0);
    const bool up = rank > 0, down = rank < kClSize - 1;  // neighbours
    if (tid == 0) {
        for (int i = 0; i < kClStages; ++i) {
            mbar_init(&ctl.w_full[i], 1);
            mbar_init(&ctl.w_empty[i], 1);
        }
        mbar_init(&ctl.in_full, 1);
        mbar_init(&ctl.acc_full, 1);
        mbar_init(&ctl.act_ready, kClEpiWarps);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ctl.halo_full[i], 1);
            mbar_init(&ctl.row_done[i], 4);
        }
        mbar_init(&ctl.mma_done, 1);
        ctl.abort_flag = 0;
        fence_mbar_init();
        prefetch_tensormap(&in5);
        prefetch_tensormap(&w0_map);
        prefetch_tensormap(&w_map);
    }
    if (warp == 1) tmem_alloc(&ctl.tmem_base, kClN);
    for (int i = tid; i < kClOffW / 16; i += kClThreads) reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async();
    __syncthreads();
    cluster_sync();  // every CTA's barriers are there before a neighbour completes bytes on them
    tc_fence_after();
    const uint32_t tmem = ctl.tmem_base;
    grid_dep_wait();
    grid_dep_launch();

    auto fail = [&](int code) {
        atomicCAS(p.err, 0, code);
        atomicExch(&ctl.abort_flag, 1);
    };
    auto aborted = [&]() { return *(volatile int *)&ctl.abort_flag != 0; };

    if (warp == 0) {
        if (lane == 0) {
            // the first layer's rows: board rows y0 - 2 .. y0 + ny + 1
            int rows = 0;
            for (int y = max(0, y0 - 2); y < min(kBoard, y0 + ny + 2); ++y) ++rows;
            mbar_arrive_expect_tx(&ctl.in_full, (uint32_t)(rows * 2 * kBoard * 128));
            for (int y = max(0, y0 - 2); y < min(kBoard, y0 + ny + 2); ++y)
                for (int h = 0; h < 2; ++h)
                    tma_load_2d(buf1 + h * kClHalf5 + (kClPre5 + (y - y0) * kClPitch) * 128, &in5, &ctl.in_full, h * 64,
                                board * kL5Board + y * kL5Pitch);
            uint32_t g = 0;
            for (int l = 0; l <= p.nl; ++l) {
                const int nt = l == 0 ? 5 : 9;
                for (int j = 0; j < 2 * nt; ++j, ++g) {
                    const int h = j / nt, t = j - h * nt;
                    const uint32_t s = g % kClStages;
                    // (a constant limit: with the parameter in this loop 24
                    // positions take 156 us, not 150)
                    if (aborted() || !mbar_wait(&ctl.w_empty[s], ((g / kClStages) & 1) ^ 1, kClWait)) {
                        fail(141);
                        l = p.nl;
                        break;
                    }
                    mbar_arrive_expect_tx(&ctl.w_full[s], kClStage);
                    tma_load_2d(wst + s * kClStage, l == 0 ? &w0_map : &w_map, &ctl.w_full[s], 0,
                                ((l == 0 ? t : (l - 1) * 9 + t) * 2 + h) * 128);
                }
            }
        }
    } else if (warp == 1) {
        const uint64_t w_desc = sdesc_sw128(smem_u32(wst));
        const uint64_t x0 = sdesc_sw128(smem_u32(buf0)), x1 = sdesc_sw128(smem_u32(buf1));
        uint32_t g = 0;
        bool ok = mbar_wait_warp(&ctl.in_full, 0, p.wait_limit) &&
                  cl_layer<true, F16>(ctl, tmem, w_desc, x1, g, p.wait_limit);
        if (!ok) fail(142);
        for (int l = 1; l <= p.nl && ok; ++l) {
            // this CTA's rows and both neighbours' (a barrier each: a fast
            // neighbour's next row must not stand in for the other's)
            if (elect_one()) {
                if (up) mbar_arrive_expect_tx(&ctl.halo_full[0], 2 * kClHalo);
                if (down) mbar_arrive_expect_tx(&ctl.halo_full[1], 2 * kClHalo);
            }
            __syncwarp();
            const uint32_t ph = (uint32_t)(l - 1) & 1;
            ok = mbar_wait_warp(&ctl.act_ready, ph, p.wait_limit) &&
                 (!up || mbar_wait_warp(&ctl.halo_full[0], ph, p.wait_limit)) &&
                 (!down || mbar_wait_warp(&ctl.halo_full[1], ph, p.wait_limit));
            if (p.stall && l == 1 && blockIdx.x == 0) ok = ok && mbar_wait_warp(&ctl.mma_done, 0, p.wait_limit);
            ok = ok && cl_layer<false, F16>(ctl, tmem, w_desc, (l & 1) ? x0 : x1, g, p.wait_limit);
            if (!ok) fail(143);
        }
        __syncwarp();
        if (elect_one()) {
            mma_commit(&ctl.mma_done);
            mbar_wait(&ctl.mma_done, 0, 1u << 20);
        }
    } else {
        const int quarter = warp & 3, rq = (warp - 2) >> 2;
        const int o = quarter * 32 + lane, cq = quarter * 32 + (lane >> 2);
        const float hw = __ldg(p.head_w + o);
        const uint32_t t_base = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(rq * 32);
        // this lane's row of the group's 32: point of the board?
        const int q = rq * 32 + lane, yl = q / kClPitch, x = q - yl * kClPitch;
        const bool valid = yl < ny && x < kBoard;
        const unsigned vmask = __ballot_sync(0xffffffffu, valid);
        const int hh = quarter >> 1;
        // rows 96..119 of the last group are its own; 120..127 are the
        // neighbour's place
        const int blocks = rq == 3 ? 3 : 4;
        // the group that holds a board row for a neighbour: rows 0..23 (group
        // 0) up, rows 96..119 (group 3) down
        const bool gives = (rq == 0 && up) || (rq == 3 && down);
        for (int l = 0; l <= p.nl; ++l) {
            const float *bl = l == 0 ? p.bias0 : p.bias + (l - 1) * 128;
            const float *sl = l == 0 ? p.scale0 : (p.scale ? p.scale + (l - 1) * 128 : nullptr);
            if (l == p.nl) {
                // last layer: the 1x1 head's sums, a part per channel quarter
                const float bias = __ldg(bl + o), scale = sl ? __ldg(sl + o) : 1.0f;
                if (!mbar_wait_warp(&ctl.acc_full, (uint32_t)l & 1, p.wait_limit)) { fail(144); break; }
                tc_fence_after();
                uint32_t v[32];
                tmem_ld32(t_base, v);
                tmem_ld_wait();
                float f[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) f[j] = fmaxf(fmaf(__uint_as_float(v[j]), scale, bias), 0.0f) * hw;
                const float sum = cl_transpose_sum(f, lane);
                if (valid)
                    p.parts[(size_t)quarter * p.part_stride + (size_t)board * kPoints + (y0 + yl) * kBoard + x] = sum;
                tc_fence_before();
                break;
            }
            float fb[4], fs[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                fb[m] = __ldg(bl + cq + 8 * m);
                fs[m] = sl ? __ldg(sl + cq + 8 * m) : 1.0f;
            }
            if (!mbar_wait_warp(&ctl.acc_full, (uint32_t)l & 1, p.wait_limit)) { fail(145); break; }
            tc_fence_after();
            uint8_t *const out = (l & 1) ? buf1 : buf0;
            if (l == 0) {
                // buffer 1 held the first layer's rows: zeros again before a
                // neighbour may write its row there (which follows this layer)
                uint4 *z = reinterpret_cast<uint4 *>(buf1);
                for (int i = tid - 64; i < 2 * kClHalf5 / 16; i += kClEpiWarps * 32) z[i] = make_uint4(0, 0, 0, 0);
            }
            uint32_t r0[16], r1[16];
            tmem_ld16x256_x4(t_base, r0);
            tmem_ld16x256_x4(t_base + (16u << 16), r1);
            tmem_ld_wait();
            tc_fence_before();
            const uint32_t tile = smem_u32(out) + (uint32_t)(hh * kClHalf + (kClPre + rq * 32) * 128);
            const uint32_t st = tile + (lane & 7) * 128 + (((((quarter & 1) * 4) + (lane >> 3)) ^ (lane & 7)) * 16);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t w[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint32_t *rr = (m < 2) ? r0 : r1;
                    float a0, a1;
                    cl_ffma2(a0, a1, __uint_as_float(rr[4 * i + 2 * (m & 1)]), __uint_as_float(rr[4 * i + 2 * (m & 1) + 1]),
                             fs[m], fb[m]);
                    w[m] = cl_pack_relu<F16>(a0, a1);
                }
                if (i < blocks) stmatrix_x4_trans(st + i * 1024, w[0], w[1], w[2], w[3]);
            }
            __syncwarp();
            // pad rows as zeros: lane L clears row 8 i + L / 4, chunk L % 4 of this quarter's 64 bytes
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = 8 * i + (lane >> 2);
                if (i < blocks && !((vmask >> row) & 1u)) {
                    const uint32_t za = tile + row * 128 + ((((quarter & 1) * 4 + (lane & 3)) ^ (row & 7)) * 16);
                    asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(za), "r"(0u) : "memory");
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                if (gives) mbar_arrive(&ctl.row_done[rq == 0 ? 0 : 1]);
                mbar_arrive(&ctl.act_ready);
                if (gives && quarter == 0) {
                    if (l == 0 && !mbar_wait(&ctl.act_ready, 0, p.wait_limit)) fail(146);  // buffer 1 is all zeros
                    if (!mbar_wait(&ctl.row_done[rq == 0 ? 0 : 1], (uint32_t)l & 1, p.wait_limit)) {
                        fail(147);
                    } else {
                        const uint32_t peer = (uint32_t)(rank + (rq == 0 ? -1 : 1));
                        const uint32_t own = smem_u32(out) + (uint32_t)((kClPre + (rq == 0 ? 0 : kClOwn - kClPitch)) * 128);
                        const uint32_t at = smem_u32(out) + (uint32_t)((kClPre + (rq == 0 ? kClOwn : -kClPitch)) * 128);
                        const uint32_t bar = map_rank(smem_u32(&ctl.halo_full[rq == 0 ? 1 : 0]), peer);
                        for (int h = 0; h < 2; ++h)
                            copy_to_cta(map_rank(at + h * kClHalf, peer), own + h * kClHalf, kClHalo, bar);
                    }
                }
            }
            __syncwarp();
        }
    }

    __syncthreads();
    if (aborted() && tid == 0) {
        // copies in flight into this CTA land, or their wait runs out: the
        // weights, the first layer's rows, the neighbours' rows (whoever sent
        // one has waited in vain for a row itself since)
        for (int i = 0; i < kClStages; ++i) {
            mbar_wait(&ctl.w_full[i], 0, 1u << 16);
            mbar_wait(&ctl.w_full[i], 1, 1u << 16);
        }
        mbar_wait(&ctl.in_full, 0, 1u << 16);
        for (int i = 0; i < 2; ++i)
            if (i == 0 ? up : down) {
                mbar_wait(&ctl.halo_full[i], 0, 1u << 16);
                mbar_wait(&ctl.halo_full[i], 1, 1u << 16);
            }
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, kClN);
    if (warp == 1) tmem_relinquish();
    cluster_sync();
}

// ------------------------------------------------------------------ host

int cluster_trunk_init_device(int *max_boards) {
    cudaError_t e = cudaFuncSetAttribute(cluster_trunk_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kClSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(cluster_trunk_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kClSmem);
    int n = 0;
    if (e == cudaSuccess) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kClSize);
        cfg.blockDim = dim3(kClThreads);
        cfg.dynamicSmemBytes = kClSmem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kClSize;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaOccupancyMaxActiveClusters(&n, cluster_trunk_kernel<false>, &cfg);
    }
    if (e != cudaSuccess) {
        lg_set_error("cluster trunk attributes: %s", cudaGetErrorString(e));
        return LG_ERR_CUDA;
    }
    *max_boards = n;
    return LG_OK;
}

int launch_cluster_trunk(const TcTrunk &T, int B, float *parts, size_t part_stride, int *err, cudaStream_t s) {
    if (T.nl < 1 || B < 1 || !T.buf5 || !T.w0 || !T.head_w || T.act != LG_ACT_RELU || T.count) {
        lg_set_error("launch_cluster_trunk: bad arguments");
        return LG_ERR_ARG;
    }
    CUtensorMap in5, w0_map, w_map;
    int rc = encode_map_2d_bf16(&in5, T.buf5, 128, (uint64_t)B * kL5Board, 64, kBoard);
    if (!rc) rc = encode_map_2d_bf16(&w0_map, T.w0, 64, (uint64_t)5 * 2 * 128, 64, 128);
    if (!rc) rc = encode_map_2d_bf16(&w_map, T.w, 64, (uint64_t)T.nl * 9 * 2 * 128, 64, 128);
    if (rc) return rc;
    ClParams p{};
    p.bias = T.bias;
    p.scale = T.scale;
    p.bias0 = T.bias0;
    p.scale0 = T.scale0;
    p.head_w = T.head_w;
    p.parts = parts;
    p.part_stride = part_stride;
    p.nl = T.nl;
    p.err = err;
    p.wait_limit = T.wait_limit ? T.wait_limit : kClWait;
    p.stall = T.stall_item >= 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(B * kClSize);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = kClSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = T.pdl ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, T.f16 ? cluster_trunk_kernel<true> : cluster_trunk_kernel<false>, in5, w0_map,
                                       w_map, p);
    if (e != cudaSuccess) {
        lg_set_error("cluster trunk launch: %s", cudaGetErrorString(e));
        return LG_ERR_CUDA;
    }
    return LG_OK;
}

}  // namespace lg
