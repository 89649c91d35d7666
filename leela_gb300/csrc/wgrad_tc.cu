// wgrad_tc.cu -- weight gradients of the student's conv layers (64 wide) on
// the tensor cores, FP32 values as sums of three BF16 parts (split_conv.cu).
//
//   dW[tap][c][o] = sum over rows q of X[q + shift(tap)][c] * dY[q][o]
// over flat rows (L3 rows for the 3x3 layers, L5 rows with the planes
// expanded along x for the 5x5 first layer; pad rows of dY are zero).  The
// contraction runs over rows, so both operands are MN-major: the row windows
// as TMA brings them, channels contiguous, a tap a row offset of the
// descriptor.
//
// 3x3 layers: M = 128 = the h and m parts of X's 64 channels (two blocks of
// the window), N = parts of dY's 64 channels side by side:
//   [xh xm] x [dh dm] -> columns 0..127, [xh xm] x [dl] and [xl 0] x [dh] ->
//   columns 64..127
// -- the products of order 1 and 2^-8 in lanes 0..63 / 64..127 of columns
// 0..63, the smaller ones in columns 64..127.  A CTA takes three of the nine
// taps (384 accumulator columns) over a range of rows, 64 rows a stage.
// First layer: planes are exact in one part, M = 128 = the 5 x c_in expanded
// channels, N = 192 = dY's three parts, two of the five taps a CTA.
//
// The tensor core truncates its accumulators (split_conv.cu): every 256 rows
// the epilogue warps add them to FP32 registers, rounding to nearest; at the
// end of its rows the CTA adds its sums to dW with vector reductions (about 50
// per weight, in no fixed order, as the FFMA kernel's).
//
// What bounds it: shared memory -- 20 KB of operands and a twelfth of a 66 KB
// stage for each 160 cycles of MMAs.  512 boards, a 3x3 layer: 91 us (150
// TFLOP/s) against 749 with FFMA tiles, the first layer 43 against 1,600.
#include "lg_kernels.h"

#include <algorithm>

namespace lg {

using namespace ptx;

namespace {

constexpr int kWgRows = 64;                          // rows per stage
constexpr int kWgStages = 3;
constexpr int kWgFlush = 4;                          // stages per accumulator chain
constexpr int kWgEpiWarps = 16;
constexpr int kWgThreads = 128 + kWgEpiWarps * 32;
constexpr uint32_t kWgWait = 1u << 21;              // default limit of a wait, in polls

template <bool FIRST>
struct WgCfg {
    static constexpr int TAPS = FIRST ? 2 : 3;       // taps per CTA
    static constexpr int NT = FIRST ? 5 : 9;
    static constexpr int GROUPS = (NT + TAPS - 1) / TAPS;
    static constexpr int PRE = FIRST ? 40 : 24;
    static constexpr int XBLK = (kWgRows + 2 * PRE) * 128;  // one 64-channel block of X rows
    static constexpr int NX = FIRST ? 2 : 3;         // blocks: channel halves, or parts
    static constexpr int DBLK = kWgRows * 128;
    static constexpr int STAGE = NX * XBLK + 3 * DBLK;
    static constexpr int ZERO = FIRST ? 0 : XBLK;    // a block of zeros
    static constexpr int COLS = FIRST ? 192 : 128;   // accumulator columns per tap
    static constexpr int CTL = kWgStages * STAGE + ZERO;
    static constexpr int SMEM = CTL + 256 + 1024;
    static_assert(XBLK % 1024 == 0 && DBLK % 1024 == 0 && SMEM <= 227 * 1024 && TAPS * COLS <= 512, "budget");
};

struct WgCtl {
    uint64_t full[kWgStages], empty[kWgStages], acc_full, acc_empty, mma_done;
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(WgCtl) <= 256, "control block");

struct WgParams {
    CUtensorMap x, d;
    int stages, ranges;   // 64-row stages in all, row ranges
    int kchan;            // real channels of X (rows of dW per tap)
    float *dW;            // [taps][kchan][64]
    int *err;
    uint32_t wait_limit;
    int stall;            // test hook: the first CTA waits for what comes only at its end
};

// MN-major operand, 128-byte swizzle: 64 channels (128 bytes) a row, 8-row
// groups 1024 bytes apart along K, 64-channel blocks `block` bytes apart.
__device__ __forceinline__ uint64_t desc_mn(uint32_t saddr, uint32_t block) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)(block >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__host__ __device__ constexpr uint32_t idesc_mn(int n) { return idesc_bf16(128, n) | (1u << 15) | (1u << 16); }

__device__ __forceinline__ void red_add4(float *p, float a, float b, float c, float d) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

}  // namespace

template <bool FIRST>
__global__ void __launch_bounds__(kWgThreads, 1) wgrad_tc_kernel(const __grid_constant__ WgParams p) {
    using C = WgCfg<FIRST>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    WgCtl &ctl = *reinterpret_cast<WgCtl *>(smem + C::CTL);
    int &abort_flag = ctl.abort_flag;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid / 32, 0), lane = tid % 32;
    // CTA -> tap group, row range
    const int grp = blockIdx.x / p.ranges, rng = blockIdx.x % p.ranges;
    const int s0 = (int)((long long)p.stages * rng / p.ranges), s1 = (int)((long long)p.stages * (rng + 1) / p.ranges);
    const int tap0 = grp * C::TAPS, ntap = min(C::TAPS, C::NT - tap0);
    if (tid == 0) {
        for (int i = 0; i < kWgStages; ++i) {
            mbar_init(&ctl.full[i], 1);
            mbar_init(&ctl.empty[i], 1);
        }
        mbar_init(&ctl.acc_full, 1);
        mbar_init(&ctl.acc_empty, kWgEpiWarps);
        mbar_init(&ctl.mma_done, 1);
        abort_flag = 0;
        fence_mbar_init();
        prefetch_tensormap(&p.x);
        prefetch_tensormap(&p.d);
    }
    for (int i = tid; i < C::ZERO / 16; i += kWgThreads)
        reinterpret_cast<uint4 *>(smem + kWgStages * C::STAGE)[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async();
    if (warp == 1) tmem_alloc(&ctl.tmem_base, 512);
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl.tmem_base;
    grid_dep_wait();
    grid_dep_launch();

    auto fail = [&](int code) {
        atomicCAS(p.err, 0, code);
        atomicExch(&abort_flag, 1);
    };

    if (warp == 0) {
        if (lane == 0) {
            for (int s = s0; s < s1 && !abort_flag; ++s) {
                const uint32_t n = (uint32_t)(s - s0), st = n % kWgStages;
                if (!mbar_wait(&ctl.empty[st], ((n / kWgStages) & 1) ^ 1, p.wait_limit)) { fail(121); break; }
                uint8_t *dst = smem + st * C::STAGE;
                mbar_arrive_expect_tx(&ctl.full[st], C::STAGE);
                const int r0 = s * kWgRows;
                for (int b = 0; b < C::NX; ++b) {
                    if (FIRST)
                        tma_load_2d(dst + b * C::XBLK, &p.x, &ctl.full[st], b * 64, r0 - C::PRE);
                    else
                        tma_load_3d(dst + b * C::XBLK, &p.x, &ctl.full[st], 0, r0 - C::PRE, b);
                }
                for (int b = 0; b < 3; ++b)
                    tma_load_3d(dst + C::NX * C::XBLK + b * C::DBLK, &p.d, &ctl.full[st], 0, r0, b);
            }
        }
    } else if (warp == 1) {
        const uint32_t base = smem_u32(smem);
        for (int s = s0; s < s1; ++s) {
            const uint32_t n = (uint32_t)(s - s0), st = n % kWgStages;
            const bool head = n % kWgFlush == 0;
            if (head && !mbar_wait_warp(&ctl.acc_empty, ((n / kWgFlush) & 1) ^ 1, p.wait_limit)) { fail(122); break; }
            if (!mbar_wait_warp(&ctl.full[st], (n / kWgStages) & 1, p.wait_limit)) { fail(123); break; }
            if (p.stall && blockIdx.x == 0 && !mbar_wait_warp(&ctl.mma_done, 0, p.wait_limit)) { fail(125); break; }
            tc_fence_after();
            const uint32_t xs = base + st * C::STAGE, ds = xs + C::NX * C::XBLK;
            const uint64_t d0 = desc_mn(ds, C::DBLK);
            if (elect_one()) {
#pragma unroll
                for (int i = 0; i < C::TAPS; ++i) {
                    if (i >= ntap) break;
                    const int t = tap0 + i;
                    const int shift = FIRST ? (t - 2) * kL5Pitch : (t / 3 - 1) * kL3Pitch + t % 3 - 1;
                    const uint32_t xo = xs + (uint32_t)(C::PRE + shift) * 128u, dt = tmem + (uint32_t)(i * C::COLS);
                    const uint64_t x01 = desc_mn(xo, C::XBLK);
                    const uint64_t x2 = desc_mn(xo + 2 * C::XBLK,
                                                base + kWgStages * C::STAGE - (xs + 2 * C::XBLK));
#pragma unroll
                    for (int ks = 0; ks < kWgRows / 16; ++ks) {
                        const uint64_t k = (uint64_t)(ks * 128);  // 16 rows = 2048 bytes
                        const uint32_t on = (head && ks == 0) ? 0u : 1u;
                        if (FIRST) {
                            mma_bf16(dt, x01 + k, d0 + k, idesc_mn(192), on);
                        } else {
                            mma_bf16(dt, x01 + k, d0 + k, idesc_mn(128), on);
                            mma_bf16(dt + 64, x01 + k, d0 + 2 * (C::DBLK >> 4) + k, idesc_mn(64), 1u);
                            mma_bf16(dt + 64, x2 + k, d0 + k, idesc_mn(64), 1u);
                        }
                    }
                }
                mma_commit(&ctl.empty[st]);
                if (n % kWgFlush == kWgFlush - 1 || s + 1 == s1) mma_commit(&ctl.acc_full);
            }
        }
        __syncwarp();
        if (elect_one()) {
            mma_commit(&ctl.mma_done);
            mbar_wait(&ctl.mma_done, 0, 1u << 20);
        }
    } else if (warp >= 4) {
        const int quarter = warp & 3, cg = ((warp - 4) >> 2) * 16;
        const uint32_t t0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)cg;
        float v[C::TAPS][16];
#pragma unroll
        for (int i = 0; i < C::TAPS; ++i)
#pragma unroll
            for (int k = 0; k < 16; ++k) v[i][k] = 0.0f;
        const int nflush = (s1 - s0 + kWgFlush - 1) / kWgFlush;
        bool bad = false;
        for (int f = 0; f < nflush; ++f) {
            if (!mbar_wait_warp(&ctl.acc_full, (uint32_t)f & 1, p.wait_limit)) { fail(124); bad = true; break; }
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < C::TAPS; ++i) {
                uint32_t a[16], b[16];
                tmem_ld16(t0 + i * C::COLS, a);
                tmem_ld16(t0 + i * C::COLS + 64, b);
                tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    if (!FIRST) v[i][k] += __uint_as_float(a[k]) + __uint_as_float(b[k]);
                if (FIRST) {
                    uint32_t c[16];
                    tmem_ld16(t0 + i * C::COLS + 128, c);
                    tmem_ld_wait();
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        v[i][k] += __uint_as_float(a[k]) + (__uint_as_float(b[k]) + __uint_as_float(c[k]));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl.acc_empty);
        }
        const int row = quarter * 32 + lane, k = FIRST ? row : row % 64;
        if (!bad && k < p.kchan && nflush > 0) {
#pragma unroll
            for (int i = 0; i < C::TAPS; ++i) {
                if (i >= ntap) break;
                float *dst = p.dW + ((size_t)(tap0 + i) * p.kchan + k) * 64 + cg;
#pragma unroll
                for (int j = 0; j < 16; j += 4) red_add4(dst + j, v[i][j], v[i][j + 1], v[i][j + 2], v[i][j + 3]);
            }
        }
    }
    __syncthreads();
    if (abort_flag && tid == 0)
        for (int i = 0; i < kWgStages; ++i) {
            mbar_wait(&ctl.full[i], 0, 1u << 16);
            mbar_wait(&ctl.full[i], 1, 1u << 16);
        }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
    if (warp == 1) tmem_relinquish();
}

// ------------------------------------------------------------------ parts
//
// FP32 rows [B*361][64] -> parts [3][cap][64] in flat rows of `pitch` a board
// row, `board` a board (L3 or L5 layout), pads zero.  With Y, the value is
// g = dY where Y > 0, else 0 (the ReLU's gradient), and db[c] += sum of g.
// Eight threads a row, eight channels each; memory-bound (read 4 or 8 bytes,
// write 6 a value).
__global__ void __launch_bounds__(256) to_parts_kernel(const float *__restrict__ src, const float *__restrict__ Y,
                                                       int rows, int pitch, int board, size_t part_stride,
                                                       __nv_bfloat16 *__restrict__ parts, float *__restrict__ db) {
    __shared__ float sb[32][65];
    const int c8 = threadIdx.x % 8, r0 = threadIdx.x / 8;
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.0f;
    for (int q = blockIdx.x * 32 + r0; q < rows; q += gridDim.x * 32) {
        const int b = q / board, r = q - b * board, y = r / pitch, x = r - y * pitch;
        uint4 out[3] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
        if (y < kBoard && x < kBoard) {
            const size_t at = ((size_t)b * kPoints + y * kBoard + x) * 64 + c8 * 8;
            float v[8];
            *reinterpret_cast<float4 *>(v) = *reinterpret_cast<const float4 *>(src + at);
            *reinterpret_cast<float4 *>(v + 4) = *reinterpret_cast<const float4 *>(src + at + 4);
            if (Y) {
                float m[8];
                *reinterpret_cast<float4 *>(m) = *reinterpret_cast<const float4 *>(Y + at);
                *reinterpret_cast<float4 *>(m + 4) = *reinterpret_cast<const float4 *>(Y + at + 4);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    v[k] = m[k] > 0.0f ? v[k] : 0.0f;
                    acc[k] += v[k];
                }
            }
            uint32_t *w = reinterpret_cast<uint32_t *>(out);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float h0, m0, l0, h1, m1, l1;
                split3(v[2 * k], h0, m0, l0);
                split3(v[2 * k + 1], h1, m1, l1);
                w[k] = pack2_bf16(h0, h1);
                w[4 + k] = pack2_bf16(m0, m1);
                w[8 + k] = pack2_bf16(l0, l1);
            }
        }
#pragma unroll
        for (int p = 0; p < 3; ++p)
            reinterpret_cast<uint4 *>(parts + p * part_stride + (size_t)q * 64)[c8] = out[p];
    }
    if (!db) return;
#pragma unroll
    for (int k = 0; k < 8; ++k) sb[r0][c8 * 8 + k] = acc[k];
    __syncthreads();
    if (threadIdx.x < 64) {
        float s = 0.0f;
        for (int i = 0; i < 32; ++i) s += sb[i][threadIdx.x];
        atomicAdd(&db[threadIdx.x], s);
    }
}

// ------------------------------------------------------------------ host

int wgrad_init_device() {
    cudaError_t e = cudaFuncSetAttribute(wgrad_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         WgCfg<false>::SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(wgrad_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, WgCfg<true>::SMEM);
    if (e != cudaSuccess) {
        lg_set_error("cudaFuncSetAttribute(weight gradient): %s", cudaGetErrorString(e));
        return LG_ERR_CUDA;
    }
    return LG_OK;
}

void launch_to_parts(const float *src, const float *Y, int B, bool l5, size_t cap_rows, __nv_bfloat16 *parts, float *db,
                     cudaStream_t s) {
    const int rows = B * (l5 ? kL5Board : kL3Board);
    to_parts_kernel<<<std::min((rows + 31) / 32, 152 * 8), 256, 0, s>>>(
        src, Y, rows, l5 ? kL5Pitch : kL3Pitch, l5 ? kL5Board : kL3Board, cap_rows * 64, parts, db);
}

template <bool FIRST>
static int launch_wgrad(const CUtensorMap &x, const CUtensorMap &d, int rows, int kchan, float *dW, int *err,
                        cudaStream_t s, uint32_t stall_polls) {
    using C = WgCfg<FIRST>;
    WgParams p{};
    p.x = x;
    p.d = d;
    p.stages = (rows + kWgRows - 1) / kWgRows;
    // one CTA an SM; the groups share them out
    p.ranges = std::max(1, std::min(152 / C::GROUPS, p.stages / kWgFlush));
    p.kchan = kchan;
    p.dW = dW;
    p.err = err;
    p.wait_limit = stall_polls ? stall_polls : kWgWait;
    p.stall = stall_polls != 0;
    wgrad_tc_kernel<FIRST><<<C::GROUPS * p.ranges, kWgThreads, C::SMEM, s>>>(p);
    return LG_OK;
}

int launch_wgrad_3x3(const __nv_bfloat16 *x, const __nv_bfloat16 *d, int B, size_t cap_rows, float *dW, int *err,
                     cudaStream_t s, uint32_t stall_polls) {
    using C = WgCfg<false>;
    const int rows = B * kL3Board;
    CUtensorMap mx, md;
    int rc = encode_map_3d_bf16(&mx, x, 64, rows, 3, cap_rows, 64, C::XBLK / 128);
    if (!rc) rc = encode_map_3d_bf16(&md, d, 64, rows, 3, cap_rows, 64, kWgRows);
    return rc ? rc : launch_wgrad<false>(mx, md, rows, 64, dW, err, s, stall_polls);
}

int launch_wgrad_first(const __nv_bfloat16 *l5, const __nv_bfloat16 *d, int B, int c_in, size_t cap_rows, float *dW,
                       int *err, cudaStream_t s, uint32_t stall_polls) {
    using C = WgCfg<true>;
    const int rows = B * kL5Board;
    CUtensorMap mx, md;
    int rc = encode_map_2d_bf16(&mx, l5, 128, rows, 64, C::XBLK / 128);
    if (!rc) rc = encode_map_3d_bf16(&md, d, 64, rows, 3, cap_rows, 64, kWgRows);
    return rc ? rc : launch_wgrad<true>(mx, md, rows, 5 * c_in, dW, err, s, stall_polls);
}

}  // namespace lg
