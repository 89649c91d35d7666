// split_conv.cu -- FP32 conv layers on the tensor cores, each FP32 value as
// the sum of three BF16 parts.
//
// The FP32 path's arithmetic (Network.cpp:345-393: im2col + sgemm + bias +
// activation) is bound by the FFMA pipes (70 TFLOP/s measured with a cuBLAS
// FP32 GEMM).  A BF16 value has 8 significant bits and FP32's exponent range,
// so x = h + m + l holds all 24 bits of an FP32 value, and
//   x * w = xh wh + (xh wm + xm wh) + (xh wl + xm wm + xl wh) + (terms below 2^-24)
// is six BF16 products, each exact in FP32: a sixth of the tensor rate, 4.5
// times the FFMA rate.
//
// Accuracy.  The tensor core truncates its FP32 accumulator after each
// 16-deep step (measured: a K = 1152 chain is 1.1e-6 off, always towards
// zero; FFMA chains 2.7e-7, K = 144 chains 1.3e-7), so a chain here is at
// most 128 deep (two taps x 64 input channels); the three orders of magnitude of the
// products have their own accumulator columns; and the epilogue warps add
// each chain's sums to the output's in FP32 registers, rounding to nearest.
// Activations are split by rounding (the parts' signs vary, so what the six
// products leave out averages out), weights by truncation with no part zero
// (the parts have the weight's sign, so an infinite activation gives the
// same infinity as one product would).
//
// Against 64 bits the benchmark nets' logits are 7.8e-7 off at every batch
// (relative 2-norm, mean of 24 seeds; the small-batch FFMA kernel 8.9e-7, the
// FFMA kernels per layer 7.0e-7 at one position to 2.3e-6 at 256, growing as
// their K splits go; 64-deep chains gain nothing over a whole net and cost
// 10%).
//
// GEMM shape (NO = 64 output channels an item; 32 for small batches, with
// half the N): M = 128 flat rows (the L3 / L5 layouts of lg_common.cuh: a tap
// is a row shift, the window of rows is loaded once and read at 9 or 5
// offsets), N = the weight parts of 64 output channels side by side:
//   xh x [wh wm wl] -> columns 0..191, xm x [wh wm] -> columns 64..191,
//   xl x [wh] -> columns 128..191,
// so columns 0..63 / 64..127 / 128..191 hold the products of order 1 / 2^-8 /
// 2^-16.  N = 192, 128 and 64 take 96, 64 and 48 cycles a step against 32
// for each of the six products alone: 92% of the MMA rate.
//
// One persistent launch runs all layers of a net: items (layer, 128-row tile,
// NO-channel group) claimed in order from a counter; an item starts once the
// tiles that its window covers are complete in the layer before (counters,
// bounded polls).  A layer has at least two items a tile, so no SM waits at
// a layer's end for more than its own dependencies.  Per CTA (one per SM):
//   warp 0     weight stages (a tap x 64 channels x 3 parts: 24 KB, ring of 3, or 6 of 12 KB)
//   warp 1     MMA issuer, TMEM owner
//   warp 2     item claims, dependency polls, windows (2 slots: one 64-channel
//              half of 3 parts x 176 rows each)
//   warps 4..19  sums, bias, activation, split, stores (a thread = a row x 32
//              channels): two groups of 8 taking items in turn, so that one's
//              stores overlap the other's sums
//
// What bounds it: the tensor pipe (832 cycles a weight stage, of ~1,090
// spent; 72% active under ncu, shared memory 71%, L2 34%), then the issuer's
// commits and waits: a barrier for each part of a stage, so that a part is
// refilled as soon as its MMAs are done, took 13.1 ms where one a stage took
// 10.2 (two commits and two waits more a stage); polls that each lane decided
// on its own, in a divergent loop, 2 to 8%.  With one epilogue group
// the MMAs waited 4.8k of 26k cycles an item for the stores.  Policy + value
// nets of 1,024 positions: 9.8 to 10.3 ms = 250 TFLOP/s of FP32 multiply-adds
// against 53.2 ms on the FFMA kernels; 77 positions of the reference's shapes
// through the host call 0.80 against 3.62 ms.  Pairs of CTAs (M = 256 MMAs,
// half of B's rows read and, with shared units, 20 KB of weights a stage) were
// correct but slower (12.3 ms against 11.8, 14.2 against 10.4 with the waits
// moved).
//
// Every wait is bounded (the limits are launch parameters); on a timeout the
// CTA records an error code, stops issuing, drains what it issued and frees
// its TMEM.  Warps that wait as a whole decide as a whole.
#include "lg_kernels.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace lg {

using namespace ptx;

namespace {

constexpr int kSpEpiWarps = 8;                    // per epilogue group
constexpr int kSpGroups = 2;                      // epilogue groups, taking items in turn
constexpr int kSpThreads = 128 + kSpGroups * kSpEpiWarps * 32;
constexpr int kSpTile = 128;                      // rows per item
constexpr int kSpPre3 = 24, kSpPre5 = 40;         // window rows before the tile
constexpr int kSpWin3 = kSpTile + 2 * kSpPre3;    // 176
constexpr int kSpWin5 = kSpTile + 2 * kSpPre5;    // 208
constexpr int kSpPart = kSpWin3 * 128;            // bytes of one part's window
constexpr int kSpSlot = 3 * kSpPart;
constexpr int kSpSlots = 2;
constexpr int kSpChain = 2;                       // taps (of 64 channels) per accumulator chain
constexpr int kSpRing = 4;                        // item descriptors in flight
constexpr uint32_t kSpWait = 1u << 21;            // default limits: mbarrier polls, counter polls
constexpr uint32_t kSpPolls = 1u << 22;
static_assert(kSpWin5 * 128 <= kSpSlot, "a first-layer window fits a slot");
static_assert(kSpPart % 1024 == 0 && kSpSlot % 1024 == 0, "swizzle alignment");

// NO = output channels per item.  Weight stages: NO rows of each part.
constexpr int kSpMaxStages = 6;
struct SpCtl {
    uint64_t win_full[kSpSlots], win_empty[kSpSlots], w_full[kSpMaxStages], w_empty[kSpMaxStages];
    uint64_t acc_full[kSpGroups][2], acc_empty[2], item_full[kSpRing], item_empty[kSpRing], mma_done;
    int item_id[kSpRing];
    uint32_t tmem_base;
    int abort_flag, last_out;
};
constexpr int kSpTileBytes = 32 * 32;             // an epilogue warp's staging tile
template <int NO_>
struct SpCfg {
    static constexpr int NO = NO_;
    static constexpr int STAGE = 3 * NO * 128;
    static constexpr int STAGES = kSpMaxStages * 32 / NO;
    static constexpr int CH = NO / 2;             // channels of an epilogue warp
    static constexpr int ACC = NO == 64 ? 256 : 128;  // columns between accumulators
    static constexpr int STG_OFF = kSpSlots * kSpSlot + STAGES * STAGE;
    static constexpr int CTL_OFF = STG_OFF + kSpGroups * kSpEpiWarps * kSpTileBytes;
    static constexpr int SMEM = CTL_OFF + (int)sizeof(SpCtl) + 1024;
    static_assert(STAGE % 1024 == 0 && STAGES <= kSpMaxStages && SMEM <= 227 * 1024, "shared memory budget");
};

struct SpLayerDev {
    int first;        // 5x5 first layer (L5 rows, planes: one part), else 3x3 (L3 rows)
    int halves;       // 64-channel halves of the input
    int groups;       // NO-channel groups of the output
    int wgroups;      // 64-channel groups in the weight layout
    int wrow;         // first row of the layer's weights in the weight map
    int item0;        // first item
    int need;         // tile counter value at which the layer before is complete
    int act;
    int cout;         // FP32 output channels (out32)
    const float *bias;        // [groups * 64]
    __nv_bfloat16 *out;       // [3][part_stride] parts, or null
    float *out32;             // [points][cout] FP32, or null
};

struct SpParams {
    CUtensorMap in[2], in5, w;  // layer l reads in[l & 1] (in5 when first)
    SpLayerDev L[kSpMaxLayers];
    int nl, rows, rows5, nitems;
    int cap_rows;             // rows between the parts of an activation buffer
    int pitch;                // channels per activation row
    int *flags;               // [n3] tile counters, [n5] first-layer tile counters, item counter, exit counter
    int *err;
    uint32_t wait_limit, poll_limit;
    int stall_item;           // test hook: this item waits for a count no item reaches (-1: none)
};

// A converged warp waits until the n counters at f reach `want`, a lane each.
__device__ __forceinline__ bool sp_poll(const int *f, int n, int want, uint32_t limit) {
    bool ok = true;
    for (int i = threadIdx.x % 32; i < n; i += 32) {
        uint32_t k = 0;
        while (ld_acquire_gpu(f + i) < want && ++k < limit) __nanosleep(32);
        ok = ok && k < limit;
    }
    return __all_sync(0xffffffffu, ok);
}

// 16 channels of 32 rows (lane = row) as parts into L3 rows `tgt` (-1: not
// stored), through a 1 KB staging tile so that two lanes store the 32 bytes
// of a row (a 16-byte store per lane and row would write half sectors of 32
// lines an instruction).  Tile rows are 32 bytes, their two 16-byte chunks
// XORed with a bit of the row: no bank conflicts either way.
__device__ __forceinline__ void store_parts(const float *v, int tgt, bool point, uint4 *tile, int lane,
                                            __nv_bfloat16 *out, size_t part_stride, int pitch) {
    uint32_t w[3][8];
    bool odd = false;  // a value that would round to infinity, an infinity or a NaN
#pragma unroll
    for (int k = 0; k < 16; ++k) odd = odd || !(fabsf(v[k]) < 3.3895e38f);
    if (!__any_sync(0xffffffffu, odd && point)) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float x0 = point ? v[2 * k] : 0.0f, x1 = point ? v[2 * k + 1] : 0.0f;
            const uint32_t h = pack2_bf16(x0, x1);
            const float r0 = x0 - __uint_as_float(h << 16), r1 = x1 - __uint_as_float(h & 0xFFFF0000u);
            const uint32_t m = pack2_bf16(r0, r1);
            w[0][k] = h;
            w[1][k] = m;
            w[2][k] = pack2_bf16(r0 - __uint_as_float(m << 16), r1 - __uint_as_float(m & 0xFFFF0000u));
        }
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float h0, m0, l0, h1, m1, l1;
            split3(point ? v[2 * k] : 0.0f, h0, m0, l0);
            split3(point ? v[2 * k + 1] : 0.0f, h1, m1, l1);
            w[0][k] = pack2_bf16(h0, h1);
            w[1][k] = pack2_bf16(m0, m1);
            w[2][k] = pack2_bf16(l0, l1);
        }
    }
    const int sub = lane >> 1, c = lane & 1, sw = (lane >> 2) & 1;
    const int t0 = __shfl_sync(0xffffffffu, tgt, sub), t1 = __shfl_sync(0xffffffffu, tgt, 16 + sub);
    const int x0 = sub * 2 + (c ^ ((sub >> 2) & 1)), x1 = x0 + 32;
    uint4 *const d0 = reinterpret_cast<uint4 *>(out + (size_t)max(t0, 0) * pitch) + c;
    uint4 *const d1 = reinterpret_cast<uint4 *>(out + (size_t)max(t1, 0) * pitch) + c;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        tile[lane * 2 + sw] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
        tile[lane * 2 + (1 ^ sw)] = make_uint4(w[p][4], w[p][5], w[p][6], w[p][7]);
        __syncwarp();
        const uint4 a = tile[x0], b = tile[x1];
        if (t0 >= 0) d0[p * (part_stride / 8)] = a;
        if (t1 >= 0) d1[p * (part_stride / 8)] = b;
        __syncwarp();
    }
}

__device__ __forceinline__ void store_zero_parts(__nv_bfloat16 *dst, size_t part_stride) {
    const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int i = 0; i < 2; ++i) reinterpret_cast<uint4 *>(dst + p * part_stride)[i] = z;
}

// The MMAs of one 64-channel half of an item, chains of kSpChain taps: the
// window in the slot of descriptor x, weight stages g, g + 1, ... of the
// ring.  Called by a converged warp.  A stage's waits come between the MMAs of
// the stage ahead of it: the tensor pipe has few MMAs queued, and ran dry while
// the issuer polled between two stages.  Policy + value nets of 1,024
// positions (polls without a vote): waits between the stages 11.8 ms, before the last four of the 12
// MMAs 10.3, before the last eight 10.2, before the last ten 11.1 (stages that
// arrive late then hold up more); the next half's first stage and window
// waited for as well: no gain.  False if a wait ran out.
template <int NO, bool FIRST>
__device__ __forceinline__ bool issue_half(SpCtl &ctl, uint32_t tmem, uint64_t x, uint64_t w_desc, int group,
                                           uint32_t &g, uint32_t &chain, uint32_t limit) {
    constexpr int NT = FIRST ? 5 : 9;
    using C = SpCfg<NO>;
    constexpr uint32_t id3 = idesc_bf16(128, 3 * NO), id2 = idesc_bf16(128, 2 * NO), id1 = idesc_bf16(128, NO);
    constexpr uint64_t kPart16 = kSpPart >> 4;
    auto ready = [&](uint32_t stage, bool head, uint32_t ch) {
        if (head && !mbar_wait_warp(&ctl.acc_empty[ch & 1], ((ch >> 1) & 1) ^ 1, limit)) return false;
        if (!mbar_wait_warp(&ctl.w_full[stage % C::STAGES], (stage / C::STAGES) & 1, limit)) return false;
        tc_fence_after();
        return true;
    };
    if (!ready(g, true, chain)) return false;
#pragma unroll
    for (int t = 0; t < NT; ++t, ++g) {
        const uint32_t s = g % C::STAGES, acc = chain & 1;
        const bool head = t % kSpChain == 0, tail = t % kSpChain == kSpChain - 1 || t == NT - 1;
        const uint32_t d = tmem + acc * C::ACC;
        const uint64_t w = w_desc + (uint64_t)(s * (uint32_t)(C::STAGE >> 4));
        const uint64_t xt = x + (uint64_t)((FIRST ? kSpPre5 + (t - 2) * kL5Pitch
                                                  : kSpPre3 + (t / 3 - 1) * kL3Pitch + (t % 3 - 1)) * 8);
        if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < (FIRST ? 2 : 4); ++kk)
                mma_bf16(d, xt + 2 * kk, w + 2 * kk, id3, head && kk == 0 ? 0u : 1u);
        }
        if (t + 1 < NT && !ready(g + 1, tail, chain + 1)) return false;
        if (elect_one()) {
            if (FIRST) {
#pragma unroll
                for (int kk = 2; kk < 4; ++kk) mma_bf16(d, xt + 2 * kk, w + 2 * kk, id3, 1u);
            } else {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) mma_bf16(d + NO, xt + kPart16 + 2 * kk, w + 2 * kk, id2, 1u);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) mma_bf16(d + 2 * NO, xt + 2 * kPart16 + 2 * kk, w + 2 * kk, id1, 1u);
            }
            mma_commit(&ctl.w_empty[s]);
            if (tail) mma_commit(&ctl.acc_full[group][acc]);
        }
        if (tail) ++chain;
    }
    return true;
}

}  // namespace

template <int NO>
__global__ void __launch_bounds__(kSpThreads, 1) split_trunk_kernel(const __grid_constant__ SpParams p) {
    using C = SpCfg<NO>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *win = smem;
    uint8_t *wst = smem + kSpSlots * kSpSlot;
    uint8_t *stg = smem + C::STG_OFF;
    SpCtl &ctl = *reinterpret_cast<SpCtl *>(smem + C::CTL_OFF);
    int &abort_flag = ctl.abort_flag;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid / 32, 0), lane = tid % 32;
    const int n3 = (p.rows + kSpTile - 1) / kSpTile, n5 = (p.rows5 + kSpTile - 1) / kSpTile;
    int *const flags3 = p.flags, *const flags5 = p.flags + n3, *const item_ctr = flags5 + n5;

    if (tid == 0) {
        for (int i = 0; i < kSpSlots; ++i) {
            mbar_init(&ctl.win_full[i], 1);
            mbar_init(&ctl.win_empty[i], 1);
        }
        for (int i = 0; i < C::STAGES; ++i) {
            mbar_init(&ctl.w_full[i], 1);
            mbar_init(&ctl.w_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            for (int k = 0; k < kSpGroups; ++k) mbar_init(&ctl.acc_full[k][i], 1);
            mbar_init(&ctl.acc_empty[i], kSpEpiWarps);
        }
        for (int i = 0; i < kSpRing; ++i) {
            mbar_init(&ctl.item_full[i], 1);
            mbar_init(&ctl.item_empty[i], 2 + kSpGroups * kSpEpiWarps);  // weights, MMA issuer, epilogue warps
        }
        mbar_init(&ctl.mma_done, 1);
        abort_flag = 0;
        fence_mbar_init();
        prefetch_tensormap(&p.in[0]);
        prefetch_tensormap(&p.in[1]);
        prefetch_tensormap(&p.in5);
        prefetch_tensormap(&p.w);
    }
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
    // item -> (layer, tile, group)
    auto decode = [&](int it, int &l, int &j, int &g) {
        l = 0;
        while (l + 1 < p.nl && it >= p.L[l + 1].item0) ++l;
        const int r = it - p.L[l].item0;
        j = r / p.L[l].groups;
        g = r - j * p.L[l].groups;
    };
    // the next item of this (converged) warp's walk over the ring; -1 at the end
    auto next_item = [&](int q, int code) -> int {
        const int slot = q % kSpRing;
        if (!mbar_wait_warp(&ctl.item_full[slot], (uint32_t)(q / kSpRing) & 1, p.wait_limit)) {
            fail(code);
            return -1;
        }
        return ctl.item_id[slot];
    };

    if (warp == 2) {
        // ------------------------------------------------ item claims + windows
        // lane 0 claims and loads, the whole warp polls the dependencies
        uint32_t wn = 0;
        for (int q = 0;; ++q) {
            int it = -1;
            if (lane == 0) {
                const int slot = q % kSpRing;
                bool ok = mbar_wait(&ctl.item_empty[slot], ((uint32_t)(q / kSpRing) & 1) ^ 1, p.wait_limit);
                // claimed once its first window slot is free, so that it is worked on at once
                ok = ok && mbar_wait(&ctl.win_empty[wn % kSpSlots], ((wn / kSpSlots) & 1) ^ 1, p.wait_limit);
                if (ok && !abort_flag) {
                    it = atomicAdd(item_ctr, 1);
                    if (it >= p.nitems) it = -1;
                } else if (!ok) {
                    fail(101);
                }
                ctl.item_id[slot] = it;
                mbar_arrive(&ctl.item_full[slot]);
            }
            it = __shfl_sync(0xffffffffu, it, 0);
            if (it < 0) break;
            int l, j, g;
            decode(it, l, j, g);
            const SpLayerDev &L = p.L[l];
            if (l > 0) {
                const int *f;
                int n;
                if (p.L[l - 1].first) {
                    // L5 tiles whose rows land on L3 rows [lo3, hi3): an L5 row is
                    // the L3 row minus (board + y), board + y <= rows / 400 + 19
                    const int lo3 = max(0, j * kSpTile - kSpPre3);
                    const int hi3 = min(p.rows, j * kSpTile + kSpTile + kSpPre3);
                    const int lo5 = max(0, lo3 - (hi3 - 1) / kL3Board - kBoard) / kSpTile;
                    f = flags5 + lo5;
                    n = min(p.rows5 - 1, hi3 - 1) / kSpTile - lo5 + 1;
                } else {
                    const int lo = max(0, j - 1);
                    f = flags3 + lo;
                    n = min(n3 - 1, j + 1) - lo + 1;
                }
                if (!sp_poll(f, n, it == p.stall_item ? 1 << 30 : L.need, p.poll_limit)) {
                    if (lane == 0) fail(102);
                    break;
                }
                fence_proxy_async_global();
                __syncwarp();
            }
            if (lane == 0) {
                for (int h = 0; h < L.halves; ++h) {
                    const uint32_t w = wn + h;
                    const int ws = w % kSpSlots;
                    if (h > 0 && !mbar_wait(&ctl.win_empty[ws], ((w / kSpSlots) & 1) ^ 1, p.wait_limit)) {
                        fail(103);
                        break;
                    }
                    uint8_t *dst = win + ws * kSpSlot;
                    if (L.first) {
                        mbar_arrive_expect_tx(&ctl.win_full[ws], kSpWin5 * 128);
                        tma_load_2d(dst, &p.in5, &ctl.win_full[ws], h * 64, j * kSpTile - kSpPre5);
                    } else {
                        mbar_arrive_expect_tx(&ctl.win_full[ws], kSpSlot);
                        for (int pt = 0; pt < 3; ++pt)
                            tma_load_3d(dst + pt * kSpPart, &p.in[l & 1], &ctl.win_full[ws], h * 64,
                                        j * kSpTile - kSpPre3, pt);
                    }
                }
            }
            wn += L.halves;
        }
    } else if (warp == 0) {
        // ------------------------------------------------ weight stages
        if (lane == 0) {
            uint32_t g = 0;
            for (int q = 0;; ++q) {
                int it = -1;
                if (mbar_wait(&ctl.item_full[q % kSpRing], (uint32_t)(q / kSpRing) & 1, p.wait_limit))
                    it = ctl.item_id[q % kSpRing];
                else
                    fail(104);
                mbar_arrive(&ctl.item_empty[q % kSpRing]);
                if (it < 0) break;
                int l, j, og;
                decode(it, l, j, og);
                const SpLayerDev &L = p.L[l];
                const int ntaps = L.first ? 5 : 9;
                bool bad = false;
                for (int h = 0; h < L.halves && !bad; ++h)
                    for (int t = 0; t < ntaps; ++t, ++g) {
                        const int s = g % C::STAGES;
                        if (!mbar_wait(&ctl.w_empty[s], ((g / C::STAGES) & 1) ^ 1, p.wait_limit)) {
                            fail(105);
                            bad = true;
                            break;
                        }
                        mbar_arrive_expect_tx(&ctl.w_full[s], C::STAGE);
                        const int row = L.wrow + ((t * L.halves + h) * L.wgroups + og * NO / 64) * 192 + og * NO % 64;
                        if (NO == 64) {
                            tma_load_2d(wst + s * C::STAGE, &p.w, &ctl.w_full[s], 0, row);
                        } else {
                            for (int pt = 0; pt < 3; ++pt)
                                tma_load_2d(wst + s * C::STAGE + pt * NO * 128, &p.w, &ctl.w_full[s], 0, row + 64 * pt);
                        }
                    }
                if (bad) break;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        // The whole warp walks the items; one elected lane issues.  (The
        // descriptors are then warp-uniform values, a base plus compile-time
        // offsets: a loop run by one lane spent 55 cycles on each MMA, as
        // long as the MMAs of N = 64 and 128 take.)
        const uint64_t w_desc = sdesc_sw128(smem_u32(wst)), x_desc = sdesc_sw128(smem_u32(win));
        uint32_t g = 0, wn = 0, chain = 0;  // weight stages, window slots, accumulator chains
        for (int q = 0;; ++q) {
            const int it = next_item(q, 106);
            __syncwarp();
            if (elect_one()) mbar_arrive(&ctl.item_empty[q % kSpRing]);
            if (it < 0) break;
            int l, j, og;
            decode(it, l, j, og);
            const bool first = p.L[l].first != 0;
            const int halves = p.L[l].halves;
            bool ok = true;
            for (int h = 0; h < halves && ok; ++h, ++wn) {
                const int ws = wn % kSpSlots;
                if (!mbar_wait_warp(&ctl.win_full[ws], (wn / kSpSlots) & 1, p.wait_limit)) { fail(107); ok = false; break; }
                const uint64_t x = x_desc + (uint64_t)(ws * (kSpSlot >> 4));
                ok = first ? issue_half<NO, true>(ctl, tmem, x, w_desc, q % kSpGroups, g, chain, p.wait_limit)
                           : issue_half<NO, false>(ctl, tmem, x, w_desc, q % kSpGroups, g, chain, p.wait_limit);
                if (!ok) { fail(108); break; }
                if (elect_one()) mma_commit(&ctl.win_empty[ws]);
            }
            if (!ok) break;
        }
        // every MMA issued has completed before the CTA frees its tensor memory
        __syncwarp();
        if (elect_one()) {
            mma_commit(&ctl.mma_done);
            mbar_wait(&ctl.mma_done, 0, 1u << 20);
        }
    } else if (warp >= 4) {
        // ------------------------------------------------ epilogue
        const int quarter = warp & 3, ch = (((warp - 4) >> 2) & 1) * C::CH, group = (warp - 4) / kSpEpiWarps;
        const int row = quarter * 32 + lane;
        const uint32_t t_row = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)ch;
        const size_t ps = (size_t)p.cap_rows * p.pitch;
        uint32_t g = 0, used[2] = {0, 0};  // chains of all items; this group's uses of each accumulator
        for (int q = 0;; ++q) {
            const int it = next_item(q, 110);
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl.item_empty[q % kSpRing]);
            if (it < 0) break;
            int l, j, og;
            decode(it, l, j, og);
            const SpLayerDev &L = p.L[l];
            const int chains = L.halves * (((L.first ? 5 : 9) + kSpChain - 1) / kSpChain);
            if (q % kSpGroups != group) {  // the other group's item
                g += chains;
                continue;
            }
            float v[C::CH];
#pragma unroll
            for (int i = 0; i < C::CH; ++i) v[i] = 0.0f;
            bool bad = false;
            for (int c = 0; c < chains; ++c, ++g) {
                const int acc = g & 1;
                const uint32_t use = acc ? used[1]++ : used[0]++;
                if (!mbar_wait_warp(&ctl.acc_full[group][acc], use & 1, p.wait_limit)) { fail(111); bad = true; break; }
                tc_fence_after();
#pragma unroll
                for (int c0 = 0; c0 < C::CH; c0 += 8) {
                    uint32_t a2[8], a1[8], a0[8];
                    tmem_ld8(t_row + acc * C::ACC + 2 * NO + c0, a2);
                    tmem_ld8(t_row + acc * C::ACC + NO + c0, a1);
                    tmem_ld8(t_row + acc * C::ACC + c0, a0);
                    tmem_ld_wait();
                    if (c0 == C::CH - 8) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&ctl.acc_empty[acc]);
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        v[c0 + i] += __uint_as_float(a0[i]) + (__uint_as_float(a1[i]) + __uint_as_float(a2[i]));
                }
            }
            if (bad) break;
            const int q0 = j * kSpTile + row;
            const int o0 = og * NO + ch;
#pragma unroll
            for (int i = 0; i < C::CH / 4; ++i) {
                const float4 bv = __ldg(reinterpret_cast<const float4 *>(L.bias + o0) + i);
                v[4 * i] += bv.x;
                v[4 * i + 1] += bv.y;
                v[4 * i + 2] += bv.z;
                v[4 * i + 3] += bv.w;
            }
            if (L.act == LG_ACT_RELU) {
#pragma unroll
                for (int i = 0; i < C::CH; ++i) v[i] = act_fn(v[i], LG_ACT_RELU);
            } else if (L.act == LG_ACT_ELU) {
#pragma unroll
                for (int i = 0; i < C::CH; ++i) {
                    const float e = expf(v[i]) - 1.0f;  // as act_fn, without a branch a value
                    v[i] = v[i] > 0.0f ? v[i] : e;
                }
            }
            // L3 rows: (board, y, x) of the row, pad rows written as zeros.
            // L5 rows land on the L3 row of their point; the threads of x = 18
            // and of y = 19 also write the pads.
            const bool in_range = q0 < (L.first ? p.rows5 : p.rows);
            const int bl = L.first ? kL5Board : kL3Board, pt = L.first ? kL5Pitch : kL3Pitch;
            const int b = q0 / bl, r = q0 - b * bl, y = r / pt, x = r - y * pt;
            const bool point = in_range && y < kBoard && x < kBoard;
            if (L.out32) {
                if (point) {
                    float *dst = L.out32 + ((size_t)b * kPoints + y * kBoard + x) * L.cout + o0;
                    if ((L.cout & 3) == 0) {
#pragma unroll
                        for (int i = 0; i < C::CH / 4; ++i)
                            if (o0 + 4 * i < L.cout)
                                reinterpret_cast<float4 *>(dst)[i] =
                                    make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < C::CH; ++i)
                            if (o0 + i < L.cout) dst[i] = v[i];
                    }
                }
            } else {
                const int tgt = in_range && y < 20 ? b * kL3Board + y * kL3Pitch + x : -1;
                uint4 *tile = reinterpret_cast<uint4 *>(stg + (warp - 4) * kSpTileBytes);
#pragma unroll
                for (int c0 = 0; c0 < C::CH; c0 += 16) {
                    store_parts(v + c0, tgt, point, tile, lane, L.out + o0 + c0, ps, p.pitch);
                    if (L.first && tgt >= 0 && x == kBoard - 1)
                        store_zero_parts(L.out + (size_t)(tgt + 1) * p.pitch + o0 + c0, ps);
                }
            }
            // publish: the generic stores, ordered before other SMs' TMA reads
            fence_proxy_async_global();
            __syncwarp();
            if (lane == 0) {
                asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"((L.first ? flags5 : flags3) + j) : "memory");
            }
        }
    }

    __syncthreads();
    if (abort_flag && tid == 0) {
        for (int i = 0; i < kSpSlots; ++i) {
            mbar_wait(&ctl.win_full[i], 0, 1u << 16);
            mbar_wait(&ctl.win_full[i], 1, 1u << 16);
        }
        for (int i = 0; i < C::STAGES; ++i) {
            mbar_wait(&ctl.w_full[i], 0, 1u << 16);
            mbar_wait(&ctl.w_full[i], 1, 1u << 16);
        }
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
    if (warp == 1) tmem_relinquish();
    // the last CTA to leave zeroes the counters for the next launch
    int *const exit_ctr = item_ctr + 1;
    if (tid == 0) {
        __threadfence();
        ctl.last_out = atomicAdd(exit_ctr, 1) == (int)gridDim.x - 1;
        if (ctl.last_out) __threadfence();
    }
    __syncthreads();
    if (ctl.last_out)
        for (int i = tid; i < n3 + n5 + 2; i += blockDim.x) p.flags[i] = 0;
}

// FP32 weights wt[k*k][cin][cout] -> [tap][half][group][part][64 outputs][64
// inputs] (k = 5: a tap is a vertical one, its inputs dx * cin + c), zero
// past the real channels.  Parts by truncation; a part that comes out zero is
// the smallest normal number with the weight's sign (unless the weight is
// below 1e-25), so that no part turns an infinite activation into a NaN.
// flip (k = 3): wt is [9][cout][cin], the weights of the conv whose input
// gradient this is -- taps in reverse, channels transposed.
__global__ void __launch_bounds__(256) split_weights_kernel(const float *__restrict__ wt, int k, int cin, int cout,
                                                            int kpad, int opad, bool flip, __nv_bfloat16 *__restrict__ out,
                                                            int n) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int kk = i % kpad, o = i / kpad % opad, t = i / kpad / opad;
    const int dx = k == 5 ? kk / cin : 0, ci = k == 5 ? kk - dx * cin : kk;
    float w = 0.0f;
    if (o < cout && kk < (k == 5 ? 5 * cin : cin))
        w = flip ? wt[((size_t)(k * k - 1 - t) * cout + o) * cin + ci]
                 : wt[((size_t)(k == 5 ? t * 5 + dx : t) * cin + ci) * cout + o];
    const float tiny = fabsf(w) > 1e-25f ? copysignf(1.17549435e-38f, w) : 0.0f;
    uint16_t *dst = reinterpret_cast<uint16_t *>(out) +
                    (((size_t)t * (kpad / 64) + kk / 64) * (opad / 64) + o / 64) * 3 * 4096 + (size_t)(o % 64) * 64 + kk % 64;
    float r = w;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const float part = __uint_as_float(__float_as_uint(r) & 0xFFFF0000u);
        r -= part;
        dst[p * 4096] = (uint16_t)(__float_as_uint(part == 0.0f ? tiny : part) >> 16);
    }
}

// ------------------------------------------------------------------ host

size_t split_flag_ints(int B) {
    return (size_t)(B * kL3Board + kSpTile - 1) / kSpTile + (size_t)(B * kL5Board + kSpTile - 1) / kSpTile + 2;
}

int split_pad(int channels) { return (channels + 63) / 64 * 64; }

size_t split_weight_elems(int k, int cin, int cout) {
    const int kper = k == 5 ? 5 * cin : cin, taps = k == 5 ? 5 : 9;
    return (size_t)taps * split_pad(kper) * split_pad(cout) * 3;
}

void launch_split_weights(const float *wt, int k, int cin, int cout, __nv_bfloat16 *out, cudaStream_t s, bool flip) {
    const int n = (int)(split_weight_elems(k, cin, cout) / 3);
    split_weights_kernel<<<(n + 255) / 256, 256, 0, s>>>(wt, k, cin, cout, split_pad(k == 5 ? 5 * cin : cin),
                                                         split_pad(cout), flip, out, n);
}

int split_init_device() {
    cudaError_t e = cudaFuncSetAttribute(split_trunk_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SpCfg<64>::SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(split_trunk_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, SpCfg<32>::SMEM);
    if (e != cudaSuccess) {
        lg_set_error("cudaFuncSetAttribute(split trunk): %s", cudaGetErrorString(e));
        return LG_ERR_CUDA;
    }
    return LG_OK;
}

int launch_split_trunk(const SplitTrunk &T, cudaStream_t s, int sm_count) {
    if (T.nl < 1 || T.nl > kSpMaxLayers || T.B < 1 || T.B * kL3Board > T.cap_rows || T.pitch % 64) {
        lg_set_error("launch_split_trunk: bad arguments");
        return LG_ERR_ARG;
    }
    SpParams p{};
    p.nl = T.nl;
    p.rows = T.B * kL3Board;
    p.rows5 = T.l5 ? T.B * kL5Board : 0;
    p.cap_rows = T.cap_rows;
    p.pitch = T.pitch;
    p.flags = T.flags;
    p.err = T.err;
    p.wait_limit = T.wait_limit ? T.wait_limit : kSpWait;
    p.poll_limit = T.poll_limit ? T.poll_limit : kSpPolls;
    p.stall_item = -1;
    const int n3 = (p.rows + kSpTile - 1) / kSpTile, n5 = (p.rows5 + kSpTile - 1) / kSpTile;
    int wide = 0;
    for (int l = 0; l < T.nl; ++l) wide = std::max(wide, T.L[l].groups);
    // 32-channel items while 64-channel ones would leave a third of the SMs
    // without any: their MMAs (N = 96, 64, 32) run at two thirds of the rate,
    // but twice as many SMs work on a layer.  Policy + value pair of the
    // benchmark nets, us, 32 / 64 channels: 5 positions 286 / 341, 16 positions
    // (100 wide items) 316 / 351, 20 positions (126) 355 / 359, 24 positions 405 /
    // 360.
    const int no = 3 * n3 * wide <= 2 * sm_count ? 32 : 64;
    int wrows = 0, items = 0, done3 = 0;
    for (int l = 0; l < T.nl; ++l) {
        const SplitLayer &S = T.L[l];
        SpLayerDev &L = p.L[l];
        L.first = l == 0 && T.l5;
        L.halves = S.halves;
        L.groups = S.groups * 64 / no;
        L.wgroups = S.groups;
        L.wrow = wrows;
        L.item0 = items;
        // a tile's counter once the layer before is complete there (the first
        // layer counts in its own tiles)
        if (l > 0) {
            const int n = kSpEpiWarps * p.L[l - 1].groups;
            L.need = p.L[l - 1].first ? n : done3 += n;
        }
        L.act = T.act;
        L.bias = S.bias;
        const bool last = l + 1 == T.nl;
        L.out = last ? nullptr : T.buf[(l + 1) & 1];
        L.out32 = last ? T.out32 : nullptr;
        L.cout = S.cout;
        wrows += (L.first ? 5 : 9) * S.halves * S.groups * 192;
        items += (L.first ? n5 : n3) * L.groups;
    }
    p.nitems = items;
    if (T.stall && T.nl > 1) p.stall_item = p.L[1].item0;
    int rc = encode_map_3d_bf16(&p.in[0], T.buf[0], T.pitch, p.rows, 3, T.cap_rows, 64, kSpWin3);
    if (!rc) rc = encode_map_3d_bf16(&p.in[1], T.buf[1], T.pitch, p.rows, 3, T.cap_rows, 64, kSpWin3);
    p.in5 = p.in[0];
    if (!rc && T.l5) rc = encode_map_2d_bf16(&p.in5, T.l5, (uint64_t)T.L[0].halves * 64, (uint64_t)p.rows5, 64, kSpWin5);
    if (!rc) rc = encode_map_2d_bf16(&p.w, T.w, 64, (uint64_t)wrows, 64, no == 64 ? 192 : 32);
    if (rc) return rc;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(std::min(items, sm_count));
    cfg.blockDim = dim3(kSpThreads);
    cfg.dynamicSmemBytes = no == 64 ? SpCfg<64>::SMEM : SpCfg<32>::SMEM;
    cfg.stream = s;
    // items are claimed in order, so what an item waits for belongs to a
    // running CTA: no co-residency needed
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, no == 64 ? split_trunk_kernel<64> : split_trunk_kernel<32>, p);
    if (e != cudaSuccess) {
        lg_set_error("split trunk launch: %s", cudaGetErrorString(e));
        return LG_ERR_CUDA;
    }
    return LG_OK;
}

}  // namespace lg
