// surrogate.cuh — the BF16 surrogate MLP on the 5th-generation tensor cores.
//
// Network (the surrogate configuration): 5 -> 256 -> 256 -> 256 -> 256 -> 4,
// SiLU after each hidden layer, BF16 weights and activations, FP32
// accumulation, FP32 biases. A pair of CTAs (a cluster of two, one per SM)
// walks 256-row tiles of the input, 128 rows each:
//
//   * tcgen05.mma.cta_group::2 (M = 256, N = 256 or 16, K = 16): each CTA holds
//     its own rows of A and D and half of the weights' N rows, so all the
//     network's weights stay in shared memory (208 KB per SM) for the whole
//     launch, and nothing is streamed per tile.
//   * B operands (weights, N x K) sit in shared memory, K-major, in the
//     no-swizzle core-matrix layout of the UMMA shared-memory descriptor:
//     element (row, k) at byte (row % 8) * 16 + (row / 8) * SBO + (k / 8) * 128
//     + (k % 8) * 2, SBO = (K / 8) * 128.
//   * Layer 1 reads its 16-wide padded input from shared memory: each feature as
//     two BF16 terms (hi, lo) against W1 repeated in two column groups, so the
//     inputs keep 16 significant bits (pack_input_row). The other layers read
//     their activations from tensor memory, where the epilogue left them in
//     place of the accumulator columns they came from.
//   * Epilogue: 8 warps read the accumulator with tcgen05.ld, add the bias,
//     apply SiLU x (1 + tanh(x / 2)) / 2 (one MUFU op), round to BF16 and write
//     the next layer's A operand with tcgen05.st, 64 columns at a time. The MMAs
//     of the next layer take each 64 columns of K as soon as both CTAs have
//     written them, so tensor core and epilogue work at the same time.
//
// Every mbarrier wait is bounded by the device clock; a role whose wait runs out
// records an error flag and leaves its loop, the others run out after it, and the
// CTAs meet (and free their TMEM) at the end in any case.
#pragma once

#include <cuda.h>  // CUtensorMap (a plain 128-byte descriptor type; nothing from the driver library is linked)
#include <cuda_bf16.h>
#include <cstdint>

#include "tcgen05.cuh"

namespace sirius {
namespace surrogate {

constexpr int kIn = 5, kInPad = 16, kHid = 256, kOut = 4, kOutPad = 16, kTileM = 128;
// packed weight image (bytes): W2 | W3 | W4 | W1 | W5 | b1 b2 b3 b4 (256 f32 each) | b5 (16 f32)
constexpr int kBigBytes = kHid * kHid * 2;            // 131072
constexpr int kW1Bytes = kHid * kInPad * 2;           // 8192
constexpr int kW5Bytes = kOutPad * kHid * 2;          // 8192
constexpr int kBiasBytes = (4 * kHid + kOutPad) * 4;  // 4160
constexpr int kOffW1 = 3 * kBigBytes, kOffW5 = kOffW1 + kW1Bytes, kOffBias = kOffW5 + kW5Bytes;
constexpr int kImageBytes = kOffBias + kBiasBytes;
// host parameter vector (PyTorch nn.Linear order, out x in): W1 b1 W2 b2 W3 b3 W4 b4 W5 b5
constexpr long long kParams = (long long)kHid * kIn + kHid + 3LL * (kHid * kHid + kHid) + kOut * kHid + kOut;

using namespace ::sirius::tc;

#ifdef __CUDACC__
// ---------------------------------------------------------------------------
// The MLP kernel.
//
// What bounds it: per 128 rows and hidden layer an SM needs 2048 cycles of tensor
// core (8.4 M multiply-adds) and 2048 of MUFU (32768 tanh at 16 a cycle). A layer's
// MMAs may start on K columns 0..63 when the epilogue of the layer before has done a
// quarter, so the two overlap but for the last quarter's MMAs (512 cycles) and the
// hand-offs between the CTAs (about 200 cycles to the issuer, 350 back): a layer takes
// about 3600 cycles. 2^22 rows: 2.91 -> 1.79 ms (573 -> 930 TFLOP/s, 57 % of the
// measured bf16 peak; MUFU 55 % and tensor pipe 43 % active) against one CTA per tile
// with a 128 KB weight buffer refilled per layer, where the two took turns; outputs
// bit for bit the same. Eight epilogue warps instead of sixteen take 1 % more; MMAs of
// N = 128, which let the first half's epilogue start earlier, 22 % more (they run at
// half the rate of N = 256 with A in tensor memory).
//
// TMEM (512 columns): two halves U and V of 256. Layer 1 accumulates in U, layer 2 in
// V, layer 3 in U, layer 4 in V, layer 5 (16 columns) in U; the next tile starts with
// the halves exchanged. Epilogue warp w owns lanes 32 (w % 4).. and, of each 64
// columns, the 16 at 16 (w / 4): it writes their 16 BF16 activations, one K step of the
// next layer, into the first 8 of those same columns, so no warp overwrites what
// another has yet to read.
//
// Roles: warps 0..15 epilogue (the first 8 also the input rows); warp 16 copies the
// CTA's weights in and, in the even CTA, one of its threads issues every MMA of the
// pair; in the even CTA a thread of warp 17 takes tiles from a counter (a cluster that
// starts late, its SMs still busy with another kernel, takes fewer).
// ---------------------------------------------------------------------------
constexpr int kEpiWarps = 16, kPairThreads = 32 * (kEpiWarps + 2);
constexpr int kSmW = 0, kSmW1 = 3 * (kBigBytes / 2), kSmW5 = kSmW1 + kW1Bytes / 2, kSmX = kSmW5 + kW5Bytes / 2,
              kSmBias = kSmX + kTileM * kInPad * 2, kSmTile = kSmBias + kBiasBytes, kSmBar = kSmTile + 16;
enum PairBar : int {  // mbarriers, 8 bytes each from kSmBar
    kBarW = 0,          // [4] this CTA's weights have landed: W1 and W5, W2, W3, W4
    kBarWReady = 4,     // [4] even CTA: the other CTA's have
    kBarX = 8,          // even CTA: both CTAs' input rows are in shared memory, and every epilogue warp has read
                        // the tile's index
    kBarA = 9,          // [4] even CTA: 64 columns of activations are in both CTAs' TMEM
    kBarD = 13,         // a hidden layer's accumulator is complete
    kBarOut = 14,       // the output layer's is
    kBarTile = 15,      // the next tile's index is in shared memory
    kBarFirst = 16,     // even CTA: a tile's first layer is complete
    kBarCount = 17
};
constexpr int kSmSlot = kSmBar + 8 * (kBarCount + 1), kPairSmBytes = kSmSlot + 16;
static_assert(kPairSmBytes <= 227 * 1024, "the MLP kernel's shared memory fits one SM");
static_assert(kSmTile % 16 == 0, "the tile index and the mbarriers are aligned");
constexpr uint32_t kTmemCols = 512;

// the TMEM column, within its half, of K step s (16 elements) of the activations
__device__ __forceinline__ uint32_t act_column(int s) { return uint32_t(16 * s); }

// The training forward pass over the same network: input rows already packed (BF16, 16
// wide), the weights the optimiser's row-major BF16 copies (layers 2..5 by TMA with the
// 128-byte swizzle, or by plain loads into the core-matrix layout where the driver encodes no
// tensor maps), and every layer's pre-activations (FP32) and activations (BF16) kept for the
// backward pass.
enum Forward : int { kInfer = 0, kTrainTma = 1, kTrainPlain = 2 };

struct TrainForward {
    const __nv_bfloat16* x0;  // n x 16
    const __nv_bfloat16* w1;  // 256 x 16
    const float* bias[5];
    float* z[4];              // n x 256
    __nv_bfloat16* h[4];      // n x 256
    CUtensorMap w[4];         // W2, W3, W4 in 128 x 64 boxes, W5 (16 x 256) in 8 x 64 boxes (kTrainTma)
    const __nv_bfloat16* wp[4];  // the same weights, row-major (kTrainPlain)
};

// 32 bytes of global memory (32-byte aligned) in one instruction
__device__ __forceinline__ void st_global_32(void* p, const uint32_t r[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

template <int MODE>
__device__ __forceinline__ void mlp_pair_body(const unsigned char* __restrict__ wimg, const float* __restrict__ feat,
                                              long long n, float* __restrict__ out, volatile int* err,
                                              unsigned long long* tile_counter, unsigned long long wait_limit_ns,
                                              const unsigned* __restrict__ rows, const TrainForward* tf) {
    constexpr bool TRAIN = MODE != kInfer;
    extern __shared__ __align__(1024) unsigned char sm[];
    float* bias = reinterpret_cast<float*>(sm + kSmBias);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + kSmSlot);
    volatile unsigned long long* tile_s = reinterpret_cast<volatile unsigned long long*>(sm + kSmTile);
    const uint32_t sm0 = smem_u32(sm), bar0 = sm0 + kSmBar;
    auto bar = [&](int b) { return bar0 + 8u * uint32_t(b); };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const long long ntiles = (n + 2 * kTileM - 1) / (2 * kTileM);

    if (tid == 0) {
        for (int i = 0; i < 4; ++i) {
            mbar_init(bar(kBarW + i), 1);
            mbar_init(bar(kBarWReady + i), 1);
            mbar_init(bar(kBarA + i), 2 * kEpiWarps);
        }
        mbar_init(bar(kBarX), 2 * kEpiWarps);
        mbar_init(bar(kBarD), 1);
        mbar_init(bar(kBarOut), 1);
        mbar_init(bar(kBarTile), 1);
        mbar_init(bar(kBarFirst), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kEpiWarps) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    if constexpr (TRAIN) {
        for (int i = tid; i < 4 * kHid; i += kPairThreads) bias[i] = tf->bias[i / kHid][i % kHid];
        if (tid < kOutPad) bias[4 * kHid + tid] = tid < kOut ? tf->bias[4][tid] : 0.f;
        // this CTA's 128 rows of W1, into the core-matrix layout
        for (int i = tid; i < kTileM * 2; i += kPairThreads)
            *reinterpret_cast<uint4*>(sm + kSmW1 + packed_offset(i >> 1, (i & 1) * 8, kInPad)) =
                reinterpret_cast<const uint4*>(tf->w1 + size_t(rank) * kTileM * kInPad)[i];
        if constexpr (MODE == kTrainPlain) {  // and of W2, W3, W4 (8 rows of W5)
            constexpr int kPieces = kHid / 8;
            for (int i = tid; i < (3 * kTileM + kOutPad / 2) * kPieces; i += kPairThreads) {
                const int l = i / (kTileM * kPieces), r = i / kPieces - l * kTileM, k = 8 * (i % kPieces);
                const int row = int(rank) * (l < 3 ? kTileM : kOutPad / 2) + r;
                *reinterpret_cast<uint4*>(sm + (l < 3 ? kSmW + l * (kBigBytes / 2) : kSmW5) + packed_offset(r, k, kHid)) =
                    *reinterpret_cast<const uint4*>(tf->wp[l] + size_t(row) * kHid + k);
            }
        }
        fence_async_smem();
    } else {
        for (int i = tid; i < kBiasBytes / 16; i += kPairThreads)
            reinterpret_cast<float4*>(bias)[i] = reinterpret_cast<const float4*>(wimg + kOffBias)[i];
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers and TMEM are set up
    tc_fence_after();
    const uint32_t tmem = *tslot;
    bool ok = true;

    if (warp == kEpiWarps) {
        if (lane == 0) {
            // this CTA's half of the weights: each layer's N rows 128 rank.. (8 rank.. of W5's 16)
            auto copy = [&](int dst, size_t src, uint32_t bytes, int b) {
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sm0 + dst),
                    "l"(wimg + src + size_t(rank) * bytes), "r"(bytes), "r"(bar(b))
                    : "memory");
            };
            if constexpr (MODE == kTrainPlain) {  // in place since the CTAs met
                for (int i = 0; i < 4; ++i) mbar_expect_tx(bar(kBarW + i), 0);
            } else if constexpr (TRAIN) {
                mbar_expect_tx(bar(kBarW), kW5Bytes / 2);
                for (int c = 0; c < 4; ++c)
                    tma_load_2d(sm0 + kSmW5 + c * 1024, &tf->w[3], 64 * c, 8 * int(rank), bar(kBarW));
                for (int l = 0; l < 3; ++l) {
                    mbar_expect_tx(bar(kBarW + 1 + l), kBigBytes / 2);
                    for (int c = 0; c < 4; ++c)
                        tma_load_2d(sm0 + kSmW + l * (kBigBytes / 2) + c * 16384, &tf->w[l], 64 * c, 128 * int(rank),
                                    bar(kBarW + 1 + l));
                }
            } else {
                mbar_expect_tx(bar(kBarW), kW1Bytes / 2 + kW5Bytes / 2);
                copy(kSmW1, kOffW1, kW1Bytes / 2, kBarW);
                copy(kSmW5, kOffW5, kW5Bytes / 2, kBarW);
                for (int l = 0; l < 3; ++l) {
                    mbar_expect_tx(bar(kBarW + 1 + l), kBigBytes / 2);
                    copy(kSmW + l * (kBigBytes / 2), size_t(l) * kBigBytes, kBigBytes / 2, kBarW + 1 + l);
                }
            }
            if (rank == 1)
                for (int i = 0; i < 4; ++i) {
                    ok = mbar_wait(bar(kBarW + i), 0, wait_limit_ns) && ok;
                    mbar_arrive_cluster(peer_addr(bar(kBarWReady + i), 0));
                }
            if (rank == 0) {
                const uint32_t id256 = instr_desc_pair(kHid), id16 = instr_desc_pair(kOutPad);
                const uint32_t sbo1 = (kInPad / 8) * 128, sbo = (kHid / 8) * 128;
                // the descriptor of K step s of a layer's weights; chunk: bytes of 64 columns (swizzled)
                auto wdesc = [&](uint32_t w, int s, uint32_t chunk) {
                    return MODE == kTrainTma ? smem_desc_sw128(w + uint32_t(s >> 2) * chunk + uint32_t(s & 3) * 32)
                                             : smem_desc(w + uint32_t(s) * 256, sbo);
                };
                uint32_t ph_x = 0, ph_a = 0, ph_out = 0, ph_tile = 0;
                auto operand = [&](int c) {  // 64 columns of the operand are there
                    ok = mbar_wait_cluster(bar(kBarA + c), ph_a, wait_limit_ns);
                    tc_fence_after();
                    return ok;
                };
                int n_w = 0;  // weight groups known to be in both CTAs' shared memory
                auto weights = [&](int i) {
                    for (; ok && n_w <= i; ++n_w)
                        ok = mbar_wait(bar(kBarW + n_w), 0, wait_limit_ns) &&
                             mbar_wait_cluster(bar(kBarWReady + n_w), 0, wait_limit_ns);
                    return ok;
                };
                auto more = [&]() {  // whether there is another tile
                    ok = ok && mbar_wait_cluster(bar(kBarTile), ph_tile, wait_limit_ns);
                    ph_tile ^= 1;
                    return ok && (long long)*tile_s < ntiles;
                };
                uint32_t U = tmem, V = tmem + 256;
                while (more()) {
                    if (!weights(0) || !(ok = mbar_wait_cluster(bar(kBarX), ph_x, wait_limit_ns))) break;
                    ph_x ^= 1;
                    tc_fence_after();
                    mma_bf16_pair(U, smem_desc(sm0 + kSmX, sbo1), smem_desc(sm0 + kSmW1, sbo1), id256, 0u);
                    mma_commit_pair(bar(kBarD));
                    mma_commit_pair_own(bar(kBarFirst));
                    uint32_t A = U, D = V;
                    for (int l = 0; l < 3; ++l) {  // layers 2, 3, 4
                        if (!weights(1 + l)) break;
                        const uint32_t wl = sm0 + kSmW + uint32_t(l) * (kBigBytes / 2);
                        for (int c = 0; c < 4; ++c) {
                            if (!operand(c)) break;
#pragma unroll
                            for (int s = 4 * c; s < 4 * c + 4; ++s)
                                mma_bf16_ts_pair(D, A + act_column(s), wdesc(wl, s, 16384), id256, s > 0);
                        }
                        if (!ok) break;
                        ph_a ^= 1;
                        mma_commit_pair(bar(kBarD));
                        const uint32_t t = A;
                        A = D;
                        D = t;
                    }
                    for (int c = 0; ok && c < 4; ++c) {  // the output layer
                        if (!operand(c)) break;
#pragma unroll
                        for (int s = 4 * c; s < 4 * c + 4; ++s)
                            mma_bf16_ts_pair(D, A + act_column(s), wdesc(sm0 + kSmW5, s, 1024), id16, s > 0);
                    }
                    if (!ok) break;
                    ph_a ^= 1;
                    mma_commit_pair(bar(kBarOut));
                    // the next tile's first layer overwrites the operand of the output layer
                    if (!(ok = mbar_wait(bar(kBarOut), ph_out, wait_limit_ns))) break;
                    ph_out ^= 1;
                    const uint32_t t = U;
                    U = V;
                    V = t;
                }
                if (!ok) {  // whatever was issued drains before the end, and no copy lands after it
                    mma_commit_pair(bar(kBarOut));
                    mbar_wait(bar(kBarOut), ph_out, wait_limit_ns);
                }
                for (; n_w < 4; ++n_w) ok = mbar_wait(bar(kBarW + n_w), 0, wait_limit_ns) && ok;
            }
            if (!ok) *err = 1;
        }
        __syncwarp();
    } else if (warp == kEpiWarps + 1) {
        if (rank == 0 && lane == 0) {
            auto next_tile = [&]() {  // taken from the counter and told to both CTAs
                const unsigned long long t = atomicAdd(tile_counter, 1ull);
#pragma unroll
                for (uint32_t r = 0; r < 2; ++r) {
                    st_cluster_u64(peer_addr(sm0 + kSmTile, r), t);
                    mbar_arrive_cluster(peer_addr(bar(kBarTile), r));
                }
                return (long long)t;
            };
            // the next one once a tile's first layer is complete: it waited for the arrivals of
            // all epilogue warps of both CTAs on kBarX, which come after they have read the
            // tile's index, and the issuer had read it too. Every
            // cluster takes one index past the end, and the last to do so leaves the counter
            // at zero for the next launch (after an error the host does).
            long long t = next_tile();
            for (uint32_t ph = 0; ok && t < ntiles; ph ^= 1)
                if ((ok = mbar_wait(bar(kBarFirst), ph, wait_limit_ns))) t = next_tile();
            if (t == ntiles + (long long)(gridDim.x / 2) - 1) *tile_counter = 0;
            if (!ok) *err = 1;
        }
        __syncwarp();
    } else {
        const uint32_t lanes = uint32_t((warp & 3) * 32) << 16;
        const int group = warp >> 2;
        const int in_r = tid >> 1, in_chunk = tid & 1;
        float xin[kIn];
        uint4 xrow;  // TRAIN: this thread's half row
        // this thread's input row (tid / 2) of a tile; rows past n read as zeros, which
        // pack to zero operands
        auto fetch_row = [&](long long t) {
            const long long gr = t * (2 * kTileM) + long(rank) * kTileM + in_r;
            const bool live = gr < n && in_r < kTileM;
            if constexpr (TRAIN) {
                xrow = live ? reinterpret_cast<const uint4*>(tf->x0)[2 * gr + in_chunk] : make_uint4(0, 0, 0, 0);
                return;
            }
            const float* f = feat + (live ? (rows ? (long long)rows[gr] : gr) : 0LL) * kIn;
#pragma unroll
            for (int k = 0; k < kIn; ++k) xin[k] = live ? f[k] : 0.f;
        };
        const uint32_t bar_x = peer_addr(bar(kBarX), 0);
        // every warp arrives, also those without rows: the first layer, after which the next
        // index is told, then waits until all have read this one. The arrival is a release:
        // the rows are ordinary stores of 32 lanes, read by an MMA that the other CTA may issue
        auto store_row = [&]() {
            if (in_r < kTileM) {  // (whole warps)
                if constexpr (!TRAIN) {
                    uint4 c0, c1;
                    pack_input_row(xin, c0, c1);
                    xrow = in_chunk == 0 ? c0 : c1;
                }
                *reinterpret_cast<uint4*>(sm + kSmX + packed_offset(in_r, in_chunk * 8, kInPad)) = xrow;
                fence_async_smem();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(bar_x);
        };
        auto all = [&](bool v) { return __all_sync(0xffffffffu, v) != 0; };
        uint32_t ph_tile = 0, ph_d = 0, ph_out = 0;
        uint32_t bar_a[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) bar_a[c] = peer_addr(bar(kBarA + c), 0);
        auto get_tile = [&](long long& t) {
            const bool got = all(mbar_wait_cluster(bar(kBarTile), ph_tile, wait_limit_ns));
            ph_tile ^= 1;
            t = (long long)*tile_s;
            return got;
        };
        long long tile = 0;
        ok = get_tile(tile);
        if (ok && tile < ntiles) {
            fetch_row(tile);
            store_row();
        }
        uint32_t U = tmem, V = tmem + 256;
        while (ok && tile < ntiles) {
            long long next = ntiles;
            uint32_t src = U;
            // the row of this thread's TMEM lane
            const long long gr_out = tile * (2 * kTileM) + long(rank) * kTileM + (warp & 3) * 32 + lane;
#pragma unroll 1
            for (int l = 0; l < 4; ++l) {
                if (!(ok = all(mbar_wait(bar(kBarD), ph_d, wait_limit_ns)))) break;
                ph_d ^= 1;
                tc_fence_after();
                const uint32_t col = src + lanes + uint32_t(16 * group);
                const float4* b4 = reinterpret_cast<const float4*>(bias + l * kHid + 16 * group);
                uint32_t v[2][16];
                tmem_ld16_async(col, v[0]);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    tmem_wait_ld16(v[c & 1]);
                    if (c < 3) tmem_ld16_async(col + 64 * (c + 1), v[(c + 1) & 1]);
                    uint32_t r[8];
                    if constexpr (TRAIN) {  // Z = acc + bias, kept
                        uint32_t* q = v[c & 1];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float4 b = b4[16 * c + i];
                            q[4 * i] = __float_as_uint(__uint_as_float(q[4 * i]) + b.x);
                            q[4 * i + 1] = __float_as_uint(__uint_as_float(q[4 * i + 1]) + b.y);
                            q[4 * i + 2] = __float_as_uint(__uint_as_float(q[4 * i + 2]) + b.z);
                            q[4 * i + 3] = __float_as_uint(__uint_as_float(q[4 * i + 3]) + b.w);
                        }
                        if (gr_out < n) {
                            float* zr = tf->z[l] + gr_out * kHid + 64 * c + 16 * group;
                            st_global_32(zr, q);
                            st_global_32(zr + 8, q + 8);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 b = TRAIN ? make_float4(0.f, 0.f, 0.f, 0.f) : b4[16 * c + i];
                        const uint32_t* q = v[c & 1] + 4 * i;
                        const float2 y0 = silu_bias2(make_float2(__uint_as_float(q[0]), __uint_as_float(q[1])),
                                                     make_float2(b.x, b.y));
                        const float2 y1 = silu_bias2(make_float2(__uint_as_float(q[2]), __uint_as_float(q[3])),
                                                     make_float2(b.z, b.w));
                        r[2 * i] = pack_bf16x2(y0.x, y0.y);
                        r[2 * i + 1] = pack_bf16x2(y1.x, y1.y);
                    }
                    tmem_st8(col + 64 * c, r);
                    if constexpr (TRAIN)
                        if (gr_out < n) st_global_32(tf->h[l] + gr_out * kHid + 64 * c + 16 * group, r);
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster_relaxed(bar_a[c]);
                }
                src = src == U ? V : U;
                if (l == 1) {  // the next tile's rows: on their way during layer 3
                    if (!(ok = get_tile(next))) break;
                    if (next < ntiles) fetch_row(next);
                } else if (l == 2 && next < ntiles) {
                    store_row();
                }
            }
            if (!ok) break;
            if (!(ok = all(mbar_wait(bar(kBarOut), ph_out, wait_limit_ns)))) break;
            ph_out ^= 1;
            tc_fence_after();
            if (warp < 4) {
                float v[16];
                tmem_ld16(U + lanes, v);
                if (gr_out < n) {
                    const float* b5 = bias + 4 * kHid;
                    *reinterpret_cast<float4*>(out + (rows ? (long long)rows[gr_out] : gr_out) * kOut) =
                        make_float4(v[0] + b5[0], v[1] + b5[1], v[2] + b5[2], v[3] + b5[3]);
                }
                tc_fence_before();
            }
            const uint32_t t = U;
            U = V;
            V = t;
            tile = next;
        }
        if (!ok && lane == 0) *err = 1;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // neither CTA leaves while the other may still reach its memory
    tc_fence_after();
    if (warp == kEpiWarps)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
    mlp_pair_kernel(const unsigned char* __restrict__ wimg, const float* __restrict__ feat, long long n,
                    float* __restrict__ out, volatile int* err, unsigned long long* tile_counter,
                    unsigned long long wait_limit_ns, const unsigned* __restrict__ rows) {
    mlp_pair_body<kInfer>(wimg, feat, n, out, err, tile_counter, wait_limit_ns, rows, nullptr);
}

// n rows of the training set's batch; y: n x 4. Bound by what it keeps, 6 KB a row: 201 MB
// for 32768 rows are 31 us at the measured copy bandwidth, and the stores, 32 bytes of a
// row per lane, take the SMs' store path about twice that (67 us; five GEMM launches that
// read every activation back took 95).
template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
    train_forward_kernel(const __grid_constant__ TrainForward tf, long long n, float* __restrict__ y, volatile int* err,
                         unsigned long long* tile_counter, unsigned long long wait_limit_ns) {
    mlp_pair_body<MODE>(nullptr, nullptr, n, y, err, tile_counter, wait_limit_ns, nullptr, &tf);
}
#endif  // __CUDACC__

// Host: pack the parameter vector (W1 b1 ... W5 b5, nn.Linear order) into the
// kernel's weight image (BF16 core-matrix layouts, FP32 biases).
inline void pack_weights(const float* p, unsigned char* img) {
    auto bf16 = [](float x) -> uint16_t {
        uint32_t u;
        __builtin_memcpy(&u, &x, 4);
        if ((u & 0x7f800000u) == 0x7f800000u) return uint16_t(u >> 16);  // inf / nan
        const uint32_t r = 0x7fffu + ((u >> 16) & 1u);                  // round to nearest even
        return uint16_t((u + r) >> 16);
    };
    for (int i = 0; i < kImageBytes; ++i) img[i] = 0;
    auto put = [&](int off, int rows, int K, int kin, const float* W) {
        for (int r = 0; r < rows; ++r)
            for (int k = 0; k < kin; ++k) {
                const uint16_t h = bf16(W[r * kin + k]);
                __builtin_memcpy(img + off + packed_offset(r, k, K), &h, 2);
            }
    };
    const float* W1 = p;
    const float* b1 = W1 + kHid * kIn;
    const float* W2 = b1 + kHid;
    const float* b2 = W2 + kHid * kHid;
    const float* W3 = b2 + kHid;
    const float* b3 = W3 + kHid * kHid;
    const float* W4 = b3 + kHid;
    const float* b4 = W4 + kHid * kHid;
    const float* W5 = b4 + kHid;
    const float* b5 = W5 + kOut * kHid;
    put(0, kHid, kHid, kHid, W2);
    put(kBigBytes, kHid, kHid, kHid, W3);
    put(2 * kBigBytes, kHid, kHid, kHid, W4);
    put(kOffW1, kHid, kInPad, kIn, W1);
    for (int r = 0; r < kHid; ++r)  // columns kIn..2 kIn - 1 repeat W1 for the inputs' low BF16 terms
        for (int k = 0; k < kIn; ++k) {
            const uint16_t h = bf16(W1[r * kIn + k]);
            __builtin_memcpy(img + kOffW1 + packed_offset(r, kIn + k, kInPad), &h, 2);
        }
    put(kOffW5, kOut, kHid, kHid, W5);
    float* bias = reinterpret_cast<float*>(img + kOffBias);
    for (int i = 0; i < kHid; ++i) {
        bias[i] = b1[i];
        bias[kHid + i] = b2[i];
        bias[2 * kHid + i] = b3[i];
        bias[3 * kHid + i] = b4[i];
    }
    for (int i = 0; i < kOut; ++i) bias[4 * kHid + i] = b5[i];
}

}  // namespace surrogate
}  // namespace sirius
