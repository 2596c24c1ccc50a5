// 3x3 convolutions (stride 1, zero padding 1) on NHWC BF16 activations as
// implicit GEMMs on the sm_100a tensor cores (tcgen05.mma kind::f16, BF16 x
// BF16 -> FP32 in TMEM). These are the dense contractions of the learned
// kernel-predicting denoiser (kpcn.cu); the reference has no learned part.
//
//   forward : out[p, n] = sum_{t, c} in[p + off(t), c] * w[t][n][c]
//   data grad: out[p, n] = sum_{t, c} g[p - off(t), c] * wt[t][n][c]
//             (wt = w transposed per tap, flip = 1)
//   weights  : dW[t][n][c] += sum_p in[p + off(t), c] * g[p, n]
//
// Three kernels:
//   k_conv3x3             forward and data gradient: 128 pixels as the MMA's
//                         M, output channels as its N; blocks of input rows
//                         TMA-loaded in swizzled layouts, the 9 taps as
//                         row-shifted descriptors, weights resident or
//                         streamed.
//   k_conv3x3_wgrad_ring  weight gradient on a ring of input rows per column
//                         strip, MN-major, accumulators resident in TMEM
//                         over each CTA's pixel range.
//   k_conv3x3_wgrad       weight gradient for layers whose ring does not fit
//                         shared memory: (tap, channel) row tiles x output
//                         channels, pixels split over CTAs, cp.async-staged
//                         MN-major operands, FP32 atomics into dW.
#include "api_internal.h"
#include "tc.cuh"
#include "kpcn_filter.cuh"
#include "conv_plan.h"
#include <algorithm>
#include <cstring>
#include <utility>
#include <cudaTypedefs.h>
#include <type_traits>

namespace crt {
namespace {

constexpr int kBM = 128;           // k_conv3x3_wgrad: (tap, c) rows per tile
constexpr int kThreads = 128;      // k_conv3x3_wgrad
constexpr int kConvThreads = 352;  // k_conv3x3, k_conv3x3_wgrad_ring: TMA warp, 2 MMA warps, 8 epilogue warps
constexpr int kStages = 4;         // k_conv3x3_wgrad pipeline depth
constexpr int kWgradBK = 64;       // k_conv3x3_wgrad: pixels per K step

struct ConvArgs {
    const float *bias;          // [N] or null
    const __nv_bfloat16 *mask;  // [P][N] or null: out *= (mask > 0)
    __nv_bfloat16 *out;         // [P][N] or null
    float *out_f32;             // [P][N] or null
    int *err;
    int nimg, h, wd, C, N;
    int Ng, groups;             // output channels of one CTA and N / Ng
    int Ws, R, P, TS;           // block: strip width, rows, row pitch Ws + 2, positions between tile starts
    int KCs, nst, S;            // channels per stage, stages per block (C / KCs), stage buffers
    int flip, relu, resident, by_tile;
    ConvExtra x;
    int vec32, vec_f32;         // out and mask 32-byte aligned; out_f32 16-byte aligned
    uint32_t region_bytes;      // one layout chunk of a stage: (R + 2) P rows, rounded up to 1 KB
    uint32_t stage_bytes, wres_bytes;
    uint32_t slot_cols, slots;  // TMEM columns per accumulator, accumulators
};

__device__ __forceinline__ uint32_t tmem_cols(int n) {
    uint32_t c = 32;
    while ((int)c < n) c <<= 1;
    return c;
}

__device__ __forceinline__ void store32(void *p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

// The epilogue of 16 consecutive channels of one pixel (offset o of the
// output): bias and ReLU in FP32, then BF16 (times the mask) and / or FP32.
__device__ __forceinline__ void conv_store16(const ConvArgs &a, const float *v, const float *bias, size_t o,
                                             __nv_bfloat16 *o2) {
    float r[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        r[i] = v[i] + bias[i];
        if (a.relu) r[i] = fmaxf(r[i], 0.f);
    }
    if (a.out_f32) {
        float *dst = a.out_f32 + o;
        if (a.vec_f32) {
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                *reinterpret_cast<float4 *>(dst + i) = make_float4(r[i], r[i + 1], r[i + 2], r[i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) dst[i] = r[i];
        }
    }
    if (!a.out) return;
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(r[2 * i], r[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t *>(&b);
    }
    if (a.mask) {
        const uint4 m0 = __ldg(reinterpret_cast<const uint4 *>(a.mask + o));
        const uint4 m1 = __ldg(reinterpret_cast<const uint4 *>(a.mask + o) + 1);
        const uint32_t m[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&m[i]));
            if (!(f.x > 0.f)) w[i] &= 0xffff0000u;
            if (!(f.y > 0.f)) w[i] &= 0x0000ffffu;
        }
    }
    if (o2) {  // 32-byte aligned
        store32(o2, w);
        if (a.x.up2) {
            const size_t row = (size_t)2 * a.wd * a.x.out2_pitch;
            store32(o2 + a.x.out2_pitch, w);
            store32(o2 + row, w);
            store32(o2 + row + a.x.out2_pitch, w);
        }
    }
    __nv_bfloat16 *dst = a.out + o;
    if (a.vec32) {
        store32(dst, w);
    } else {
        *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        *(reinterpret_cast<uint4 *>(dst) + 1) = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

// Forward and data gradient with 128 pixels on the MMA's M side (one TMEM
// lane per pixel) and the output channels on its N side: an MMA then costs
// what its output channels cost and both halves of the array work from 16
// channels up (the transposed form, channels as M, ran half-empty arrays at
// 64 channels and a quarter at 32), and the epilogue reads whole pixels, so
// it needs no transposition. Measured against that form (us): 1920 x 1080
// 16 -> 32 200 -> 67, 32 -> 32 202 -> 78, 96 -> 32 310 -> 161; 960 x 540
// 64 -> 64 73 -> 49, 160 -> 64 179 -> 106; 480 x 270 96 -> 96 46 -> 30. The
// tensor core's operand reads (4 KB + 32 N B of shared memory per MMA, 40
// cycles at 32 channels, 48 at 64) take 58% (32 -> 32) to 83% (96 -> 32) of the
// time; the rest is the issue of MMAs and the waits around each tile.
//
// A CTA walks blocks of R rows of a strip of Ws columns. A block's input is
// one TMA box per layout chunk of kc channels, (R + 2) x (Ws + 2) pixels
// (zero-filled outside the image), which lands as consecutive pixel rows of
// RB = 2 kc bytes in the swizzled K-major layout with pitch P = Ws + 2
// pixels. In this flat order tap (dy, dx) of every pixel of the block is
// the row dy P + dx further on, so an A operand is any 128 consecutive
// rows: tile t starts at row t TS. With TS = P a tile is one image row
// (Ws = 128); with TS = 128 the tiles run on across the rows of the block
// (narrow images and ragged widths), and the two pitch columns per row are
// computed and dropped. (The swizzle is a function of the absolute
// shared-memory address, so shifted starts read the rows TMA wrote. The
// last tile may read past the block: its surplus rows are dropped too.)
// The channels of a block come in nst stages of KCs channels; with nst > 1
// all tiles of the block keep their accumulators until the last stage.
// Weights (B, [layout chunk][tap][n][kc channels], the same swizzled K-major
// rows, one TMA box per chunk) are loaded once per CTA when they fit next to
// the stages, else with every stage. (As 16 B rows in the no-swizzle layout
// the 72 KB of a 64 -> 64 layer took 17 us to load.) Layers whose
// weights do not fit are split into groups of output channels.
// Warp roles (no block-wide barrier inside the loop):
//   warp 0     one thread issues the TMA loads of a stage once the MMAs of
//              the stage S before it released the buffer.
//   warps 1-2  issue the MMAs of alternate blocks or tiles; commit to
//              tfull[slot] after a tile's last stage and to empty[stage].
//   warps 3-10 epilogue, two groups of four warps taking alternate tiles;
//              warp % 4 is the TMEM lane quarter (32 pixels). Bias / ReLU in
//              FP32, 32 B stores.
// Every wait is bounded and also ends when another role has given up.
//
// The order of the sums is fixed per layer shape (ConvOrder) and does not
// depend on the tiling: kKK = K steps per channel chunk of the order, kRows:
// tap rows outside the channel chunks, else the channel chunks outermost.
// kFilter: the epilogue applies the 5x5 filter (ConvExtra).
template <int kKK, bool kRows, bool kFilter = false>
__global__ void __launch_bounds__(kConvThreads, 1)
    k_conv3x3(const __grid_constant__ CUtensorMap map_in, const __grid_constant__ CUtensorMap map_w, ConvArgs a,
              int kcl) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t full[kMaxStages], empty[kMaxStages], tfull[kMaxSlots], tempty[kMaxSlots], wbar, mma_done[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ float s_bias[256];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int N = a.N, Ng = a.Ng, W = a.wd, H = a.h, S = a.S, P = a.P, kc = 1 << kcl, RB = 2 << kcl;
    const int grp = blockIdx.x % a.groups, ctas = gridDim.x / a.groups, ci = blockIdx.x / a.groups, n0 = grp * Ng;
    const int ntx = (W + a.Ws - 1) / a.Ws, nrb = (H + a.R - 1) / a.R, nblk = a.nimg * ntx * nrb;
    const int b_beg = (int)((int64_t)nblk * ci / ctas), b_end = (int)((int64_t)nblk * (ci + 1) / ctas);
    const uint32_t tap_bytes = (uint32_t)(Ng * RB), wch_bytes = 9 * tap_bytes;  // weights of a tap, of kc channels
    // 1 KB aligned: TMA swizzle atoms and the descriptors' address phase
    unsigned char *const base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char *const wres = base;
    unsigned char *const stages = base + a.wres_bytes;
    const uint32_t a_bytes = (uint32_t)(a.KCs >> kcl) * a.region_bytes;  // weights of a streamed stage follow
    const uint32_t ncols = tmem_cols((int)(a.slots * a.slot_cols));
    // Walks the CTA's blocks (strip by strip, rows downwards) without
    // divisions, which cost the MMA thread as much as a tile's MMAs.
    struct Block {
        int img, y0, x0, rows, w, tiles;
    };
    auto fill = [&](Block &k) {
        k.rows = min(a.R, H - k.y0);
        k.w = min(a.Ws, W - k.x0);
        k.tiles = a.TS == P ? k.rows : ((k.rows - 1) * P + k.w + 127) >> 7;
    };
    auto first_block = [&]() {
        Block k;
        const int r2 = b_beg / nrb;
        k.y0 = (b_beg - r2 * nrb) * a.R;
        k.img = r2 / ntx;
        k.x0 = (r2 - k.img * ntx) * a.Ws;
        fill(k);
        return k;
    };
    auto next_block = [&](Block &k) {
        k.y0 += a.R;
        if (k.y0 >= H) {
            k.y0 = 0;
            k.x0 += a.Ws;
            if (k.x0 >= W) {
                k.x0 = 0;
                ++k.img;
            }
        }
        fill(k);
    };
    volatile int *abort = &abort_flag;
    // How the two MMA warps share the work: alternate tiles, or alternate
    // blocks. A barrier's phases are told apart by parity only, so whoever
    // waits on one must see every phase of it: each accumulator belongs to one
    // MMA warp (by tiles: the warp of its parity; by blocks: half of them each)
    // and to one epilogue group (of its parity), and by blocks, S being even,
    // so does each stage buffer.
    const bool by_tile = a.by_tile;
    const uint32_t half_slots = a.slots >> 1;

    if (tid == 0) {
        for (int i = 0; i < S; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], by_tile ? 2 : 1);
        }
        for (int i = 0; i < (int)a.slots; ++i) {
            tc::mbar_init(&tfull[i], 1);
            tc::mbar_init(&tempty[i], 4);
        }
        tc::mbar_init(&wbar, 1);
        tc::mbar_init(&mma_done[0], 1);
        tc::mbar_init(&mma_done[1], 1);
        abort_flag = 0;
        tc::fence_mbar_init();
    }
    for (int i = tid; i < Ng; i += kConvThreads) s_bias[i] = a.bias ? a.bias[n0 + i] : 0.f;
    if (warp == 1) tc::tmem_alloc(&tmem_slot, ncols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer ----
            if (a.resident) {
                tc::mbar_arrive_expect_tx(&wbar, (uint32_t)(a.C / kc) * wch_bytes);
                for (int ch = 0; ch < a.C / kc; ++ch)
                    tc::tma_load_3d(wres + ch * wch_bytes, &map_w, ch * kc, n0, 0, &wbar);
            }
            const int nch = a.KCs >> kcl;
            const uint32_t tx = (uint32_t)nch * (uint32_t)((a.R + 2) * P * RB) +
                                (a.resident ? 0u : (uint32_t)nch * wch_bytes);
            int buf = 0, issued = -1;
            uint32_t par = 1;
            Block k = first_block();
            for (int b = b_beg; b < b_end && !*abort; ++b, next_block(k)) {
                bool ok = true;
                for (int st = 0; st < a.nst; ++st) {
                    // (a fresh barrier passes a wait for parity 1)
                    if (!tc::mbar_wait_or_abort(&empty[buf], par, abort)) {
                        ok = false;
                        break;
                    }
                    unsigned char *sa = stages + (size_t)buf * a.stage_bytes;
                    tc::mbar_arrive_expect_tx(&full[buf], tx);
                    for (int ch = 0; ch < nch; ++ch)
                        tc::tma_load_4d(sa + ch * a.region_bytes, &map_in, st * a.KCs + ch * kc, k.x0 - 1, k.y0 - 1,
                                        k.img, &full[buf]);
                    if (!a.resident)
                        for (int ch = 0; ch < nch; ++ch)
                            tc::tma_load_3d(sa + a_bytes + ch * wch_bytes, &map_w, st * a.KCs + ch * kc, n0, 0,
                                            &full[buf]);
                    issued = buf > issued ? buf : issued;
                    if (++buf == S) {
                        buf = 0;
                        par ^= 1;
                    }
                }
                if (!ok) break;
            }
            // no TMA write may land after the CTA has exited: wait for the
            // last phase issued on every stage (immediate when consumed).
            // par is the parity a buffer's next load would wait for on
            // empty: from buf on the last load's phase is par, before it the
            // one after.
            for (int st = 0; st <= issued; ++st) tc::mbar_wait(&full[st], st < buf ? par ^ 1 : par);
            if (a.resident) tc::mbar_wait(&wbar, 0);
        }
    } else if (warp <= 2) {
        // ---- MMA issuers: one lane of each issues, the control flow is the
        // whole warp's. Two warps, because the waits and commits around a
        // tile take a warp as long as a small tile's MMAs take the tensor
        // core. They take alternate blocks, which keeps them out of step, or
        // alternate tiles where a block has several stages. ----
        // Descriptor offsets (16 B units in the start-address field, which
        // never carries: shared addresses stay below 256 KB) of the 9 taps
        // (mirrored weight taps for the data gradient).
        const uint32_t leader = tc::elect_one() ? 1u : 0u, group = (uint32_t)warp - 1;
        const uint32_t idesc = tc::idesc_bf16(128, Ng, false, false);
        uint32_t aoff[9], boff[9];
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            aoff[t] = (uint32_t)(((t / 3) * P + t % 3) * RB) >> 4;
            boff[t] = ((a.flip ? 8 - t : t) * tap_bytes) >> 4;
        }
        const uint64_t adesc0 = tc::smem_desc_sw(tc::smem_addr(stages), RB);
        const uint64_t bdesc0 = tc::smem_desc_sw(tc::smem_addr(a.resident ? wres : stages + a_bytes), RB);
        const uint32_t stage16 = a.stage_bytes >> 4, region16 = a.region_bytes >> 4;
        const uint32_t wch16 = wch_bytes >> 4, ts16 = (uint32_t)(a.TS * RB) >> 4;
        constexpr int KCo = 16 * kKK;
        const int subs = a.KCs / KCo;
        auto wait = [&](uint64_t *bar, uint32_t parity) {
            return __all_sync(0xffffffffu, tc::mbar_ready(bar, parity)) ||
                   tc::mbar_wait_or_abort_warp(bar, parity, abort);
        };
        int buf = 0;  // stage buffer and the parity of its next phase
        uint32_t buf_par = 0;
        // this warp's accumulators [lo, hi), the next of them and the parity
        // of its release (a fresh barrier passes a wait for parity 1)
        const uint32_t lo = by_tile ? 0 : group * half_slots, hi = by_tile ? a.slots : lo + half_slots;
        uint32_t slot0 = lo, par0 = 1;
        const uint32_t tstep = by_tile ? 2 : 1;
        bool run = !a.resident || wait(&wbar, 0);
        Block k = first_block();
        for (int b = b_beg; b < b_end && run; ++b, next_block(k)) {
            const uint32_t tiles = (uint32_t)k.tiles;
            const bool mine = by_tile || ((uint32_t)(b - b_beg) & 1) == group;
            // by tiles: the tiles whose accumulator has this warp's parity
            const uint32_t first = by_tile ? (slot0 ^ group) & 1 : 0;
            for (int st = 0; st < a.nst && run && mine; ++st) {
                if (!wait(&full[buf], buf_par)) {
                    run = false;
                    break;
                }
                tc::fence_after_sync();
                uint64_t ad = adesc0 + buf * stage16 + first * ts16;
                const uint64_t bd_stage =
                    bdesc0 + (a.resident ? (uint32_t)(st * (a.KCs >> kcl)) * wch16 : buf * stage16);
                uint32_t slot = slot0 + first, par = par0;
                for (uint32_t t = first; t < tiles; t += tstep, ad += tstep * ts16, slot += tstep) {
                    if (slot >= hi) {
                        slot -= hi - lo;
                        par ^= 1;
                    }
                    if (st == 0) {
                        if (!wait(&tempty[slot], par)) {
                            run = false;
                            break;
                        }
                        tc::fence_after_sync();
                    }
                    const uint32_t d = tmem + slot * a.slot_cols;
                    if (kRows) {
                        // rows of taps, channel chunks, columns of taps
#pragma unroll
                        for (int r = 0; r < 3; ++r)
                            for (int ch = 0; ch < subs; ++ch) {
                                const uint64_t adc = ad + ch * region16;
                                const uint64_t bdc = bd_stage + (uint32_t)ch * wch16;
#pragma unroll
                                for (int c = 0; c < 3; ++c)
#pragma unroll
                                    for (int kk = 0; kk < kKK; ++kk)
                                        tc::mma_bf16_pred(leader, d, adc + aoff[3 * r + c] + kk * 2,
                                                          bdc + boff[3 * r + c] + kk * 2, idesc,
                                                          st > 0 || r > 0 || ch > 0 || c > 0 || kk > 0);
                            }
                    } else {
                        for (int ch = 0; ch < subs; ++ch) {
                            const int co = ch * KCo;
                            const uint32_t chunk = (uint32_t)co >> kcl, in_chunk = (uint32_t)(co & (kc - 1)) >> 3;
                            const uint64_t adc = ad + chunk * region16 + in_chunk;
                            const uint64_t bdc = bd_stage + chunk * wch16 + in_chunk;
#pragma unroll
                            for (int tp = 0; tp < 9; ++tp)
#pragma unroll
                                for (int kk = 0; kk < kKK; ++kk)
                                    tc::mma_bf16_pred(leader, d, adc + aoff[tp] + kk * 2,
                                                      bdc + boff[tp] + kk * 2, idesc,
                                                      st > 0 || ch > 0 || tp > 0 || kk > 0);
                        }
                    }
                    if (st == a.nst - 1) tc::mma_commit_pred(leader, tc::smem_addr(&tfull[slot]));
                }
                tc::mma_commit_pred(leader, tc::smem_addr(&empty[buf]));
                if (++buf == S) {
                    buf = 0;
                    buf_par ^= 1;
                }
            }
            if (!mine && ++buf == S) {  // (one stage per block)
                buf = 0;
                buf_par ^= 1;
            }
            if (mine)
                for (slot0 += tiles; slot0 >= hi; slot0 -= hi - lo) par0 ^= 1;
        }
        // every MMA issued has finished before TMEM is released
        tc::mma_commit_pred(leader, tc::smem_addr(&mma_done[group]));
        wait(&mma_done[group], 0);
    } else {
        // ---- epilogue: one thread per pixel of the tile ----
        const int q = warp & 3;
        const uint32_t group = (uint32_t)(warp - 3) >> 2;
        // next accumulator and its parity, of all blocks or (by blocks) of the
        // even and of the odd ones
        uint32_t next_slot[2] = {0, half_slots}, next_par[2] = {0, 0};
        bool run = true;
        Block k = first_block();
        for (int b = b_beg; b < b_end && run; ++b, next_block(k)) {
            const bool odd = !by_tile && ((b - b_beg) & 1);
            const uint32_t lo = odd ? half_slots : 0, hi = by_tile || odd ? a.slots : half_slots;
            uint32_t at = odd ? next_slot[1] : next_slot[0], at_par = odd ? next_par[1] : next_par[0];
            for (int t = 0; t < k.tiles; ++t) {
                const uint32_t slot = at, par = at_par;
                if (++at == hi) {
                    at = lo;
                    at_par ^= 1;
                }
                if ((slot & 1) != group) continue;
                if (!tc::mbar_wait_or_abort(&tfull[slot], par, abort)) {
                    run = false;
                    break;
                }
                __syncwarp();
                tc::fence_after_sync();
                const int pos = t * a.TS + q * 32 + lane;
                const int row = pos / P, col = pos - row * P;
                const bool valid = row < k.rows && col < k.w;
                const int y = k.y0 + row, x = k.x0 + col;
                const size_t o = (((size_t)k.img * H + y) * W + x) * N + n0;
                __nv_bfloat16 *o2 = nullptr;
                if (a.x.out2)
                    o2 = a.x.out2 + n0 +
                         (a.x.up2 ? ((size_t)k.img * 2 * H + 2 * y) * 2 * W + 2 * x : ((size_t)k.img * H + y) * W + x) *
                             a.x.out2_pitch;
                const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + slot * a.slot_cols;
                for (int c = 0; c < Ng; c += 32) {
                    float v[32];
                    __syncwarp();
                    if (c + 32 <= Ng) {
                        tc::tmem_ld32(taddr + c, v);
                    } else {
                        float h16[16];
                        tc::tmem_ld16(taddr + c, h16);
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = h16[i];
                    }
                    if (kFilter && valid) {  // one group of 32 channels, 25 of them logits
                        float wt[kTaps5];
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] += s_bias[i];
                        softmax25(v, wt);
                        const size_t img = (size_t)k.img * H * W;
                        a.x.filtered[img + (size_t)y * W + x] = filter25(wt, a.x.noisy + img, x, y, H, W);
                    } else if (valid) {
                        conv_store16(a, v, s_bias + c, o + c, o2 ? o2 + c : nullptr);
                        if (c + 32 <= Ng)
                            conv_store16(a, v + 16, s_bias + c + 16, o + c + 16, o2 ? o2 + c + 16 : nullptr);
                    }
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&tempty[slot]);  // this quarter's TMEM reads are done
            }
            next_slot[0] = odd ? next_slot[0] : at;
            next_par[0] = odd ? next_par[0] : at_par;
            next_slot[1] = odd ? at : next_slot[1];
            next_par[1] = odd ? at_par : next_par[1];
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0 && abort_flag) atomicOr(a.err, kErrWaitGaveUp);
    if (warp == 1) tc::tmem_dealloc(tmem, ncols);
}

// ---- weight gradient on the row ring ----
//
// dW[t][n][c] += sum_p in[p + off(t)][c] * g[p][n] as one GEMM per CTA with
// rows (tap, channel), columns n and K = the CTA's pixels, accumulated in
// TMEM over its whole contiguous range of row tiles (same order as the
// forward's ring mode: consecutive rows of one column strip).
// A = the input rows of the ring, read MN-major: a 128-row block is the
// channel chunk (KC channels per 2 KC-byte swizzled row) of 128 / KC
// dx-adjacent taps of one input row; consecutive taps are the same rows
// shifted by one pixel, i.e. MN groups one row apart (LBO = one row). Taps
// past the third and channels past C fill the block's spare rows; their
// results are not read. B = the output gradient tile (NP pixels x N
// channels, TMA-loaded, MN-major). Blocks of one CTA group: TMEM holds
// (blocks per group) x N columns; with more blocks than fit, the grid is
// split into groups that each accumulate a subset and read all inputs.
// Bound by the MMAs' issue and, for small batches, by the start-up and the
// atomics of the epilogue. One issuing lane per warp in a warp-uniform loop,
// two issuing warps and the rotated epilogue against one warp with an
// elect.sync per MMA (us): 960 x 540 64 x 64 86 -> 56, 1920 x 1080 32 x 32
// 214 -> 143, 8 x 64 x 64 160 x 64 47 -> 34, 8 x 128 x 128 32 x 32 27 -> 21.
struct WgradRingArgs {
    float *dw;  // [9][N][C], accumulated
    int *err;
    int nimg, h, wd, C, N;
    int NP, R;  // pixels per tile, ring rows
    int G, blocks_per_group, total_blocks;
    uint32_t region_bytes, row_bytes;     // input: one channel chunk of a ring row, one ring row
    uint32_t gregion_bytes, gtile_bytes;  // gradient: one channel group of a tile, one tile
};

template <int kKS, int kGS>  // input chunk KC = 16 kKS, gradient channel group 16 kGS
__global__ void __launch_bounds__(kConvThreads, 1)
    k_conv3x3_wgrad_ring(const __grid_constant__ CUtensorMap map_in, const __grid_constant__ CUtensorMap map_edge,
                         const __grid_constant__ CUtensorMap map_g, WgradRingArgs a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t full[kMaxStages], empty[kMaxStages], gfull[2], gempty[2], mma_done;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    constexpr int KC = 16 * kKS, RB = 2 * KC, GKC = 16 * kGS, RBG = 2 * GKC;
    constexpr int TPB = KC == 64 ? 2 : 3;  // valid taps (dx) per 128-row block
    constexpr int BPD = KC == 64 ? 2 : 1;  // blocks per (input row, channel chunk)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int C = a.C, N = a.N, W = a.wd, H = a.h, NP = a.NP, S = a.R;
    const int chunks = C / KC, ggroups = N / GKC;
    const int ntx = (W + NP - 1) / NP, ntiles = a.nimg * H * ntx;
    const int grp = blockIdx.x % a.G, ctas = gridDim.x / a.G, ci = blockIdx.x / a.G;
    const int b_beg = grp * a.blocks_per_group, b_end = min(a.total_blocks, b_beg + a.blocks_per_group);
    const int t_beg = (int)((int64_t)ntiles * ci / ctas);
    const int my_tiles = (int)((int64_t)ntiles * (ci + 1) / ctas) - t_beg;
    const uint32_t ncols = tmem_cols(a.blocks_per_group * N);
    unsigned char *const base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char *const ring = base;
    unsigned char *const gbuf = base + (size_t)S * a.row_bytes;
    auto tile_of = [&](int tl, int &b, int &y, int &x0) {
        const int t = t_beg + tl, r2 = t / H;
        y = t - r2 * H;
        x0 = (r2 % ntx) * NP;
        b = r2 / ntx;
    };
    volatile int *abort = &abort_flag;

    if (tid == 0) {
        for (int i = 0; i < S; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 2);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&gfull[i], 1);
            tc::mbar_init(&gempty[i], 2);
        }
        tc::mbar_init(&mma_done, 2);
        abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == 1) tc::tmem_alloc(&tmem_slot, ncols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer: ring rows (as the forward's ring mode) and
            // one gradient tile per row tile (two buffers) ----
            const uint32_t tx_row = (uint32_t)chunks * (NP + 2) * RB, tx_g = (uint32_t)ggroups * NP * RBG;
            int s = 0, tl = 0;
            for (; tl < my_tiles && !*abort; ++tl) {
                int b, y, x0;
                tile_of(tl, b, y, x0);
                const bool seg = tl == 0 || y == 0;
                bool ok = true;
                for (int yy = seg ? y - 1 : y + 1; yy <= y + 1; ++yy, ++s) {
                    const int st = s % S;
                    if (s >= S && !tc::mbar_wait_or_abort(&empty[st], ((s / S) - 1) & 1, abort)) {
                        ok = false;
                        break;
                    }
                    unsigned char *sa = ring + (size_t)st * a.row_bytes;
                    tc::mbar_arrive_expect_tx(&full[st], tx_row);
                    for (int ch = 0; ch < chunks; ++ch) {
                        tc::tma_load_4d(sa + ch * a.region_bytes, &map_in, ch * KC, x0 - 1, yy, b, &full[st]);
                        tc::tma_load_4d(sa + ch * a.region_bytes + NP * RB, &map_edge, ch * KC, x0 - 1 + NP, yy, b,
                                        &full[st]);
                    }
                }
                if (!ok) break;
                const int gs = tl & 1;
                if (tl >= 2 && !tc::mbar_wait_or_abort(&gempty[gs], ((tl >> 1) - 1) & 1, abort)) break;
                unsigned char *gb = gbuf + (size_t)gs * a.gtile_bytes;
                tc::mbar_arrive_expect_tx(&gfull[gs], tx_g);
                for (int gg = 0; gg < ggroups; ++gg)
                    tc::tma_load_4d(gb + gg * a.gregion_bytes, &map_g, gg * GKC, x0, y, b, &gfull[gs]);
                // (a break above leaves this tile's gradient unissued: tl is
                // then not counted below)
            }
            // no TMA write may land after the CTA has exited
            for (int st = 0; st < S && st < s; ++st) {
                const int last = s - 1 - ((s - 1 - st) % S);
                tc::mbar_wait(&full[st], (last / S) & 1);
            }
            for (int t2 = tl > 2 ? tl - 2 : 0; t2 < tl; ++t2) tc::mbar_wait(&gfull[t2 & 1], (t2 >> 1) & 1);
        }
    } else if (warp <= 2) {
        // ---- MMA issuers: one lane of each issues, the control flow is the
        // whole warp's; the two warps take alternate blocks ----
        const uint32_t leader = tc::elect_one() ? 1u : 0u;
        const int group = warp - 1;
        const uint32_t idesc = tc::idesc_bf16(128, N, true, true);
        const uint32_t ring_addr = tc::smem_addr(ring), gbuf_addr = tc::smem_addr(gbuf);
        const int ksteps = NP / 16;
        int s = 0, top = 0;
        bool run = true;
        for (int tl = 0; tl < my_tiles && run; ++tl) {
            int b, y, x0;
            tile_of(tl, b, y, x0);
            if (tl == 0 || y == 0) {
                top = s;
                s += 3;
            } else {
                top += 1;
                s += 1;
            }
            const int gs = tl & 1;
            if (!tc::mbar_wait_or_abort_warp(&gfull[gs], (tl >> 1) & 1, abort)) break;
            tc::fence_after_sync();
            const uint64_t bd0 = tc::smem_desc_sw(gbuf_addr + gs * a.gtile_bytes, RBG, a.gregion_bytes);
            for (int ri = 0; ri < 3 && run; ++ri) {
                const int ld = top + ri, st = ld % S;
                if (!tc::mbar_wait_or_abort_warp(&full[st], (ld / S) & 1, abort)) {
                    run = false;
                    break;
                }
                tc::fence_after_sync();
                for (int ch = 0; ch < chunks; ++ch)
#pragma unroll
                    for (int bb = 0; bb < BPD; ++bb) {
                        const int blk = (ri * chunks + ch) * BPD + bb;
                        if (blk < b_beg || blk >= b_end || (blk & 1) != group) continue;
                        const uint32_t d = tmem + (uint32_t)(blk - b_beg) * N;
                        const uint64_t ad0 = tc::smem_desc_sw(
                            ring_addr + st * a.row_bytes + ch * a.region_bytes + bb * TPB * RB, RB, RB);
                        for (int kk = 0; kk < ksteps; ++kk)
                            tc::mma_bf16_pred(leader, d, ad0 + ((kk * 16 * RB) >> 4), bd0 + ((kk * 16 * RBG) >> 4), idesc,
                                              tl > 0 || kk > 0);
                    }
            }
            if (!run) break;
            const bool strip_ends = tl + 1 == my_tiles || y + 1 == H;
            for (int r = 0; r < (strip_ends ? 3 : 1); ++r) tc::mma_commit_pred(leader, tc::smem_addr(&empty[(top + r) % S]));
            tc::mma_commit_pred(leader, tc::smem_addr(&gempty[gs]));
        }
        tc::mma_commit_pred(leader, tc::smem_addr(&mma_done));
        tc::mbar_wait_or_abort_warp(&mma_done, 0, abort);
    } else {
        // ---- epilogue: add the accumulators into dW ----
        const int q = warp & 3, half = (warp - 3) >> 2, r = q * 32 + lane;
        const bool ok = tc::mbar_wait_or_abort(&mma_done, 0, abort);
        tc::fence_after_sync();
        // All CTAs add into the same 9 N C sums at about the same time: each
        // starts at columns of its own.
        const int rot = (ci * 16) % N;
        if (ok && my_tiles > 0 && !*abort)
            for (int blk = b_beg + half; blk < b_end; blk += 2) {
                const int bb = blk % BPD, rc = blk / BPD, ch = rc % chunks, ri = rc / chunks;
                const int gtap = bb * TPB + r / KC, c = ch * KC + r % KC;
                const bool valid = r / KC < TPB && gtap < 3;
                const int t = ri * 3 + gtap;
                const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(blk - b_beg) * N;
                for (int nr = 0; nr < N; nr += 16) {
                    const int n0 = nr + rot < N ? nr + rot : nr + rot - N;
                    float v[16];
                    __syncwarp();
                    tc::tmem_ld16(taddr + n0, v);
                    if (valid)
#pragma unroll
                        for (int i = 0; i < 16; ++i) atomicAdd(a.dw + ((size_t)t * N + n0 + i) * C + c, v[i]);
                }
            }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0 && abort_flag) atomicOr(a.err, kErrWaitGaveUp);
    if (warp == 1) tc::tmem_dealloc(tmem, ncols);
}

struct WgradArgs {
    const __nv_bfloat16 *in;   // [P][C] layer input
    const __nv_bfloat16 *g;    // [P][N] gradient of the layer's pre-activation output
    float *dw;                 // [9][N][C], accumulated
    int *err;
    int nimg, h, wd, C, N;
    int pix_per_cta;           // multiple of kWgradBK
};

// dW[t][n][c] += sum_p in[p + off(t), c] * g[p, n] over this CTA's pixels.
// Tile rows m = t * C + c (blockIdx.y selects 128 of them), columns n.
__global__ void __launch_bounds__(kThreads) k_conv3x3_wgrad(WgradArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t bars[kStages + 1];
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int C = a.C, N = a.N;
    const int P = a.nimg * a.h * a.wd, HW = a.h * a.wd;
    const int rows = 9 * C, m0 = blockIdx.y * kBM;
    const int k0 = blockIdx.x * a.pix_per_cta, k1 = min(P, k0 + a.pix_per_cta);
    const int steps = (k1 - k0 + kWgradBK - 1) / kWgradBK;
    const uint32_t a_bytes = kBM * kWgradBK * 2, b_bytes = (uint32_t)N * kWgradBK * 2;
    const uint32_t stage_bytes = a_bytes + b_bytes;
    const uint32_t sbo = 128, lbo_a = (kBM / 8) * 128, lbo_b = (uint32_t)(N / 8) * 128;
    const uint32_t idesc = tc::idesc_bf16(kBM, N, true, true);
    const uint32_t ncols = tmem_cols(N);
    if (steps <= 0) return;

    if (tid == 0) {
        for (int s = 0; s <= kStages; ++s) tc::mbar_init(&bars[s], 1);
        tc::fence_mbar_init();
    }
    if (warp == 0) tc::tmem_alloc(&tmem_slot, ncols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    bool failed = false;

    for (int s = 0; s < steps + kStages - 1; ++s) {
        bool ok = true;
        if (s < steps) {
            const uint32_t st = s % kStages;
            if (s >= kStages) ok = tc::mbar_wait(&bars[st], ((s / kStages) - 1) & 1);
            unsigned char *sa = smem_raw + st * stage_bytes, *sb = sa + a_bytes;
            const int kb = k0 + s * kWgradBK;
            // A: 16 row groups x 64 pixels, one 16 B vector (8 channels of one tap) each
            for (int v = tid; v < (kBM / 8) * kWgradBK; v += kThreads) {
                const int k = v % kWgradBK, mg = v / kWgradBK;
                const int m = m0 + mg * 8, p = kb + k;
                bool valid = m < rows && p < k1;
                const __nv_bfloat16 *src = a.in;
                if (valid) {
                    const int tap = m / C, c0 = m - tap * C;
                    const int b = p / HW, r = p - b * HW, y = r / a.wd, x = r - y * a.wd;
                    const int sy = y + tap / 3 - 1, sx = x + tap % 3 - 1;
                    valid = sy >= 0 && sy < a.h && sx >= 0 && sx < a.wd;
                    if (valid) src = a.in + (size_t)(b * HW + sy * a.wd + sx) * C + c0;
                }
                tc::cp_async16(sa + mg * sbo + (k >> 3) * lbo_a + (k & 7) * 16, src, valid ? 16u : 0u);
            }
            // B: N/8 column groups x 64 pixels
            for (int v = tid; v < (N / 8) * kWgradBK; v += kThreads) {
                const int k = v % kWgradBK, ng = v / kWgradBK;
                const int p = kb + k;
                const bool valid = p < k1;
                const __nv_bfloat16 *src = valid ? a.g + (size_t)p * N + ng * 8 : a.g;
                tc::cp_async16(sb + ng * sbo + (k >> 3) * lbo_b + (k & 7) * 16, src, valid ? 16u : 0u);
            }
        }
        tc::cp_async_commit();
        const int c = s - (kStages - 1);
        if (c >= 0) {
            tc::cp_async_wait<kStages - 1>();
            tc::fence_proxy_async();
            if (__syncthreads_or(!ok)) {
                failed = true;
                break;
            }
            if (tid == 0) {
                const uint32_t st = c % kStages;
                const uint32_t sa = tc::smem_addr(smem_raw + st * stage_bytes), sb = sa + a_bytes;
                tc::fence_after_sync();
                for (int j = 0; j < kWgradBK / 16; ++j)
                    tc::mma_bf16(tmem, tc::smem_desc(sa + 2 * j * lbo_a, lbo_a, sbo),
                                 tc::smem_desc(sb + 2 * j * lbo_b, lbo_b, sbo), idesc, c > 0 || j > 0);
                tc::mma_commit(tc::smem_addr(&bars[st]));
            }
        } else if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
    }
    if (!failed) {
        if (tid == 0) tc::mma_commit(tc::smem_addr(&bars[kStages]));
        const bool ok = tc::mbar_wait(&bars[kStages], 0);
        if (__syncthreads_or(!ok)) {
            failed = true;
        } else {
            tc::fence_after_sync();
            const int m = m0 + tid;
            const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
            for (int n0 = 0; n0 < N; n0 += 16) {
                float v[16];
                tc::tmem_ld16(lane_base + n0, v);
                if (m < rows) {
                    const int tap = m / C, c = m - tap * C;
                    float *dst = a.dw + ((size_t)tap * N + n0) * C + c;
                    for (int i = 0; i < 16; ++i) atomicAdd(dst + (size_t)i * C, v[i]);
                }
            }
        }
    }
    if (failed && tid == 0) atomicOr(a.err, kErrWaitGaveUp);
    tc::cp_async_wait_all();
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

int g_sms = 0;

int sm_count() {
    if (!g_sms) {
        int dev;
        CRT_CUDA(cudaGetDevice(&dev));
        CRT_CUDA(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev));
    }
    return g_sms;
}

int host_tmem_cols(int n) {
    int c = 32;
    while (c < n) c <<= 1;
    return c;
}

// cuTensorMapEncodeTiled from the driver, found once through the runtime
// (the library links no driver library).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        CRT_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q));
        CRT_CHECK(f && q == cudaDriverEntryPointSuccess, CRT_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
        fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    }
    return fn;
}

void encode_map(CUtensorMap *m, const void *ptr, cuuint32_t rank, const cuuint64_t *dims,
                const cuuint64_t *strides_bytes, const cuuint32_t *box, CUtensorMapSwizzle swz) {
    const cuuint32_t ones[5] = {1, 1, 1, 1, 1};
    const CUresult r = tensor_map_encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(ptr), dims,
                                            strides_bytes, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CRT_CHECK(r == CUDA_SUCCESS, CRT_ERR_CUDA, "conv3x3: tensor map encoding failed");
}

}  // namespace

void conv3x3_check(int C, int N) {
    CRT_CHECK(C > 0 && C % 16 == 0 && C <= 512, CRT_ERR_INVALID, "conv3x3: input channels must be a multiple of 16");
    CRT_CHECK(N >= 16 && N % 16 == 0 && N <= 256, CRT_ERR_INVALID,
              "conv3x3: output channels must be a multiple of 16 in [16, 256]");
}

// out = conv3x3(in) (+ bias, ReLU) or the data gradient (flip = 1, weights
// transposed per tap, optional ReLU mask of the layer below).
void conv3x3_launch(const __nv_bfloat16 *in, const __nv_bfloat16 *wgt, const float *bias, const __nv_bfloat16 *mask,
                    __nv_bfloat16 *out, float *out_f32, int *err, int nimg, int h, int w, int C, int N, bool flip,
                    bool relu, cudaStream_t s, const ConvExtra &x) {
    conv3x3_check(C, N);
    const int64_t P = (int64_t)nimg * h * w;
    CRT_CHECK(nimg > 0 && h > 0 && w > 0 && P < (1LL << 31), CRT_ERR_INVALID, "conv3x3: bad image size");
    CRT_CHECK((reinterpret_cast<uintptr_t>(in) & 15) == 0 && (reinterpret_cast<uintptr_t>(wgt) & 15) == 0,
              CRT_ERR_INVALID, "conv3x3: input and weights must be 16-byte aligned");
    CRT_CHECK((!out || (reinterpret_cast<uintptr_t>(out) & 15) == 0) &&
                  (!out_f32 || (reinterpret_cast<uintptr_t>(out_f32) & 3) == 0) &&
                  (!mask || (reinterpret_cast<uintptr_t>(mask) & 15) == 0),
              CRT_ERR_INVALID, "conv3x3: output and mask must be 16-byte aligned");
    thread_local ConvPlans plans;
    const auto [ord, pl] = plans.get(nimg, h, w, C, N, x.filtered != nullptr, sm_count());
    ConvArgs a;
    a.bias = bias;
    a.mask = mask;
    a.out = out;
    a.out_f32 = out_f32;
    a.err = err;
    a.nimg = nimg;
    a.h = h;
    a.wd = w;
    a.C = C;
    a.N = N;
    a.Ng = pl.Ng;
    a.groups = pl.groups;
    a.Ws = pl.Ws;
    a.R = pl.R;
    a.P = pl.Ws + 2;
    a.TS = pl.TS;
    a.KCs = pl.KCs;
    a.nst = C / pl.KCs;
    // (by blocks each warp needs two buffers of its own to load ahead)
    a.by_tile = a.nst > 1 || pl.S < 4;
    a.S = a.by_tile ? pl.S : 4;
    a.flip = flip ? 1 : 0;
    a.relu = relu ? 1 : 0;
    a.resident = pl.resident;
    a.x = x;
    CRT_CHECK(!x.filtered || (C == 32 && N == 32 && ord.KCo == 32 && pl.groups == 1 && !relu && !flip),
              CRT_ERR_INVALID, "conv3x3: the filter follows a 32 -> 32 layer");
    CRT_CHECK(!x.out2 || ((reinterpret_cast<uintptr_t>(x.out2) | (uintptr_t)x.out2_pitch * 2) & 31) == 0,
              CRT_ERR_INVALID, "conv3x3: the second output must be 32-byte aligned");
    a.vec32 = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
    a.vec_f32 = (reinterpret_cast<uintptr_t>(out_f32) & 15) == 0;
    const int RB = 2 * pl.kc;
    a.region_bytes = (uint32_t)round1k((size_t)(a.R + 2) * a.P * RB);
    a.stage_bytes = (uint32_t)((a.KCs / pl.kc) * a.region_bytes +
                               (a.resident ? 0 : round1k((size_t)18 * a.Ng * a.KCs)));
    a.wres_bytes = a.resident ? (uint32_t)round1k((size_t)18 * a.Ng * C) : 0u;
    a.slot_cols = 32;
    while ((int)a.slot_cols < a.Ng) a.slot_cols <<= 1;
    a.slots = std::min<uint32_t>(kMaxSlots, 512 / a.slot_cols);
    const int tiles = a.TS == a.P ? a.R : ((a.R - 1) * a.P + a.Ws + 127) / 128;
    const size_t smem =
        1024 + a.wres_bytes + (size_t)a.S * a.stage_bytes + conv_over_rows(tiles, a.TS, a.R, a.P) * RB;

    // input [nimg][h][w][C] as 4D (C, w, h, nimg); weights [9][N][C] as 3D (C, N, 9)
    CUtensorMap map_in, map_w;
    const CUtensorMapSwizzle swz = RB == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                   : RB == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                              : CU_TENSOR_MAP_SWIZZLE_32B;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)nimg};
    const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)w * C * 2, (cuuint64_t)h * w * C * 2};
    const cuuint32_t box[4] = {(cuuint32_t)pl.kc, (cuuint32_t)a.P, (cuuint32_t)(a.R + 2), 1};
    encode_map(&map_in, in, 4, dims, strides, box, swz);
    const cuuint64_t wdims[3] = {(cuuint64_t)C, (cuuint64_t)N, 9};
    const cuuint64_t wstrides[2] = {(cuuint64_t)C * 2, (cuuint64_t)N * C * 2};
    const cuuint32_t wbox[3] = {(cuuint32_t)pl.kc, (cuuint32_t)a.Ng, 9};
    encode_map(&map_w, wgt, 3, wdims, wstrides, wbox, swz);

    using Kfn = void (*)(CUtensorMap, CUtensorMap, ConvArgs, int);
    const Kfn kfns[2][3] = {{k_conv3x3<1, false>, k_conv3x3<2, false>, k_conv3x3<4, false>},
                            {k_conv3x3<1, true>, k_conv3x3<2, true>, k_conv3x3<4, true>}};
    const Kfn kfn = x.filtered ? k_conv3x3<2, false, true>
                               : kfns[ord.rows_outer ? 1 : 0][ord.KCo == 16 ? 0 : ord.KCo == 32 ? 1 : 2];
    CRT_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kfn<<<pl.grid, kConvThreads, smem, s>>>(map_in, map_w, a, pl.kc == 64 ? 6 : pl.kc == 32 ? 5 : 4);
    CRT_CUDA(cudaGetLastError());
}

// dw[9][N][C] += weight gradient of a 3x3 conv with input `in` [P][C] and
// pre-activation output gradient `g` [P][N].
namespace {
// Weight gradient on the row ring when the ring and two gradient tiles fit
// in shared memory; returns false (nothing launched) otherwise.
bool wgrad_ring_launch(const __nv_bfloat16 *in, const __nv_bfloat16 *g, float *dw, int *err, int nimg, int h, int w,
                       int C, int N, cudaStream_t s) {
    if ((reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(g) & 15)) return false;
    const int KC = C % 64 == 0 ? 64 : C % 32 == 0 ? 32 : 16, GKC = N % 64 == 0 ? 64 : N % 32 == 0 ? 32 : 16;
    const int RB = 2 * KC, RBG = 2 * GKC;
    WgradRingArgs a;
    a.dw = dw;
    a.err = err;
    a.nimg = nimg;
    a.h = h;
    a.wd = w;
    a.C = C;
    a.N = N;
    a.total_blocks = 3 * (C / KC) * (KC == 64 ? 2 : 1);
    a.blocks_per_group = std::min(a.total_blocks, 512 / N);
    a.G = (a.total_blocks + a.blocks_per_group - 1) / a.blocks_per_group;
    const size_t kCap = 220 * 1024 - 1024;
    a.NP = 0;
    for (int np : {256, 128}) {
        if (a.NP || (np == 256 && w <= 128)) continue;
        const size_t region = round1k((size_t)(np + 2) * RB), row = (size_t)(C / KC) * region;
        const size_t gregion = round1k((size_t)np * RBG), gtile = (size_t)(N / GKC) * gregion;
        for (int ns : {5, 4})
            if (!a.NP && ns * row + 2 * gtile <= kCap) {
                a.NP = np;
                a.R = ns;
                a.region_bytes = (uint32_t)region;
                a.row_bytes = (uint32_t)row;
                a.gregion_bytes = (uint32_t)gregion;
                a.gtile_bytes = (uint32_t)gtile;
            }
    }
    if (!a.NP) return false;
    const size_t smem = 1024 + (size_t)a.R * a.row_bytes + 2 * (size_t)a.gtile_bytes;
    CUtensorMap map_in, map_edge, map_g;
    auto swz = [](int rb) {
        return rb == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : rb == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    };
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)nimg};
    const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)w * C * 2, (cuuint64_t)h * w * C * 2};
    const cuuint32_t box[4] = {(cuuint32_t)KC, (cuuint32_t)a.NP, 1, 1}, box_edge[4] = {(cuuint32_t)KC, 2, 1, 1};
    encode_map(&map_in, in, 4, dims, strides, box, swz(RB));
    encode_map(&map_edge, in, 4, dims, strides, box_edge, swz(RB));
    const cuuint64_t gdims[4] = {(cuuint64_t)N, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)nimg};
    const cuuint64_t gstrides[3] = {(cuuint64_t)N * 2, (cuuint64_t)w * N * 2, (cuuint64_t)h * w * N * 2};
    const cuuint32_t gbox[4] = {(cuuint32_t)GKC, (cuuint32_t)a.NP, 1, 1};
    encode_map(&map_g, g, 4, gdims, gstrides, gbox, swz(RBG));
    using Kfn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, WgradRingArgs);
    const Kfn kfns[3][3] = {{k_conv3x3_wgrad_ring<1, 1>, k_conv3x3_wgrad_ring<1, 2>, k_conv3x3_wgrad_ring<1, 4>},
                            {k_conv3x3_wgrad_ring<2, 1>, k_conv3x3_wgrad_ring<2, 2>, k_conv3x3_wgrad_ring<2, 4>},
                            {k_conv3x3_wgrad_ring<4, 1>, k_conv3x3_wgrad_ring<4, 2>, k_conv3x3_wgrad_ring<4, 4>}};
    const Kfn kfn = kfns[KC == 16 ? 0 : KC == 32 ? 1 : 2][GKC == 16 ? 0 : GKC == 32 ? 1 : 2];
    CRT_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t tiles = (int64_t)nimg * h * ((w + a.NP - 1) / a.NP);
    const int ctas = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, sm_count() / a.G > 0 ? sm_count() / a.G : 1));
    kfn<<<ctas * a.G, kConvThreads, smem, s>>>(map_in, map_edge, map_g, a);
    CRT_CUDA(cudaGetLastError());
    return true;
}
}  // namespace

void conv3x3_wgrad_launch(const __nv_bfloat16 *in, const __nv_bfloat16 *g, float *dw, int *err, int nimg, int h, int w,
                          int C, int N, cudaStream_t s) {
    conv3x3_check(C, N);
    const int64_t P = (int64_t)nimg * h * w;
    CRT_CHECK(P > 0 && P < (1LL << 31) - kWgradBK, CRT_ERR_INVALID, "conv3x3_wgrad: bad image size");
    if (wgrad_ring_launch(in, g, dw, err, nimg, h, w, C, N, s)) return;
    WgradArgs a;
    a.in = in;
    a.g = g;
    a.dw = dw;
    a.err = err;
    a.nimg = nimg;
    a.h = h;
    a.wd = w;
    a.C = C;
    a.N = N;
    const int mtiles = (9 * C + kBM - 1) / kBM;
    const size_t smem = (size_t)kStages * (kBM * kWgradBK * 2 + (size_t)N * kWgradBK * 2);
    CRT_CHECK(smem <= 200 * 1024, CRT_ERR_INVALID, "conv3x3_wgrad: tile does not fit shared memory");
    CRT_CUDA(cudaFuncSetAttribute(k_conv3x3_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    CRT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_conv3x3_wgrad, kThreads, smem));
    per_sm = std::max(1, std::min(per_sm, 512 / host_tmem_cols(N)));
    // enough pixel splits for about two waves, at least 8 K steps per CTA
    const int64_t want = std::max<int64_t>(1, 2LL * sm_count() * per_sm / mtiles);
    int64_t ppc = (P + want - 1) / want;
    ppc = std::max<int64_t>(ppc, 8 * kWgradBK);
    ppc = (ppc + kWgradBK - 1) / kWgradBK * kWgradBK;
    a.pix_per_cta = (int)ppc;
    dim3 grid((unsigned)((P + ppc - 1) / ppc), (unsigned)mtiles);
    k_conv3x3_wgrad<<<grid, kThreads, smem, s>>>(a);
    CRT_CUDA(cudaGetLastError());
}

}  // namespace crt

using namespace crt;

extern "C" crt_status crt_check_device_errors(crt_ctx *ctx) {
    return guard([&] {
        CRT_CHECK(ctx, CRT_ERR_INVALID, "crt_check_device_errors: null context");
        CRT_CUDA(cudaSetDevice(ctx->device));
        int e = 0;
        CRT_CUDA(cudaDeviceSynchronize());
        CRT_CUDA(cudaMemcpy(&e, ctx->d_err, sizeof(int), cudaMemcpyDeviceToHost));
        if (e) {
            CRT_CUDA(cudaMemset(ctx->d_err, 0, sizeof(int)));
            if (e & kErrTraversalBounds)
                throw Error(CRT_ERR_CUDA, "a BVH traversal met an out-of-range node, leaf or stack depth and stopped");
            throw Error(CRT_ERR_TIMEOUT, "a tensor-core kernel gave up waiting on an mbarrier");
        }
    });
}

extern "C" crt_status crt_conv3x3_forward(crt_ctx *ctx, const void *d_in, int32_t n, int32_t h, int32_t w,
                                          int32_t cin, const void *d_weights, const float *d_bias, int32_t cout,
                                          int32_t relu, void *d_out_bf16, float *d_out_f32, void *stream) {
    return guard([&] {
        CRT_CHECK(ctx && d_in && d_weights && (d_out_bf16 || d_out_f32), CRT_ERR_INVALID,
                  "crt_conv3x3_forward: null argument");
        CRT_CUDA(cudaSetDevice(ctx->device));
        cudaStream_t s = stream ? (cudaStream_t)stream : ctx->stream;
        conv3x3_launch((const __nv_bfloat16 *)d_in, (const __nv_bfloat16 *)d_weights, d_bias, nullptr,
                       (__nv_bfloat16 *)d_out_bf16, d_out_f32, ctx->d_err, n, h, w, cin, cout, false, relu != 0, s);
    });
}

extern "C" crt_status crt_conv3x3_backward_data(crt_ctx *ctx, const void *d_grad_out, int32_t n, int32_t h, int32_t w,
                                                int32_t cout, const void *d_weights_t, int32_t cin, const void *d_mask,
                                                void *d_grad_in, void *stream) {
    return guard([&] {
        CRT_CHECK(ctx && d_grad_out && d_weights_t && d_grad_in, CRT_ERR_INVALID,
                  "crt_conv3x3_backward_data: null argument");
        CRT_CUDA(cudaSetDevice(ctx->device));
        cudaStream_t s = stream ? (cudaStream_t)stream : ctx->stream;
        conv3x3_launch((const __nv_bfloat16 *)d_grad_out, (const __nv_bfloat16 *)d_weights_t, nullptr,
                       (const __nv_bfloat16 *)d_mask, (__nv_bfloat16 *)d_grad_in, nullptr, ctx->d_err, n, h, w, cout,
                       cin, true, false, s);
    });
}

extern "C" crt_status crt_conv3x3_backward_weights(crt_ctx *ctx, const void *d_in, const void *d_grad_out, int32_t n,
                                                   int32_t h, int32_t w, int32_t cin, int32_t cout, float *d_grad_w,
                                                   void *stream) {
    return guard([&] {
        CRT_CHECK(ctx && d_in && d_grad_out && d_grad_w, CRT_ERR_INVALID,
                  "crt_conv3x3_backward_weights: null argument");
        CRT_CUDA(cudaSetDevice(ctx->device));
        cudaStream_t s = stream ? (cudaStream_t)stream : ctx->stream;
        conv3x3_wgrad_launch((const __nv_bfloat16 *)d_in, (const __nv_bfloat16 *)d_grad_out, d_grad_w, ctx->d_err, n,
                             h, w, cin, cout, s);
    });
}
