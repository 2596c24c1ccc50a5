// Host side of k_conv3x3 (conv.cu): the order of a layer's sums and its tiling,
// functions of the shape alone, and the plans a thread keeps.
#pragma once
#include "common.cuh"
#include <algorithm>
#include <array>
#include <cstdint>
#include <unordered_map>
#include <utility>

namespace crt {

constexpr int kMaxStages = 5;  // stage buffers of the convolution kernels
constexpr int kMaxSlots = 8;   // TMEM accumulators of k_conv3x3

inline size_t round1k(size_t v) { return (v + 1023) & ~(size_t)1023; }

// The order in which a layer sums its products, a function of its shape
// only: the MMAs of one output run over channel chunks of KCo channels (all
// nine taps of a chunk, then the next chunk) or, with rows_outer, over the
// three tap rows with the chunks inside. BF16 activations round the sums,
// so a different order would flip roundings layer by layer; the thresholds
// below keep every shape's order, and with it every output bit, as it was
// under the tiling they came from (channels as M, 256 pixels as N).
struct ConvOrder {
    int KCo;
    bool rows_outer;
};

inline ConvOrder conv_order(int C, int N, int w) {
    const int np = (N > 128 || w <= 128) ? 128 : 256;
    const size_t cap = 220 * 1024 - 1024 - 2048 - 8192, wbytes = round1k((size_t)9 * N * C * 2);
    auto region = [&](int rb) { return round1k((size_t)(np + 2) * rb); };
    const int kc = C % 64 == 0 ? 64 : C % 32 == 0 ? 32 : 16;
    if (wbytes + 4 * (C / kc) * region(2 * kc) <= cap) return {kc, C > kc};
    for (int c : {64, 32, 16})
        if (C % c == 0 && wbytes + 9 * region(2 * c) <= cap) return {c, false};
    for (int ns : {4, 3, 2})
        for (int c : {64, 32, 16})
            if ((ns >= 3 || c == 16) && C % c == 0 && ns * (3 * region(2 * c) + round1k((size_t)c * 18 * N)) <= cap)
                return {c, false};
    throw Error(CRT_ERR_INVALID, "conv3x3: tile does not fit shared memory");
}

// The tiling of a layer, by a cost model in SM cycles: an MMA of 128 x Ng
// x 16 reads 4 KB + 32 Ng B of shared memory at 128 B per cycle or
// multiplies at 4096 MAC per cycle, whichever is longer; a CTA's loads run
// at about 32 B per cycle; an epilogue group needs about 400 + 10 Ng cycles
// per tile and there are two; an MMA warp needs about 58 cycles per MMA and
// 250-300 per tile, and there are two. A block takes the longest of these,
// and the layer the CTA with the most blocks.
struct ConvPlan {
    int Ng, groups, Ws, R, TS, KCs, kc, S, resident, grid;
    double cost;
};

// Rows of shared memory that a block's last tile reads past its stage
// (their results are dropped).
inline size_t conv_over_rows(int tiles, int TS, int R, int P) { return (size_t)std::max(0, (tiles - 1) * TS + 130 - R * P); }

// one_group: all output channels in one CTA (the filter needs a pixel's 32).
inline ConvPlan conv_plan(const ConvOrder &ord, int nimg, int h, int w, int C, int N, int sms, bool one_group) {
    ConvPlan best{};
    best.cost = 1e30;
    const size_t cap = 227 * 1024 - 1024 - 4096;  // minus base alignment and static shared memory
    for (int groups = 1; groups <= (one_group ? 1 : N / 16); ++groups) {
        if (N % (16 * groups)) continue;
        const int Ng = N / groups;
        const size_t wall = (size_t)18 * Ng * C;
        int stride = 32;
        while (stride < Ng) stride <<= 1;
        const int slots = std::min(kMaxSlots, 512 / stride);
        const double mma = 9.0 * (C / 16) * std::max(0.5 * Ng, 34.0 + 0.25 * Ng);
        const double epi = 0.5 * (400.0 + 10.0 * Ng);
        // at least: the tiles of a CTA, each at its MMAs' issue (by one warp
        // where that is the longer, else by two) or operand reads
        const int64_t all = ((int64_t)nimg * h * w + 127) / 128, ctas_most = std::max(1, sms / groups);
        const double tile = 9.0 * (C / 16) * std::max(29.0, std::min(58.0, std::max(0.5 * Ng, 34.0 + 0.25 * Ng)));
        if ((double)((all + ctas_most - 1) / ctas_most) * tile + 2 * epi >= best.cost) continue;
        for (int part : {0, 64, 32, 16}) {  // 0: all channels in one stage
            const int KCs = part ? part : C;
            if ((part && part >= C) || C % KCs || KCs % ord.KCo || (ord.rows_outer && KCs != C)) continue;
            const int kc = KCs % 64 == 0 ? 64 : KCs % 32 == 0 ? 32 : 16;
            const int nst = C / KCs;
            for (int resident = 1; resident >= 0; --resident) {
                if (resident && wall > cap) continue;
                if (!resident && KCs > 64) continue;
                // (strips of at most 126 pixels are the same tiling twice)
                for (int mode = 0; mode < (w <= 126 ? 2 : 3); ++mode) {
                    // one image row of 128 pixels per tile, or tiles across
                    // the rows of strips of equal width (at most 254; at
                    // most 126 for shorter blocks)
                    const int lim = mode == 1 ? 254 : 126;
                    const int strips = mode == 0 ? (w + 127) / 128 : (w + lim - 1) / lim;
                    const int Ws = mode == 0 ? 128 : (w + strips - 1) / strips;
                    const int P = Ws + 2, TS = mode == 0 ? P : 128;
                    for (int R : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32}) {
                        if (R > h && R > 1) break;
                        const int tiles = mode == 0 ? R : ((R - 1) * P + Ws + 127) / 128;
                        if (nst > 1 && tiles > slots) break;
                        const size_t region = round1k((size_t)(R + 2) * P * 2 * kc);
                        const size_t stage = (KCs / kc) * region + (resident ? 0 : round1k((size_t)18 * Ng * KCs));
                        const size_t fixed = (resident ? round1k(wall) : 0) + conv_over_rows(tiles, TS, R, P) * 2 * kc;
                        if (fixed + stage > cap) break;
                        const int S = (int)std::min<size_t>(kMaxStages, (cap - fixed) / stage);
                        const int64_t nblk = (int64_t)nimg * strips * ((h + R - 1) / R);
                        const int ctas = (int)std::max<int64_t>(1, std::min<int64_t>(nblk, sms / groups));
                        const int64_t rounds = (nblk + ctas - 1) / ctas;
                        const double load = ((double)(R + 2) * P * 2 * C + (resident ? 0.0 : (double)wall)) / 32;
                        double total;
                        if (nst == 1) {  // the warps take alternate blocks
                            const double issue = tiles * (9.0 * (C / 16) * 58 + 300) + 400;
                            const double pipe = std::max(std::max(tiles * mma, load), tiles * epi);
                            total = S > 1 || rounds == 1 ? std::max(rounds * pipe, (rounds + 1) / 2 * issue)
                                                         : rounds * (issue + load + 1000);
                        } else {  // alternate tiles of each stage
                            const double issue = (tiles + 1) / 2 * (9.0 * (KCs / 16) * 58 + 250) + 350;
                            const double stage_t = std::max(std::max(tiles * mma / nst, load / nst), issue);
                            total = rounds * std::max(nst * (S > 1 ? stage_t : stage_t + load / nst + 1000), tiles * epi);
                        }
                        const double cost = total + load / nst + 2 * epi + (resident ? wall / 40.0 : 0.0);
                        if (cost < best.cost)
                            best = ConvPlan{Ng, groups, Ws, R, TS, KCs, kc, S, resident, ctas * groups, cost};
                    }
                }
            }
        }
    }
    CRT_CHECK(best.cost < 1e30, CRT_ERR_INVALID, "conv3x3: tile does not fit shared memory");
    return best;
}

// The orders and plans of the shapes a thread has launched: the search takes
// longer than a launch. At most kMost shapes (about 150 B each) are kept, after
// that all are dropped and searched again; a training step of the denoiser
// uses 21, so one of varying batch size stays within it.
class ConvPlans {
  public:
    using Plan = std::pair<ConvOrder, ConvPlan>;
    static constexpr size_t kMost = 1024;
    Plan get(int nimg, int h, int w, int C, int N, bool one_group, int sms) {
        const Key key{nimg, h, w, C, N, one_group, sms};
        const auto it = kept_.find(key);
        if (it != kept_.end()) return it->second;
        ++searches;
        const ConvOrder ord = conv_order(C, N, w);
        const Plan plan{ord, conv_plan(ord, nimg, h, w, C, N, sms, one_group)};
        if (kept_.size() >= kMost) kept_.clear();
        kept_.emplace(key, plan);
        return plan;
    }
    size_t size() const { return kept_.size(); }
    int64_t searches = 0;

  private:
    using Key = std::array<int, 7>;
    struct Hash {
        size_t operator()(const Key &k) const {
            uint64_t h = 1469598103934665603ull;
            for (int v : k) h = (h ^ (uint32_t)v) * 1099511628211ull;
            return (size_t)(h ^ h >> 32);
        }
    };
    std::unordered_map<Key, Plan, Hash> kept_;
};

}  // namespace crt
