// How a decode attention launch is laid out (decode_ops.cu); plain C++, so that the choice can be looked at without a GPU.
#pragma once

#include <stddef.h>

#include <initializer_list>

constexpr int ATT_MAX_WARPS = 12;                      // of a CTA
constexpr int ATT_SPLITS = 8;                          // CTAs of a cluster at most
constexpr int ATT_MAX_STAGES = 24;
// Bytes of dynamic shared memory one CTA may take so that two CTAs fit on an SM; alone on its SM.
constexpr size_t ATT_SMEM_BUDGET = 110 * 1024;
constexpr size_t ATT_SMEM_BUDGET_ALONE = 200 * 1024;

// The partial sums that the CTAs of a cluster leave with its first one.
static inline size_t att_cluster_part(int D, int G, int nsplit) { return nsplit > 1 ? size_t(nsplit) * G * (D + 2) * sizeof(float) : 0; }

struct AttPlan {
    int nsplit;                                        // CTAs that share a sequence and kv head
    int warps, stages_per_warp;                        // of the streaming kernel; no stages: the blocks do not fit it
    int table_cap;                                     // block ids a CTA holds
    size_t fixed;                                      // shared memory beside the ring
};

static inline AttPlan att_plan(int D, int G, int batch, int num_kv_heads, int block_size, int max_blocks_per_seq, int sm_count) {
    AttPlan p;
    const size_t chunk = size_t(block_size) * D * 2;
    p.nsplit = ATT_SPLITS;                             // the most splits that still run as a single wave of two CTAs per SM
    while (p.nsplit > 1 && (long long)batch * num_kv_heads * p.nsplit > 2LL * sm_count) p.nsplit /= 2;
    // (Halving sequences for the width of their table, so that none is waited for alone, was measured and is not done: the width is a
    // capacity and not a length, and clusters of two start later.  32 sequences of 500 to 2048 tokens, in a stream of such calls, 39.7 us
    // whole and 41.1 halved, of 250 to 1000 in a table of 2048 21.6 and 33.2; 20 of 500 to 2048 36.9 and 30.2.)
    p.table_cap = max_blocks_per_seq / p.nsplit + 2;
    p.fixed = att_cluster_part(D, G, p.nsplit) + size_t((p.table_cap + 1) & ~1) * 4 + ATT_MAX_STAGES * 8 + 1024 + 128;
    // alone on its SM: 8 warps and a deep ring; otherwise 4 or 6 warps and about half an SM's shared
    // memory.  The big CTA (48 K registers, ~200 KB) shares its SM with no CTA of the kernels before and after it in
    // the stream, so it pays only while the grid leaves most SMs to them: up to half the SMs.  (Llama-3.2-3B decode
    // step, measured inside the step: batch 1, 64 CTAs — 1.074 ms with the big CTA, 1.116 with the small one; batch 2,
    // 128 CTAs — 1.341 ms with the big one, 1.193 with the small one.)  Every warp owns stages / warps ring stages
    // and wants at least two of them, so that its next block loads while it works on the current one.
    const bool alone = 2LL * batch * num_kv_heads * p.nsplit <= sm_count;
    const size_t budget = alone ? ATT_SMEM_BUDGET_ALONE : ATT_SMEM_BUDGET;
    // Six warps of two stages where a CTA has four blocks or more for each and they fit (beside the cluster's sums, which grow with the query heads and
    // which one CTA a sequence does without: with room kept for eight CTAs' sums all the same, tables of 129 blocks and more of 3 query heads left four
    // warps, and a step of the 3B Llama at 32 sequences of up to 2048 tokens took 2168 us for 2059), otherwise four of three
    // (16 sequences of up to 2048 tokens 23.9 us with four warps, 20.8 with six; 4 sequences, 16 blocks a CTA, 13.0 and 14.6).
    // Large blocks: two, with one stage each if it must be.
    const int most = alone ? 8 : max_blocks_per_seq / p.nsplit >= 24 ? 6 : 4;
    for (int w : {most, 4, 2}) {
        const size_t fit = budget > p.fixed ? (budget - p.fixed) / (2 * chunk * w) : 0;
        p.warps = w;
        p.stages_per_warp = fit < 3 ? int(fit) : 3;
        if (p.stages_per_warp >= 2) break;
    }
    return p;
}

// Whole sequences dealt to CTAs alone on their SMs, `bins` CTAs per kv head, back and forth by falling length (rank r goes to CTA r % bins in even
// rounds, from the other end in odd ones): the longest CTA has little more than the mean or than the longest sequence.  Only where a CTA for each
// sequence and kv head (two to an SM, three of those with heads of 64 and a narrow table: 40 sequences of 64 tokens 5.0 us, dealt 9.8, of 300 8.2 and 11.5, but of 1000,
// where they are two, 21.9 and 18.4) would start a second round of them, up to three sequences a CTA.  With one round the small CTAs overlap the kernels
// before and after, which a CTA of a whole SM does not, and equally long sequences make whole rounds here: steps of the 3B Llama with 8 kv heads
// at contexts of 2000, us packed / not, equal lengths and a quarter of it to all:  19 sequences 2208 / 1836, 1680 / 1791;  24 2290 / 2033, 1844 / 1915;
// 32 2401 / 2347, 2041 / 2030;  37 2894 / 2546, 2205 / 2160;  38 2950 / 3111, 2232 / 2266;  48 3211 / 3326, 2587 / 2713;  52 3317 / 3381, 2689 / 2762;
// four a CTA: 56 3796 / 3408, 2897 / 2956;  72 4126 / 4025, 3242 / 3217.  Contexts of 400: 24 1488 / 1386, 1390 / 1341;  48 1876 / 1907, 1712 / 1728.
// (Lengths are the device's; the width of the table, which the host knows, says little of them.)
constexpr int ATT_MAX_ITEMS = 3;
constexpr size_t ATT_SMEM_SM = 228 * 1024;             // shared memory of an SM; each of its CTAs costs 1 KB beside its own
constexpr size_t ATT_SMEM_BLOCK = 227 * 1024;          // shared memory that a CTA of sm_100a may have, dynamic and static together
constexpr size_t ATT_SMEM_STATIC = 1024;               // of it the kernel's own arrays (AttShared, and the merge's weights) at most
constexpr size_t ATT_SMEM_PACKED = ATT_SMEM_BLOCK - ATT_SMEM_STATIC;
struct AttShared {
    int item_seq[ATT_MAX_ITEMS], item_len[ATT_MAX_ITEMS];
};
struct AttMergeShared {
    float wgt[8][ATT_MAX_WARPS + 2];                   // per query head: the warps' weights, the merged maximum and sum
};
struct AttBins {
    int bins, items;                                   // CTAs per kv head; sequences a CTA takes at most (0: not this way)
    int warps, stages, table_cap;
    size_t smem;
};
static inline AttBins att_bins(int D, int G, int batch, int num_kv_heads, int block_size, int max_blocks_per_seq, int sm_count, int nsplit) {
    AttBins p{};
    p.bins = sm_count / num_kv_heads;
    const AttPlan one = att_plan(D, G, batch, num_kv_heads, block_size, max_blocks_per_seq, sm_count);
    const size_t ring = size_t(one.warps) * one.stages_per_warp * block_size * D * 4, part = size_t(one.warps) * G * (D + 2) * sizeof(float);
    const long long by_smem = (long long)(ATT_SMEM_SM / ((ring > part ? ring : part) + one.fixed + ATT_SMEM_STATIC + 1024));
    const long long by_regs = 65536 / (one.warps * 32 * (D > 64 ? 168 : 128)), per_sm = by_smem < by_regs ? by_smem : by_regs;
    if (nsplit > 1 || (long long)batch * num_kv_heads <= per_sm * sm_count || batch > ATT_MAX_ITEMS * p.bins) return p;
    const int items = (batch + p.bins - 1) / p.bins;
    const size_t stage = size_t(block_size) * D * 4;
    p.table_cap = items * max_blocks_per_seq;
    for (int w : {12, 8}) {                            // two stages each, more warps before more stages
        const size_t fixed = size_t(items) * w * G * (D + 2) * sizeof(float) + size_t((p.table_cap + 1) & ~1) * 4 + size_t(batch) * 4 + ATT_MAX_STAGES * 8 +
                             1024 + 128;
        const size_t fit = ATT_SMEM_PACKED > fixed ? (ATT_SMEM_PACKED - fixed) / (stage * w) : 0;
        if (fit < 2) continue;
        p.warps = w;
        p.stages = w * 2;
        p.smem = size_t(p.stages) * stage + fixed;
        p.items = items;
        break;
    }
    return p;
}
