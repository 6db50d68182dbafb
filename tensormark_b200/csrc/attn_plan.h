// attn_plan.h — how decode attention is split over the SMs of a device, and where its splits are merged in one launch. Plain
// C++ of its arguments alone: a caller names the SM count of the device that it launches on.
#pragma once

#include <stddef.h>

namespace tmc {

struct AttnPlan {
    unsigned nsplit;        // 0: the scratch cannot hold even one split
    unsigned chunk;         // positions per split
    size_t part_floats;     // floats of partial outputs; the (max, sum) stats follow them
    unsigned sms;           // SMs of the device that the plan is for
};

inline unsigned attn_cdiv(unsigned a, unsigned b) { return (a + b - 1) / b; }

// scratch_bytes: size of the buffer that will receive partials and stats (1 << 40: no limit from it). Enough (K/V head,
// split) CTAs to cover the machine, every split at least 32 positions, and the partials fit the buffer.
inline AttnPlan plan_attention_sms(unsigned sms, unsigned H, unsigned KVH, unsigned dh, unsigned allow, size_t scratch_bytes) {
    AttnPlan pl{};
    pl.sms = sms;
    unsigned nsplit = attn_cdiv(sms, KVH);
    nsplit = nsplit < attn_cdiv(allow, 32u) ? nsplit : attn_cdiv(allow, 32u);
    const size_t per_split = (size_t)H * (dh + 2) * sizeof(float);
    const unsigned fit = (unsigned)(scratch_bytes / per_split);
    if (fit == 0) return pl;
    if (nsplit > fit) nsplit = fit;
    if (nsplit == 0) nsplit = 1;
    pl.chunk = attn_cdiv(allow, nsplit);
    pl.nsplit = attn_cdiv(allow, pl.chunk);
    pl.part_floats = (size_t)pl.nsplit * H * dh;
    return pl;
}

// The splits of the two-launch form. The plan's bound the scratch; no more CTAs than SMs, since a CTA fills one and one CTA over
// a whole wave would double the time (8 K/V heads on 148 SMs: 18 splits of the 19 planned). fixed: the number stays as it is
// when fewer positions are attended, whose count the kernel reads on the device.
struct AttnSplits { unsigned nsplit, chunk; };
inline AttnSplits attn_splits(const AttnPlan& pl, unsigned KVH, unsigned allow, bool fixed) {
    AttnSplits s{pl.nsplit, pl.chunk};
    const unsigned most = pl.sms / KVH;
    if (most && s.nsplit > most) {
        s.nsplit = most; s.chunk = attn_cdiv(allow, most);
        if (!fixed) s.nsplit = attn_cdiv(allow, s.chunk);
    }
    return s;
}

// The one-launch form: clusters of `cs` CTAs per K/V head, cs the largest that the device holds of cs, cs / 2, ... 1 whose ranges
// cdiv(allow, cs) are at most `longest` positions; two launches where none is.
//
// A cluster has a power of two of CTAs, so fewer than the SMs allow: its CTAs read for longer by what their ranges are
// longer, and that is to cost less than the merging kernel (1-1.5 us). The line is a number of elements per head by which
// the ranges are longer. Measured on both sides of it, us for two launches / one, K and V partly in L2:
//   four heads, fp16 (4608): 4.0k 7.3 / 6.4 (32/8 heads of 128, 500 positions), 4.5k 7.5 / 6.8 (20/5, 1250); 6.4k 7.5 / 7.9 (20/5, 1800),
//     7.6k 7.3 / 7.5 (32/8, 850)
//   eight heads, fp16 (3072): 2.9k 7.8 / 6.9 (32/4 of 64, 1250), 3.0k 7.2 / 6.9 (16/2 of 64, 1250); 4.0k 8.1 / 8.4 (64/8 of 128, 500),
//     4.1k 7.8 / 8.4 (32/4, 1800)
//   four or eight heads, fp32 (2048): 1.0k 6.2 / 5.5 (32/8 of 128, 300), 1.4k 6.0 / 5.5 (32/4 of 64, 850), 1.7k 6.5 / 6.6 (28/7 of 128, 850);
//     2.8k 6.1 / 6.5 (8/2 of 128, 850), 2.9k 6.0 / 6.4 (32/4, 1250)
//   one or two heads, less arithmetic per position (10752): 8.0k 6.6 / 5.7 (16/8 of 64, 1800), 10.6k 7.4 / 6.3 and fp32 7.5 / 7.1 (40/40 of
//     128, 500); 11.1k 6.7 / 6.8 (16/8, 2500), 18k fp32 10.6 / 10.7 (40/40, 850)
// The elements are not all that counts: a range is read in whole stages, and the merge of more than 40 splits makes more than one trip.
// Of 330 calls 24 are more than 2 % slower than the other form would be, the most 8/2 of 128, 2500 positions (two) 8.6 / 7.8 and 16/2
// of 64, 2500 (two) 9.3 / 8.3; 28/7 of 128, 1800 (one) is the only one where the line lets ranges grow too long, 7.4 / 7.9.
constexpr unsigned kMaxCluster = 16;                        // splits that one launch merges
struct AttnClusters { unsigned cs, longest; };
inline AttnClusters attn_clusters(unsigned sms, unsigned KVH, unsigned REP, unsigned dh, unsigned elem_bytes, unsigned allow, unsigned nsplit) {
    const unsigned more = REP <= 2 ? 10752u : elem_bytes == 4 ? 2048u : REP == 8 ? 3072u : 4608u;
    AttnClusters c{kMaxCluster, attn_cdiv(allow, nsplit) + more / dh};
    // 32 positions are a short stage; eight heads of 128 need the CTAs for the merge too (16/2, 140 fp32 positions: 6.4 us with 32, 6.1 with 8)
    while (c.cs > 1 && (c.cs * KVH > sms || (c.cs > 4 && c.cs > attn_cdiv(allow, REP * dh >= 1024 ? 8u : 32u)))) c.cs >>= 1;
    return c;
}

}  // namespace tmc
