// Definitions shared by the decode translation units.
#pragma once

#include "common.cuh"
#include "tmem.cuh"

namespace reskv {

struct DecodeParams;
// Launches the tensor-core partial kernel of a non-bitmap layout (decode_packed_mma.cu).
// layout: 0 = INT4, 1 = INT2 (unstructured), 2 = tiled FP16, 3 = structured FP16, 4 = structured INT4,
// 5 / 6 = compact INT4 with 64 / 32 codes, 7 = compact INT2 with 64 codes.
int launch_packed_mma(const DecodeParams& p, int layout, int gqa, int units, cudaStream_t stream);

namespace {

constexpr int kGranule = 32;  // tokens: the tensor-core kernel's segments start and end at multiples of this
constexpr int kMinChunk = 2;  // granules a CTA takes at least: 64 tokens, one warp per scheduler
constexpr int kTile = 64;     // tokens per pipeline stage of the warp-per-token kernel
constexpr int kWarps = 8;    // warps per CTA
constexpr int kThreads = kWarps * 32;
constexpr int kTokPerWarp = kTile / kWarps;
constexpr int kReseedTiles = 16;
constexpr int kWsHeader = 256;  // bytes reserved at the start of the workspace (status word)

}  // namespace

struct DecodeParams {
    const __half* q;
    const __half* kc;
    const int8_t* kid;
    const void* kp;   // payload rows
    const void* kb;   // metadata rows (bitmaps, tile masks / indices) or null
    const int8_t* vid;
    const void* vp;
    const void* vb;
    const __half* ks;  // per-token scales of quantised layouts or null
    const __half* vs;
    float* ws_m;
    float* ws_l;
    float* ws_delta;
    float* ws_beta;
    uint32_t* status;
    const float* inv_freq;
    int64_t tok_stride;
    int kh, nh, tokens, ck, cv;
    // splits = partial slots per query head in the workspace; chunk = granules (tensor-core kernel) or tiles (warp-per-
    // token kernel) per CTA
    int start_pos, pos_q, splits, chunk;
    // units = batch * kv heads.  n_pad: granules a unit is padded to (see partial_schedule).  balanced != 0: the tensor-
    // core kernel's own schedule, recomputed on the device when the token count lives there; balanced == 0: one CTA per
    // (unit, split) with `chunk` granules or tiles each.
    int units, balanced, grid, n_pad;  // grid = CTAs of the tensor-core kernel
    float theta, scaling;
    // optional device-resident step state {query position, dense-window tokens, compressed tokens
    // or -1, reserved}: when set it overrides pos_q, the merge kernel's recent-token count and
    // (third word, if not negative) `tokens`, so that a captured CUDA graph can be replayed for
    // consecutive decode steps and across group compressions
    const int32_t* dyn;
};

struct MergeParams {
    const float* ws_m;      // log2-domain maxima [BNH][splits], or natural-log m [BNH] when splits == 0
    const float* ws_l;
    const float* ws_delta;
    const float* ws_beta;
    const __half* vc;       // [B*KH,CV,128]
    const __half* comp_out; // splits == 0: finished compressed result to merge with
    const __half* rq;       // rotated query [BNH,128] or null
    const __half* rk;       // rotated recent keys [B*KH,Tr,128] or null
    const __half* rv;       // recent values
    const float* rscores;   // precomputed scaled scores [BNH,Tr] (natural units) or null
    __half* out;
    float* out_m;
    float* out_l;
    int kh, nh, splits, cv, tr;
    float scaling;
    const int32_t* dyn;  // device step state: dyn[1] = recent tokens (overrides tr), or null
    int64_t recent_cap;  // tokens between units in rk / rv (== tr for contiguous windows)
    uint32_t* status;    // device status word of the call's workspace, or null
};

constexpr int kMaxRecent = 1024;  // window tokens of one call

// Launches the merge kernel (decode_merge.cu): one CTA per unit; recent_max bounds a device-side window count.
int launch_merge(const MergeParams& mp, int units, int recent_max, cudaStream_t stream);

// compressed tokens of this launch: from the device step state when it carries a count
__device__ __forceinline__ int token_count(const DecodeParams& p) {
    if (p.dyn) {
        const int t = p.dyn[2];
        if (t >= 0) return static_cast<int>(min(static_cast<int64_t>(t), p.tok_stride));
    }
    return p.tokens;
}

// tiles per split: the host's figure, or the same formula on the device-side token count
__device__ __forceinline__ int split_tiles(const DecodeParams& p, int total_tiles) {
    return p.dyn ? (total_tiles + p.splits - 1) / p.splits : p.chunk;
}

// query position of this launch: from the device step state when one is attached
__device__ __forceinline__ int query_position(const DecodeParams& p) { return p.dyn ? p.dyn[0] : p.pos_q; }

// How the tensor-core kernel's granules are dealt out to `ctas` CTAs: the granules of all units are laid end to end, every
// unit padded to n_pad of them, and CTA c takes [c * chunk, (c + 1) * chunk).
struct PartialSchedule {
    int chunk, n_pad;
};

// Either an even share of everything (n_pad = the unit's granules; a CTA may then end one unit and start the next), or
// ctas / units equal pieces of every unit, whichever has the shorter slowest CTA.  In cycles: a pass of 16 rows on each of
// 4, 8, 12 or 16 warps 4500, 5700, 6800 or 8000, a further segment in a CTA 11500 (centroids, query, combining, writing,
// and that two segments leave two passes unfilled).
//
// Measured with 144 units, one CTA each, up to 32 granules: a full pass takes 6200 (INT2), 6400 (INT4), 7500 (32 of 128 in
// a bitmap), 8100 (4:16), 8800 (64 of 128) with four query heads per KV head, 8100 and 7700 (32 of 128, 1-of-4 INT4) with
// eight; a last pass on 4 or 8 warps 3200 to 5000 and 2000 to 3600 less.  One set of figures serves all: with five of these
// forms, batch 1 to 16 and 192 to 16320 tokens, what it picks is within 1.5 % of the better of both (mean 0.05 %; with 5000
// for a further segment up to 15 %, batch 16 at 1100 tokens 32.2 instead of 28.5 us).
__host__ __device__ inline long long segment_cycles(long long granules) {
    constexpr int kPass = 8;  // granules per pass: 256 tokens
    const long long rest = granules % kPass;
    return granules / kPass * 8000 + (rest ? 4500 + (rest - 1) / 2 * 1167 : 0);
}
__host__ __device__ inline PartialSchedule partial_schedule(int units, int granules, int ctas) {
    long long even = (static_cast<long long>(units) * granules + ctas - 1) / ctas;
    if (even < kMinChunk) even = kMinChunk;
    PartialSchedule s{static_cast<int>(even), granules};
    if (units <= ctas) {
        const int pieces = ctas / units;
        int piece = (granules + pieces - 1) / pieces;
        if (piece < kMinChunk) piece = kMinChunk;
        const bool crosses = granules % even != 0;
        if (segment_cycles(piece) <= segment_cycles(even) + (crosses ? 11500 : 0))
            s.chunk = piece, s.n_pad = (granules + piece - 1) / piece * piece;
    }
    return s;
}

namespace {

__device__ __forceinline__ float rope_freq(const float* inv_freq, float theta, int i) {
    return inv_freq ? inv_freq[i] : powf(theta, -static_cast<float>(i) / 64.0f);
}

}  // namespace
}  // namespace reskv
