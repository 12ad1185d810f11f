// Tensor-core partial kernel of the decode attention, generic over the residual layout (the *Field structs say how a
// lane obtains the 16 coordinates of a field).  Included by decode_bitmap.cu and decode_packed_mma.cu.
//
// A warp handles blocks of 16 tokens; both contractions run on mma.sync.m16n8k16 tiles:
//
//   S[16 tok x 8 cols]   = K'[16 tok x 128] . Qt^T           (8 k-steps, K' and Qt split hi + lo FP16)
//   O^T[128 x 8 cols]   += Vres^T[128 x 16 tok] . P[16 tok x 8 cols]   (8 m-blocks)
//
// The contraction order of an MMA is free, so coordinates are assigned to fragment slots such that every lane owns
// *contiguous 16-coordinate fields* of a token: lane (g = lane / 4, q = lane % 4) builds, for K, two tokens, coordinates
// [16q, 16q+16) and their RoPE partners [64+16q, 64+16q+16); for V, four tokens, coordinates [16g, 16g+16).
//
// What bounds it: instructions per token (decoding, centroid add, rotation, hi/lo split), not bytes -- so the split of
// the work is made for warps in flight and for few instructions:
//
//  * One CTA of 16 warps per SM with 128 registers a thread: four warps per scheduler.  (Two CTAs of four warps at 255
//    registers kept two per scheduler and issued on 58 % of the cycles.)
//  * What makes 128 registers enough: the accumulators and the 32 sin/cos values of a lane live in tensor memory, whose
//    loads and stores do not touch the shared-memory pipe (the other busy unit): a k-step's eight sin/cos values are
//    loaded while its residuals are walked, the accumulators for the value phase only, half of them at a time.  And the
//    two tokens of a lane have the *same* offset j = 8 warp + g inside two sub-tiles X and Y of (up to) 128 tokens, so one
//    set of 16 (cos, sin) values rotates both.  RoPE: a token at offset j of a sub-tile starting at position P0 scores
//    < R(pos_q) q, R(P0 + j) k > = < R(pos_q - P0) q, R(j) k >; the query is rotated once per sub-tile, and the eight columns of the score MMA hold X's heads (0..3) next to Y's (4..7).  Rows
//    of X use the one half of the columns, rows of Y the other; the columns stay apart to the end of the segment
//    (running maxima, sums, cluster masses and numerators are per column), where they are added.  With eight query heads
//    per KV head X and Y get MMAs of their own.
//  * Every warp copies its own 16 rows (16-byte asynchronous copies, rows 16 bytes apart from dense, so that lanes that
//    walk the same field of different tokens start in different banks): keys as soon as the key phase has read them,
//    values after the value phase, so that either has the other phase's time to arrive and one set of rows is enough.
//    Key centroids are held twice, for even and odd g, so that the 16-byte loads of eight lanes never collide.
//  * Warps meet only for the rotated query: double buffered, written by the warps in turn after their key phase, one
//    mbarrier arrival per warp and pass, waited for (bounded) before the next key phase.
//  * Rotations are packed FP32 pairs (fma.rn.f32x2), quantised codes are decoded two at a time by one AND-XOR and one
//    HFMA2.
//
// Measured (batch 32, 8 KV heads, 8128 tokens, 32 of 128 values kept): 0.219 ms; of active cycles 67 % of the issue slots,
// 76 % of the shared-memory pipe, 46 % of the integer pipe; 75 instructions and 21 shared-memory wavefronts per token and
// KV head.  Neither unit is full: four warps per scheduler do not cover the latencies of a pass, so a shorter instruction
// stream alone gives little.  The fields' walks in groups of four, half of the accumulators in registers at a time, two
// score accumulators and the maximum taken across lanes only where it grows: 83 -> 75 instructions, calls with their merge,
// us: batch 32 228 -> 225, batch 8, 16320 tokens INT4 105.4 -> 100.5, batch 16, 8128 tokens INT2 105 -> 100, batch 8, 65536
// tokens 426 -> 420.
// Tried and slower (same call, from 224): the rotated query in tensor memory, 19 wavefronts fewer per pass and 47
// instructions more, 232; 20 warps at 96 registers 239; a fused multiply-add for the rotation's subtraction 228; the
// k-steps or the halves as loops 226 to 232.
// Before (two CTAs of four warps, sin/cos and accumulators in registers): 0.280 ms.  INT4, batch 8, 16320 tokens: 0.128
// -> 0.100 ms.  A 128-token call costs ~9 us, most of it the set-up (tables, centroids, first query) and one pass.
//
// Softmax keeps a lazily updated running maximum per column (rescale only when it grows by more than 2^8), P is rounded
// to FP16 once and that rounded value is used for the sum, the cluster masses and the PV product alike.  The cluster
// masses beta[value cluster][column] are a third contraction on the same P, onehot(value id)^T . P.
//
// Precision: a single FP16 rounding of the rotated key is not enough (outlier channels put the score error at ~1e-3, ten
// times the output tolerance on short contexts), so K' enters the MMA as hi + lo FP16 halves:
// S = K'hi.Qhi + K'hi.Qlo + K'lo.Qhi.  add.f32.f16 adds the FP16 residual to the FP32 centroid in one instruction and
// fma.f32.f16 forms lo = k' - hi without unpacking.
#pragma once

namespace mma {

constexpr int kWarpsM = 16;
constexpr int kThreadsM = kWarpsM * 32;
constexpr int kSub = 8 * kWarpsM;     // tokens of a sub-tile: eight per warp
constexpr int kTileM = 2 * kSub;      // tokens per pass of the CTA
constexpr int kCenStride = 256;       // floats per centroid row in shared memory: 128 coordinates, twice (see cen_index)
constexpr int kQStride = 132;         // halfs per query row
static_assert(kTileM % kGranule == 0, "passes start at granules");
constexpr float kRescaleThreshold = 8.0f;  // log2 units
constexpr float kNoMax = -1e30f;      // running maximum before the first token: finite, so that differences are

// A warp's slice of one pass: rows 0..7 are X's tokens, 8..15 Y's.  The value side's metadata arrives with the keys (rank
// bases of both sides are formed at once) while the previous one is still in use: two buffers.
template <class ML>
struct WarpRows {
    static constexpr int kRow = ML::kPayloadBytes + ML::kPad, kMeta = ML::kMetaBytes ? ML::kMetaBytes : 1;
    alignas(16) unsigned char kp[16 * kRow];
    alignas(16) unsigned char vp[16 * kRow];
    alignas(16) unsigned char km[16 * kMeta];
    alignas(16) unsigned char vm[2][16 * kMeta];
};

template <int GQA>
constexpr int query_rows() {  // rows of the score MMA's B operand: X's and Y's heads
    return GQA == 8 ? 16 : 8;
}

// centroid row (FP32): 16-byte unit (field f = d / 16 = 4 hl + q, step ks = d / 4 % 4) of copy `odd`.  The eight lanes
// (g, g + 1; q = 0..3) of a quarter warp read one (ks, hl) of two rows: q and the copy alone choose the banks.
__device__ __forceinline__ int cen_index(int d, int odd) {
    const int f = d >> 4, ks = (d >> 2) & 3;
    return (ks * 2 + (f >> 2)) * 32 + (f & 3) * 8 + odd * 4 + (d & 3);
}

// d = fp16(bits) + c, one instruction (sm_100 mixed-precision add)
__device__ __forceinline__ float add_f16_f32(unsigned short bits, float c) {
    float d;
    asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"(bits), "f"(c));
    return d;
}
// d = fp16(a) * fp16(b) + c
__device__ __forceinline__ float fma_f16_f16_f32(unsigned short a, unsigned short b, float c) {
    float d;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"(a), "h"(b), "f"(c));
    return d;
}
// (hi, lo) FP16 pairs of two FP32 values: hi = fp16(x), lo = fp16(x - hi)
__device__ __forceinline__ void split_h2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x0, x1);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const unsigned short minus_one = 0xbc00;
    const float l0 = fma_f16_f16_f32(__half_as_ushort(__low2half(h)), minus_one, x0);
    const float l1 = fma_f16_f16_f32(__half_as_ushort(__high2half(h)), minus_one, x1);
    const __half2 l = __floats2half2_rn(l0, l1);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}


// two FP32 values in one register pair
__device__ __forceinline__ uint64_t pack_f2(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpack_f2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul_f2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t sub_f2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma_f2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Tensor memory of a warp, in columns: sin/cos values (eight per k-step: two pairs of cosines, two of sines), value
// accumulators, cluster-mass accumulators.  The four warps of a lane quarter share its columns.
constexpr int kColTrig = 0, kColAcc = 32, kColBeta = 64, kColsWarp = 80, kTmemCols = 512;
static_assert(kColsWarp * (kWarpsM / 4) <= kTmemCols, "tensor memory");

// A lane quarter's (one head per KV head: a warp's) results of one head at the end of a segment: coordinate d at red_pos(d), cluster masses.  The
// strides keep the stores of a warp (lanes g, q; one coordinate of the field) in distinct banks.
constexpr int kRedAcc = 152, kRedBeta = 72;
constexpr int kStatsWarp = 64;  // floats between the warps' column maxima and sums (one warp's rank bases)
__device__ __forceinline__ int red_pos(int d) { return (d & 15) * 9 + (d >> 4); }

// Dynamic shared memory, in this order: the warps' rows and, for the set-up, the offset tables (the end of a segment
// reuses their memory for the quarters' results), key centroids, rotated queries, query items, step table, rank bases.
template <int GQA, class ML>
struct Smem {
    static constexpr size_t kRing = sizeof(WarpRows<ML>) * kWarpsM;
    static constexpr size_t kRed =  // warps' or quarters' results
        (GQA == 1 ? kWarpsM * (kRedAcc + kRedBeta + 2) : 4 * GQA * (kRedAcc + kRedBeta)) * sizeof(float);
    static constexpr size_t kTrig = (kWarpsM + 8) * 64 * sizeof(float2);
    static constexpr size_t kRegion = ((kRing + kTrig > kRed ? kRing + kTrig : kRed) + 127) / 128 * 128;
    static constexpr size_t kQuery = 2 * 2 * query_rows<GQA>() * kQStride * sizeof(__half);  // [buffers][hi, lo][rows]
    static constexpr size_t kItems = static_cast<size_t>(2 * GQA) * 32 * 2 * sizeof(float4);  // raw query, angle state
    static constexpr size_t kStep = 64 * (sizeof(float2) + sizeof(float));  // (cos, sin) of a pass's step, frequencies
    static constexpr size_t kPre = kWarpsM * 32 * sizeof(uint2);
    static constexpr size_t kFixed = kRegion + kQuery + kItems + kStep + kPre;
    static_assert(kFixed + kMaxClusters * kCenStride * sizeof(float) <= 227 * 1024 - 256, "shared memory");
    static constexpr size_t bytes(int ck) {
        return kRegion + static_cast<size_t>(ck) * kCenStride * sizeof(float) + kQuery + kItems + kStep + kPre;
    }
};

// sin and cos of n f: the product's rounding error, up to 2e-3 rad at 32K tokens and more beyond, is added to first order.
__device__ __forceinline__ void sincos_product(float n, float f, float& s, float& c) {
    const float a = n * f, e = fmaf(n, f, -a);
    float s0, c0;
    sincosf(a, &s0, &c0);
    s = fmaf(c0, e, s0), c = fmaf(-s0, e, c0);
}

__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}

// Byte offset, inside a token's 16-byte bitmap, of the 16-bit field that covers
// coordinates [16f, 16f+16) (bit 15 = first coordinate).
__device__ __forceinline__ int field_offset(int f) { return ((f & 4) ? 8 : 0) + 6 - 2 * (f & 3); }

// Number of retained coordinates before each of the eight fields, one byte each.
__device__ __forceinline__ uint2 rank_bases(const uint4 bm) {
    const uint32_t w0 = bm.y, w1 = bm.x, w2 = bm.w, w3 = bm.z;
    const uint32_t r1 = __popc(w0 >> 16), r2 = __popc(w0);
    const uint32_t r3 = r2 + __popc(w1 >> 16), r4 = r2 + __popc(w1);
    const uint32_t r5 = r4 + __popc(w2 >> 16), r6 = r4 + __popc(w2);
    const uint32_t r7 = r6 + __popc(w3 >> 16);
    return make_uint2((r1 << 8) | (r2 << 16) | (r3 << 24), r4 | (r5 << 8) | (r6 << 16) | (r7 << 24));
}

__device__ __forceinline__ float h2f_bits(uint32_t bits) {
    return __half2float(__ushort_as_half(static_cast<unsigned short>(bits)));
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t as_bits(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
// (low halves of a and b), (high halves of a and b)
__device__ __forceinline__ uint32_t low_halves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5410); }
__device__ __forceinline__ uint32_t high_halves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }

// ---- fields: the 16 coordinates [16 f, 16 f + 16) of one token, as a lane consumes them --------
// keys:   order(i) = which four coordinates [4 ks, 4 ks + 4) come i-th; add4(ks, k, scale): k[e] += residual of
//         coordinate 4 ks + e (k holds the FP32 centroid), called in that order.
// values: half_block(half, f0..f3, a): A operands of the value MMAs i = 4 half .. 4 half + 3 for the tokens of f0, f1
//         (k columns 2q, 2q + 1) and f2, f3 (2q + 8, 2q + 9): coordinate first(i) in the rows g (a[0], a[2]), coordinate
//         second(i) in the rows g + 8 (a[1], a[3]); called for half = 0, then 1.
// `meta` and `pay` point at the token's own rows, `pre` at its eight rank bases.

// Sparse FP16 layouts: a 16-bit keep mask (bit 15 = first coordinate) and a pointer to the
// field's first retained value; retained values are consecutive in the payload row.
struct WalkField {
    static constexpr bool kSlotwise = true;  // offers add1, a single coordinate
    uint32_t mask;
    const __half* ptr;
    __device__ static constexpr int order(int i) { return i; }
    __device__ static constexpr int first(int i) { return 2 * i; }
    __device__ static constexpr int second(int i) { return 2 * i + 1; }
    __device__ __forceinline__ void add1(int slot, float& k) {
        if (mask & (0x8000u >> slot)) {
            k = add_f16_f32(*reinterpret_cast<const unsigned short*>(ptr), k);
            ++ptr;
        }
    }
    // FP16 bits of the coordinates [s0, s0 + 4) of two tokens (low and high half), 0 where dropped.  One field's four steps
    // follow one another: 3.2 instructions per coordinate by the counters instead of 3.8 with the two fields in turn (eight
    // at a time: fewer still, but slower).
    __device__ static __forceinline__ void pairs(WalkField& lo, WalkField& hi, int s0, uint32_t (&v)[4]) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v[e] = 0;
            if (lo.mask & (0x8000u >> (s0 + e))) {
                v[e] = *reinterpret_cast<const unsigned short*>(lo.ptr);
                ++lo.ptr;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (hi.mask & (0x8000u >> (s0 + e))) {
                v[e] = low_halves(v[e], *reinterpret_cast<const unsigned short*>(hi.ptr));
                ++hi.ptr;
            }
        }
    }
    // The same of one coordinate, the two walks in turn: more instructions, less waiting.
    __device__ static __forceinline__ uint32_t pair(WalkField& lo, WalkField& hi, int slot) {
        uint32_t v = 0;
        if (lo.mask & (0x8000u >> slot)) {
            v = *reinterpret_cast<const unsigned short*>(lo.ptr);
            ++lo.ptr;
        }
        if (hi.mask & (0x8000u >> slot)) {
            v = low_halves(v, *reinterpret_cast<const unsigned short*>(hi.ptr));
            ++hi.ptr;
        }
        return v;
    }
    __device__ static __forceinline__ void half_block(int half, WalkField& f0, WalkField& f1, WalkField& f2, WalkField& f3, uint32_t (&a)[4][4]) {
#pragma unroll
        for (int s0 = 0; s0 < 8; s0 += 4) {
            uint32_t x[4], y[4];
            pairs(f0, f1, 8 * half + s0, x);
            pairs(f2, f3, 8 * half + s0, y);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                uint32_t (&to)[4] = a[s0 / 2 + j];
                to[0] = x[2 * j], to[1] = x[2 * j + 1], to[2] = y[2 * j], to[3] = y[2 * j + 1];
            }
        }
    }
};

// Unstructured FP16: MSB-first bitmap; rank bases from the warp's table `pre` (8 bytes per token).
template <int NNZ>
struct LayoutMmaBitmap {
    static constexpr int kPayloadBytes = NNZ * 2, kMetaBytes = 16, kPad = 16;
    static constexpr bool kScale = false, kPrefix = true;
    using Field = WalkField;
    __device__ static __forceinline__ Field field(const unsigned char* pay, const unsigned char* meta,
                                                  const unsigned char* pre, int f, bool ok) {
        Field fd;
        fd.mask = ok ? *reinterpret_cast<const unsigned short*>(meta + field_offset(f)) : 0u;
        fd.ptr = reinterpret_cast<const __half*>(pay) + pre[f];
        return fd;
    }
};

// Tiled FP16 (INDEXED = false): one LSB-first 16-bit mask per tile = field.  Structured 4:16
// (INDEXED = true): four 4-bit in-tile indices.  Metadata word w carries tile 2w (low half) and
// 2w + 1 (high half), i.e. tile f sits at byte 2 f; its values start at f * NNZ / 8.
template <int NNZ, bool INDEXED>
struct LayoutMmaTiled {
    static constexpr int kPayloadBytes = NNZ * 2, kMetaBytes = 16, kPad = 16;
    static constexpr bool kScale = false, kPrefix = false;
    using Field = WalkField;
    __device__ static __forceinline__ Field field(const unsigned char* pay, const unsigned char* meta,
                                                  const unsigned char*, int f, bool ok) {
        const uint32_t code = ok ? *reinterpret_cast<const unsigned short*>(meta + 2 * f) : 0u;
        Field fd;
        if constexpr (INDEXED) {
            // four in-tile indices -> keep mask with bit 15 = first coordinate
            const uint32_t c = code;
            fd.mask = ok ? ((0x8000u >> (c & 15u)) | (0x8000u >> ((c >> 4) & 15u)) | (0x8000u >> ((c >> 8) & 15u)) |
                            (0x8000u >> (c >> 12)))
                         : 0u;
        } else {
            fd.mask = __brev(code) >> 16;  // LSB-first -> bit 15 = first coordinate
        }
        fd.ptr = reinterpret_cast<const __half*>(pay) + f * (NNZ / 8);
        return fd;
    }
};

// Integer codes -> exact FP16 integers, two at a time: code a at bits [S, S + BITS) and code b at [16 + S, 16 + S + BITS)
// of `w` (as stored, two's complement).  One AND-XOR leaves 1024 + (code ^ sign) * 2^S in each half, one HFMA2 rescales
// and removes the offsets (all exact).
template <int BITS, int S>
__device__ __forceinline__ uint32_t codes_to_h2(uint32_t w) {
    constexpr uint32_t kSign = 1u << (BITS - 1), kOne = ((1u << BITS) - 1u) << S, kXor = 0x6400u | (kSign << S);
    const uint32_t y = (w & (kOne * 0x10001u)) ^ (kXor * 0x10001u);
    constexpr float kDown = 1.0f / static_cast<float>(1 << S);
    return as_bits(__hfma2(as_h2(y), __float2half2_rn(kDown), __float2half2_rn(-1024.0f * kDown - static_cast<float>(kSign))));
}

// Unstructured INT4 / INT2: all 16 coordinates of a field are stored (2 words / 1 word), code i at bit BITS * i of its
// word; residual = code * scale (scale FP16 per token).  A decoded pair holds the coordinates (k, k + kHalf) of a word.
template <int BITS>
struct QuantField {
    static constexpr bool kSlotwise = false;
    static constexpr int kHalf = 16 / BITS;  // codes per half word
    uint32_t w0, w1;
    uint32_t p[4];  // the four pairs decoded last
    __device__ static constexpr int order(int i) { return BITS == 4 ? i : (i & 1) * 2 + (i >> 1); }
    __device__ static constexpr int first(int i) { return BITS == 4 ? i + (i & 4) : i; }
    __device__ static constexpr int second(int i) { return first(i) + kHalf; }
    // pair k of word `w`: coordinates k and k + kHalf
    template <int K>
    __device__ static __forceinline__ uint32_t pair(uint32_t w) {
        return codes_to_h2<BITS, (BITS * K) % 8>(BITS * K >= 8 ? w >> 8 : w);
    }
    template <int K0>
    __device__ __forceinline__ void decode(uint32_t w) {
        p[0] = pair<K0>(w), p[1] = pair<K0 + 1>(w), p[2] = pair<K0 + 2>(w), p[3] = pair<K0 + 3>(w);
    }
    __device__ __forceinline__ void add4(int ks, float (&k)[4], unsigned short scale) {
        bool high;
        if constexpr (BITS == 4) {
            if (ks == 0) decode<0>(w0);
            if (ks == 2) decode<0>(w1);
            high = ks & 1;
        } else {
            if (ks == 0) decode<0>(w0);
            if (ks == 1) decode<4>(w0);
            high = ks >= 2;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) k[e] = fma_f16_f16_f32(static_cast<unsigned short>(high ? p[e] >> 16 : p[e] & 0xffffu), scale, k[e]);
    }
    __device__ __forceinline__ uint32_t value(int i) const {
        if constexpr (BITS == 4) {
            const uint32_t w = i < 4 ? w0 : w1;
            return (i & 3) == 0 ? pair<0>(w) : (i & 3) == 1 ? pair<1>(w) : (i & 3) == 2 ? pair<2>(w) : pair<3>(w);
        } else {
            return i == 0 ? pair<0>(w0) : i == 1 ? pair<1>(w0) : i == 2 ? pair<2>(w0) : i == 3 ? pair<3>(w0)
                   : i == 4 ? pair<4>(w0) : i == 5 ? pair<5>(w0) : i == 6 ? pair<6>(w0) : pair<7>(w0);
        }
    }
    __device__ static __forceinline__ void half_block(int half, QuantField& f0, QuantField& f1, QuantField& f2, QuantField& f3, uint32_t (&a)[4][4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) block(4 * half + i, f0, f1, f2, f3, a[i]);
    }
    __device__ static __forceinline__ void block(int i, QuantField& f0, QuantField& f1, QuantField& f2, QuantField& f3, uint32_t (&a)[4]) {
        const uint32_t v0 = f0.value(i), v1 = f1.value(i), v2 = f2.value(i), v3 = f3.value(i);
        a[0] = low_halves(v0, v1), a[1] = high_halves(v0, v1), a[2] = low_halves(v2, v3), a[3] = high_halves(v2, v3);
    }
};

template <int BITS>
struct LayoutMmaQuant {
    static constexpr int kPayloadBytes = 16 * BITS, kMetaBytes = 0, kPad = 16;
    static constexpr bool kScale = true, kPrefix = false;
    using Field = QuantField<BITS>;
    __device__ static __forceinline__ Field field(const unsigned char* pay, const unsigned char*, const unsigned char*, int f, bool ok) {
        Field fd;
        fd.w0 = fd.w1 = 0u;
        if (ok) {
            if constexpr (BITS == 4) {
                const uint2 w = *reinterpret_cast<const uint2*>(pay + 8 * f);
                fd.w0 = w.x, fd.w1 = w.y;
            } else {
                fd.w0 = *reinterpret_cast<const uint32_t*>(pay + 4 * f);
            }
        }
        return fd;
    }
};

// Fields that yield the FP16 bits of a coordinate group by group (bits4): the pairs of two tokens are put together here.
template <class F>
struct GroupBlock {
    __device__ static constexpr int order(int i) { return i; }
    __device__ static constexpr int first(int i) { return 2 * i; }
    __device__ static constexpr int second(int i) { return 2 * i + 1; }
    __device__ static __forceinline__ void half_block(int half, F& f0, F& f1, F& f2, F& f3, uint32_t (&a)[4][4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) block(4 * half + i, f0, f1, f2, f3, a[i]);
    }
    __device__ static __forceinline__ void block(int i, F& f0, F& f1, F& f2, F& f3, uint32_t (&a)[4]) {
        const uint32_t v0 = f0.pair(i), v1 = f1.pair(i), v2 = f2.pair(i), v3 = f3.pair(i);
        a[0] = low_halves(v0, v1), a[1] = high_halves(v0, v1), a[2] = low_halves(v2, v3), a[3] = high_halves(v2, v3);
    }
};

// Compact quantised layout: a 16-bit keep mask like the FP16 bitmap layout, but the field's retained
// coordinates are BITS-wide codes inside the token's packed row.  At most 16 codes of 4 bits: the
// field's codes fit one 64-bit window, fetched once (three aligned words, funnel-shifted to the
// field's first code) and consumed from the low end.  A code enters arithmetic as the FP16 number
// 1024 + (code ^ sign), i.e. bits 0x6400 | (code ^ sign); the offset 1024 + sign is removed by the
// consumer.
template <int BITS>
struct CompactField : GroupBlock<CompactField<BITS>> {
    static constexpr bool kSlotwise = false;
    static constexpr uint32_t kSign = 1u << (BITS - 1);
    static constexpr uint32_t kZero = 0x6400u | kSign;  // FP16 bits of the value that stands for code 0
    uint32_t mask, lo, hi;
    __device__ __forceinline__ uint32_t next() {  // FP16 bits of the next retained code; advances the window
        const uint32_t h = ((lo & ((1u << BITS) - 1u)) ^ kZero);
        lo = __funnelshift_r(lo, hi, BITS);
        hi >>= BITS;
        return h;
    }
    __device__ __forceinline__ void add4(int ks, float (&k)[4], unsigned short scale) {
        // k += code * scale for retained coordinates (code = h - (1024 + sign), exact in FP16)
        const __half off = __float2half_rn(1024.f + static_cast<float>(kSign));
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (mask & (0x8000u >> (4 * ks + e))) {
                const __half code = __hsub(__ushort_as_half(static_cast<unsigned short>(next())), off);
                k[e] = fma_f16_f16_f32(__half_as_ushort(code), scale, k[e]);
            }
        }
    }
    // coordinates 2 i and 2 i + 1 as FP16 integers, 0 where dropped
    __device__ __forceinline__ uint32_t pair(int i) {
        const uint32_t r0 = (mask & (0x8000u >> (2 * i))) ? next() : kZero, r1 = (mask & (0x8000u >> (2 * i + 1))) ? next() : kZero;
        return as_bits(__hadd2(as_h2(low_halves(r0, r1)), __float2half2_rn(-(1024.f + static_cast<float>(kSign)))));
    }
};

template <int BITS, int NNZ>
struct LayoutMmaCompact {
    static constexpr int kPayloadBytes = NNZ * BITS / 8, kMetaBytes = 16, kPad = 16;
    static constexpr bool kScale = true, kPrefix = true;
    static_assert(kPayloadBytes % 16 == 0, "packed rows must be whole 16-byte pieces");
    using Field = CompactField<BITS>;
    __device__ static __forceinline__ Field field(const unsigned char* pay, const unsigned char* meta,
                                                  const unsigned char* pre, int f, bool ok) {
        Field fd;
        fd.mask = ok ? *reinterpret_cast<const unsigned short*>(meta + field_offset(f)) : 0u;
        // first code of the field = rank base * BITS bits into the row; words past the row's end are
        // never consumed (a field holds at most popcount(mask) codes), so their index is clamped
        constexpr int kWords = kPayloadBytes / 4;
        const uint32_t* row = reinterpret_cast<const uint32_t*>(pay);
        const int bit = pre[f] * BITS, w = bit >> 5, sh = bit & 31;
        const uint32_t w0 = row[min(w, kWords - 1)], w1 = row[min(w + 1, kWords - 1)], w2 = row[min(w + 2, kWords - 1)];
        fd.lo = __funnelshift_r(w0, w1, sh);
        fd.hi = __funnelshift_r(w1, w2, sh);
        return fd;
    }
};

// 1-of-4 structured INT4: per 4-coordinate group one signed nibble and a 2-bit position.
struct StructInt4Field : GroupBlock<StructInt4Field> {
    static constexpr bool kSlotwise = false;
    uint32_t c02, c13;  // the field's four group codes as FP16: groups (0, 2) and (1, 3)
    uint32_t sel;       // four 2-bit in-group positions, times 16 (shift amounts)
    __device__ __forceinline__ uint32_t code(int ks) const {  // in the low half
        const uint32_t p = (ks & 1) ? c13 : c02;
        return (ks & 2) ? p >> 16 : p & 0xffffu;
    }
    // coordinates 2 i and 2 i + 1, half a group: the code shifted to its place; shifts beyond the word leave zero
    __device__ __forceinline__ uint32_t pair(int i) const {
        const uint32_t at = ((sel >> (2 * (i >> 1))) & 0x30u) - 32u * (i & 1);
        uint32_t v;
        asm("shl.b32 %0, %1, %2;" : "=r"(v) : "r"(code(i >> 1)), "r"(at));
        return v;
    }
    __device__ __forceinline__ void add4(int ks, float (&k)[4], unsigned short scale) const {
        const uint32_t lo = pair(2 * ks), hi = pair(2 * ks + 1);
        k[0] = fma_f16_f16_f32(static_cast<unsigned short>(lo & 0xffffu), scale, k[0]);
        k[1] = fma_f16_f16_f32(static_cast<unsigned short>(lo >> 16), scale, k[1]);
        k[2] = fma_f16_f16_f32(static_cast<unsigned short>(hi & 0xffffu), scale, k[2]);
        k[3] = fma_f16_f16_f32(static_cast<unsigned short>(hi >> 16), scale, k[3]);
    }
};

struct LayoutMmaStructInt4 {
    static constexpr int kPayloadBytes = 16, kMetaBytes = 8, kPad = 16;
    static constexpr bool kScale = true, kPrefix = false;
    using Field = StructInt4Field;
    __device__ static __forceinline__ Field field(const unsigned char* pay, const unsigned char* meta, const unsigned char*, int f, bool ok) {
        Field fd;
        fd.c02 = fd.c13 = fd.sel = 0u;
        if (ok) {
            // groups 4f..4f+3: nibbles = 16 bits at byte 2f of the packed row, positions = byte f of the metadata row
            const uint32_t nib = *reinterpret_cast<const unsigned short*>(pay + 2 * f);
            const uint32_t two = nib | (nib << 8);  // nibbles 0, 1 at bits 0, 4 and nibbles 2, 3 at bits 16, 20
            fd.c02 = codes_to_h2<4, 0>(two), fd.c13 = codes_to_h2<4, 4>(two);
            fd.sel = static_cast<uint32_t>(meta[f]) << 4;
        }
        return fd;
    }
};

// The cluster-mass accumulators of one warp.
template <int BETA>
__device__ __forceinline__ void tmem_load_beta(uint32_t taddr, float (&r)[4 * BETA]) {
    if constexpr (BETA == 2) tmem_ld8(taddr, r); else tmem_ld16(taddr, r);
}
template <int BETA>
__device__ __forceinline__ void tmem_store_beta(uint32_t taddr, const float (&r)[4 * BETA]) {
    if constexpr (BETA == 2) tmem_st8(taddr, r); else tmem_st16(taddr, r);
}

// BETA = 16-cluster blocks of the cluster-mass accumulators: 4 serves every value-centroid count, 2 serves counts up to
// 32 with eight registers less (what the launchers pick while the table is that small).
template <int GQA, class ML, int BETA>
__global__ void __launch_bounds__(kThreadsM, 1) decode_mma_kernel(const DecodeParams p) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using SM = Smem<GQA, ML>;
    using Rows = WarpRows<ML>;
    using Field = typename ML::Field;
    constexpr int kRows = query_rows<GQA>(), kRow = Rows::kRow, kMeta = ML::kMetaBytes;
    constexpr bool kDual = GQA == 8;  // X and Y need all eight columns each: MMAs of their own
    // One head per KV head, walked layouts: the walks in turn and all accumulators in registers (8 units x 30000 tokens, 64 of
    // 128 kept: 40.1 us, in groups and halves 41.3; with four heads the groups are faster, see above).
    constexpr bool kWhole = GQA == 1 && Field::kSlotwise;
    constexpr int kQItems = 2 * GQA;  // rows of the rotated query: X's heads, Y's heads
    float* kc_s = reinterpret_cast<float*>(smem_raw + SM::kRegion);
    __half* qf = reinterpret_cast<__half*>(kc_s + static_cast<size_t>(p.ck) * kCenStride);  // [2 bufs][hi, lo][kRows][kQStride]
    float4* items = reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(qf) + SM::kQuery);  // [kQItems][32][query, state]
    float2* step_s = reinterpret_cast<float2*>(items + kQItems * 64);                        // [64] (cos, sin) of kTileM f
    float* freq_s = reinterpret_cast<float*>(step_s + 64);                                    // [64]
    uint2* pre = reinterpret_cast<uint2*>(freq_s + 64) + (threadIdx.x >> 5) * 32;             // rank bases: K's 16 rows, V's
    // (cos, sin) of 8 w f and of g f: [pair i][w or g][q], the pair of frequencies 16 q + 2 i, + 1 in 16 bytes
    float2 *trig_w = reinterpret_cast<float2*>(smem_raw + SM::kRing), *trig_g = trig_w + kWarpsM * 64;
    static_assert(SM::kRing % 16 == 0, "16-byte loads of the tables");
    __shared__ uint64_t query_bar;  // one arrival per warp when its rows of the next rotated query are written
    __shared__ uint32_t tmem_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, qd = lane & 3;
    Rows& rows = reinterpret_cast<Rows*>(smem_raw)[warp];
    // ---- what touches no memory of others: this may run while the kernel before drains -------------------------------
    if (tid == 0) {
        mbar_init(&query_bar, kWarpsM);
        mbar_fence_init();
    }
    if (warp == kWarpsM - 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    auto free_tmem = [&] {  // after a barrier that every warp has passed
        if (warp == kWarpsM - 1)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "r"(kTmemCols) : "memory");
    };
    wait_for_previous_launch();
    let_next_launch_start();

    const float my_freq = rope_freq(p.inv_freq, p.theta, tid & 63);
    const float q_freq[2] = {rope_freq(p.inv_freq, p.theta, 2 * lane), rope_freq(p.inv_freq, p.theta, 2 * lane + 1)};
    const int tokens = token_count(p);
    const int granules = max((tokens + kGranule - 1) / kGranule, 1);
    // Work of the launch (see partial_schedule): CTA c takes the granules [c * chunk, (c + 1) * chunk) of all units laid
    // end to end and walks them unit by unit; the part of one unit inside the range is a *segment* and produces one
    // partial result (slot = number of CTAs that started earlier on the same unit).
    int n_pad = p.n_pad, chunk = p.chunk;
    if (p.dyn) {
        if (p.balanced) {
            const PartialSchedule sched = partial_schedule(p.units, granules, gridDim.x);
            n_pad = sched.n_pad, chunk = sched.chunk;
        } else {
            chunk = (granules + p.splits - 1) / p.splits;
            n_pad = chunk * p.splits;
        }
    }
    const uint32_t work_total = static_cast<uint32_t>(p.units) * n_pad;  // the host keeps it below 2^31
    uint32_t work = blockIdx.x * static_cast<uint32_t>(chunk);
    const uint32_t work_end = min(work_total, work + chunk);
    // a device-side token count beyond the buffers is cut to the token stride: tell the host
    if (p.dyn && blockIdx.x == 0 && tid == 0 && p.dyn[2] > p.tok_stride) atomicOr(p.status, RESKV_STATUS_STATE_RANGE);
    if (work >= work_end) {
        __syncthreads();
        free_tmem();
        return;
    }

    uint32_t query_phase = 0, tmem = 0;
    bool lost = false;
    bool set_up = false;

    while (work < work_end) {
        // ---- the segment: unit, its token range, its partial slot -------------------------------------------------
        const int unit = work / static_cast<uint32_t>(n_pad), t_pad = work - static_cast<uint32_t>(unit) * n_pad;
        const int len = min(static_cast<uint32_t>(n_pad - t_pad), work_end - work);
        const int t_begin = min(t_pad * kGranule, tokens), t_end = min((t_pad + len) * kGranule, tokens);
        const int ntiles = (t_end - t_begin + kTileM - 1) / kTileM;
        const int slot = static_cast<int>(blockIdx.x) - static_cast<int>(static_cast<uint32_t>(unit) * n_pad / static_cast<uint32_t>(chunk));
        const bool closes_unit = t_pad + len == n_pad;
        work += len;
        const int b = unit / p.kh, hkv = unit % p.kh;
        const size_t unit_tok = static_cast<size_t>(unit) * p.tok_stride + t_begin;
        const int n_tok = t_end - t_begin;
        const unsigned char* kp_g = static_cast<const unsigned char*>(p.kp) + unit_tok * ML::kPayloadBytes;
        const unsigned char* vp_g = static_cast<const unsigned char*>(p.vp) + unit_tok * ML::kPayloadBytes;

        // global loads of the set-up, requested before the copies below queue up in front of them
        uint4 cen_raw[2];  // key centroids: 8 coordinates per thread and step, at most 64 rows
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int idx = tid + k * kThreadsM;
            if (idx < p.ck * (kHeadDim / 8)) cen_raw[k] = reinterpret_cast<const uint4*>(p.kc + static_cast<size_t>(unit) * p.ck * kHeadDim)[idx];
        }
        static_assert(2 * kThreadsM * 8 >= kMaxClusters * kHeadDim, "two steps cover the table");
        // query item of this warp (see write_query): coordinates 2 lane, + 1 and their partners; the upper warps begin,
        // they have fewer rows of the tables below to fill
        constexpr int kQFirst = kWarpsM - kQItems;
        __half q_raw[4] = {};
        if (warp >= kQFirst) {
            const __half* qrow = p.q + (static_cast<size_t>(b) * p.nh + hkv * GQA + (warp - kQFirst) % GQA) * kHeadDim + 2 * lane;
            q_raw[0] = qrow[0], q_raw[1] = qrow[1], q_raw[2] = qrow[64], q_raw[3] = qrow[65];
        }

        // A pass: sub-tile length (the last pass of a segment halves what is left, so that its tokens sit in as few warps
        // as possible), and how many tokens of X and of Y there are from the warp's first one on.
        struct Pass {
            int sub, left_x, left_y;
        };
        auto pass_at = [&](int it) {
            const int rem = n_tok - it * kTileM;
            Pass ps;
            ps.sub = rem >= kTileM ? kSub : (rem + 15) / 16 * 8;
            const bool active = 8 * warp < ps.sub;
            ps.left_x = active ? rem - 8 * warp : 0, ps.left_y = active ? rem - 8 * warp - ps.sub : 0;
            return ps;
        };
        // One pass's payload rows of one side -> this warp's rows, kPieces 16-byte pieces each; the eight rows of a
        // sub-tile are contiguous in memory, so a copy instruction of the warp takes whole runs of them.  The lanes'
        // source pointers move on by a pass per call.
        constexpr int kPieces = ML::kPayloadBytes / 16, kRun = 8 * kPieces, kAll = 2 * kRun;
        constexpr int kLanes = kRun < 32 ? kRun : 32;  // lanes on one run
        // the lane's part of the offsets, of piece `lane`: sub-tile (rows of up to 32 bytes), row, piece
        const int lane_sub = kRun < 32 ? lane / kRun & 1 : 0, lane_row = lane % kLanes / kPieces, lane_piece = lane % kPieces;
        auto copy_payload = [&](const Pass& ps, const unsigned char*& src, uint32_t dst) {
            const bool full = ps.left_y >= 8;  // every row is there
            const int y_off = ps.sub * ML::kPayloadBytes;
#pragma unroll
            for (int i = 0; i < (kAll + 31) / 32; ++i) {  // piece i * 32 + lane
                const int sub = i * 32 / kRun, in_run = i * 32 % kRun;
                const bool is_y = kRun < 32 ? lane_sub != 0 : sub != 0;
                if ((kAll >= 32 || lane < kAll) && (full || in_run / kPieces + lane_row < (is_y ? ps.left_y : ps.left_x)))
                    cp_async16(dst + (sub * 8 + in_run / kPieces) * kRow, src + (is_y ? y_off : 0) + in_run * 16);
            }
            src += kTileM * ML::kPayloadBytes;
        };
        const size_t lane_src = static_cast<size_t>(8 * warp + lane_row) * ML::kPayloadBytes + lane_piece * 16;
        const uint32_t lane_dst = (lane_sub * 8 + lane_row) * kRow + lane_piece * 16;
        const unsigned char *kp_src = kp_g + lane_src, *vp_src = vp_g + lane_src;
        const uint32_t kp_dst = smem_u32(rows.kp) + lane_dst, vp_dst = smem_u32(rows.vp) + lane_dst;
        // metadata, ids and scales: one row per lane, lanes 0..15 the key side, 16..31 the value side; 8 rows of X, 8 of Y
        const bool my_y = lane & 8;
        const size_t my_tok = unit_tok + 8 * warp + (lane & 7);
        const unsigned char* meta_src = static_cast<const unsigned char*>(lane < 16 ? p.kb : p.vb) + my_tok * kMeta;
        const uint32_t meta_dst = smem_u32(lane < 16 ? rows.km : rows.vm[0]) + (lane & 15) * kMeta;
        auto issue_keys = [&](int it, const Pass& ps) {  // and the metadata of both sides
            copy_payload(ps, kp_src, kp_dst);
            if constexpr (kMeta != 0) {
                const uint32_t dst = meta_dst + (lane < 16 ? 0u : (it & 1) * (16u * kMeta));
                const unsigned char* src = meta_src + (my_y ? ps.sub * kMeta : 0);
                if ((lane & 7) < (my_y ? ps.left_y : ps.left_x)) {
                    if constexpr (kMeta == 16) cp_async16(dst, src); else cp_async8(dst, src);
                }
                meta_src += kTileM * kMeta;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        auto issue_values = [&](const Pass& ps) {
            copy_payload(ps, vp_src, vp_dst);
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        // cluster ids (and FP16 scales) of the warp's rows of a pass
        const int8_t* id_src = ((lane < 16) ? p.kid : p.vid) + my_tok;
        const __half* sc_src = ML::kScale ? ((lane < 16) ? p.ks : p.vs) + my_tok : nullptr;
        auto load_ids = [&](const Pass& ps, int& id, uint32_t& scale) {
            id = 0, scale = 0u;
            const int off = my_y ? ps.sub : 0;
            if ((lane & 7) < (my_y ? ps.left_y : ps.left_x)) {
                // volatile: issue the loads here, a whole pass ahead of their use, instead of letting the
                // compiler sink them next to the consumer
                asm volatile("ld.global.s8 %0, [%1];" : "=r"(id) : "l"(id_src + off));
                if constexpr (ML::kScale) {
                    unsigned short h;
                    asm volatile("ld.global.u16 %0, [%1];" : "=h"(h) : "l"(sc_src + off));
                    scale = h;
                }
            }
            id_src += kTileM;
            if constexpr (ML::kScale) sc_src += kTileM;
        };
        Pass next = pass_at(0);
        int ids_next;
        uint32_t scl_next;
        load_ids(next, ids_next, scl_next);
        issue_keys(0, next);
        issue_values(next);

        // ---- once per CTA: sin/cos tables of the warps' first offsets, of the eight offsets of a warp, of a pass -----
        if (!set_up) {
            static_assert(kThreadsM == 512, "four groups of 64 threads, of one frequency each, in either half");
            // rows: first offsets of the warps that get tokens, the eight offsets of a warp, a pass's step.  The warps of the
            // upper half have a row of the first query to make as well (see below) and take fewer.  (All 25 rows, dealt out
            // evenly, device time of a call in a captured graph: 192 tokens 10.97 instead of 10.76 us, 8128 tokens 18.91
            // instead of 18.79.)
            const int rows_w = ntiles <= 1 && work == work_end ? next.sub / 8 : kWarpsM, rows_all = rows_w + 9;
            const int rows_low = kQItems < kWarpsM ? rows_all * 2 / 3 : rows_all / 2;
            const bool low = tid < 256;
            const int i = tid & 63;
            if (tid < 64) freq_s[tid] = my_freq;
#pragma unroll 1
            for (int r = (low ? 0 : rows_low - 4) + (tid >> 6); r < (low ? rows_low : rows_all); r += 4) {
                const int n = r < rows_w ? 8 * r : r < rows_w + 8 ? r - rows_w : kTileM;
                float s, c;
                sincosf(static_cast<float>(n) * my_freq, &s, &c);
                const int at = (i >> 4) * 2 + (i & 1), pair = (i >> 1) & 7;
                float2* dst = r < rows_w ? trig_w + (pair * kWarpsM + r) * 8 + at
                              : r < rows_w + 8 ? trig_g + (pair * 8 + r - rows_w) * 8 + at : step_s + i;
                *dst = make_float2(c, s);
            }
            if constexpr (GQA == 1) {  // columns without a head: rows 0 and 4 of every buffer have one
                for (int i = tid; i < static_cast<int>(SM::kQuery / 4); i += kThreadsM)
                    if (i / (kQStride / 2) % 4 != 0) reinterpret_cast<uint32_t*>(qf)[i] = 0u;
            }
        }

        // ---- per unit: key centroids (FP32, two copies) ----------------------------------------------------------
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int idx = tid + k * kThreadsM, row = idx / (kHeadDim / 8), d = (idx % (kHeadDim / 8)) * 8;
            if (row >= p.ck) break;
            const __half2* h = reinterpret_cast<const __half2*>(&cen_raw[k]);
            const float2 v0 = __half22float2(h[0]), v1 = __half22float2(h[1]), v2 = __half22float2(h[2]), v3 = __half22float2(h[3]);
#pragma unroll
            for (int odd = 0; odd < 2; ++odd) {
                *reinterpret_cast<float4*>(kc_s + row * kCenStride + cen_index(d, odd)) = make_float4(v0.x, v0.y, v1.x, v1.y);
                *reinterpret_cast<float4*>(kc_s + row * kCenStride + cen_index(d + 4, odd)) = make_float4(v2.x, v2.y, v3.x, v3.y);
            }
        }

        // ---- rotated query: Qt = R(pos_q - P0) q of sub-tile P0, FP16 hi + lo.  A row (sub-tile, head) is one warp's
        // work, two frequencies per lane; the rows move on to other warps from pass to pass.  The angle goes down by
        // kTileM f per pass and is seeded exactly every kReseedTiles passes and where the sub-tile is shorter.
        auto write_query = [&](int it, int sub_len) {
            for (int r = (warp + kWarpsM - kQFirst + it * 4) % kWarpsM; r < kQItems; r += kWarpsM) {
                const int sub = r / GQA, h = r % GQA, i2 = 2 * lane;
                float4* item = items + (r * 32 + lane) * 2;
                float4 qv, st;
                if (it == 0) {
                    const float q_mul = p.scaling * kLog2e;
                    qv = make_float4(__half2float(q_raw[0]) * q_mul, __half2float(q_raw[1]) * q_mul, __half2float(q_raw[2]) * q_mul,
                                     __half2float(q_raw[3]) * q_mul);
                    item[0] = qv;
                } else {
                    const float4 old = item[1], dn = *reinterpret_cast<const float4*>(step_s + i2);  // angle - kTileM f
                    qv = item[0];
                    st = make_float4(old.x * dn.x + old.y * dn.y, old.y * dn.x - old.x * dn.y, old.z * dn.z + old.w * dn.w,
                                     old.w * dn.z - old.z * dn.w);
                }
                if (it % kReseedTiles == 0 || sub_len != kSub) {
                    const float delta = static_cast<float>(query_position(p) - (p.start_pos + t_begin + it * kTileM + sub * sub_len));
                    const float f0 = it == 0 ? q_freq[0] : freq_s[i2], f1 = it == 0 ? q_freq[1] : freq_s[i2 + 1];
                    sincos_product(delta, f0, st.y, st.x);
                    sincos_product(delta, f1, st.w, st.z);
                }
                item[1] = st;
                const float lo0 = qv.x * st.x - qv.z * st.y, hi0 = qv.z * st.x + qv.x * st.y;
                const float lo1 = qv.y * st.z - qv.w * st.w, hi1 = qv.w * st.z + qv.y * st.w;
                uint32_t lh, ll, hh, hl;
                split_h2(lo0, lo1, lh, ll);
                split_h2(hi0, hi1, hh, hl);
                __half* row_hi = qf + ((it & 1) * 2 * kRows + (kDual ? r : sub * 4 + h)) * kQStride + i2;
                __half* row_lo = row_hi + kRows * kQStride;
                *reinterpret_cast<uint32_t*>(row_hi) = lh, *reinterpret_cast<uint32_t*>(row_hi + 64) = hh;
                *reinterpret_cast<uint32_t*>(row_lo) = ll, *reinterpret_cast<uint32_t*>(row_lo + 64) = hl;
            }
        };
        static_assert(kQItems <= kWarpsM, "one query item per warp");
        if (ntiles > 0) write_query(0, next.sub);

        tc_fence_before();
        __syncthreads();  // tables, centroids and the first rotated query in place (and tensor memory allocated)
        tc_fence_after();
        if (!set_up) {
            tmem = tmem_s + (static_cast<uint32_t>(warp % 4 * 32) << 16) + warp / 4 * kColsWarp;
            const float4 *ta = reinterpret_cast<const float4*>(trig_w) + warp * 4 + qd, *tb = reinterpret_cast<const float4*>(trig_g) + lane;
            if (8 * warp < next.sub || ntiles > 1 || work < work_end) {  // else the warp gets no tokens in this call
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    float v[8];
#pragma unroll
                    for (int e2 = 0; e2 < 2; ++e2) {
                        const float4 a = ta[(2 * ks + e2) * kWarpsM * 4], e = tb[(2 * ks + e2) * 32];
                        v[2 * e2] = a.x * e.x - a.y * e.y, v[2 * e2 + 1] = a.z * e.z - a.w * e.w;
                        v[4 + 2 * e2] = a.y * e.x + a.x * e.y, v[5 + 2 * e2] = a.w * e.z + a.z * e.w;
                    }
                    tmem_st8(tmem + kColTrig + 8 * ks, v);
                }
            }
            set_up = true;
        }

        // ---- per-warp running state ------------------------------------------------------------------------------------
        // O^T in tensor memory, m-block i -> coordinate 16g + first(i) (c0, c1) and 16g + second(i) (c2, c3), columns 2q,
        // 2q+1; beta[value cluster 16 mb + g (+ 8)][columns 2q, 2q + 1] behind it
        float m_used[2] = {kNoMax, kNoMax}, l_part[2] = {0.f, 0.f};
        {
            float zero[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) zero[i] = 0.f;
            tmem_st32(tmem + kColAcc, zero);
            tmem_store_beta<BETA>(tmem + kColBeta, reinterpret_cast<float(&)[4 * BETA]>(zero));
        }
        tmem_st_wait();
        const int busy_warps = min(next.sub >> 3, kWarpsM);  // warps that get tokens (all of them unless there is one short pass)

        for (int it = 0; it < ntiles; ++it) {
            const int ids_cur = ids_next;
            const uint32_t scl_cur = scl_next;
            const Pass now = next;
            next = pass_at(it + 1);
            load_ids(next, ids_next, scl_next);
            const bool any = now.left_x > 0;
            const unsigned char* vm = rows.vm[it & 1];
            float sc[4] = {0.f, 0.f, 0.f, 0.f};
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();  // every lane's copies of this pass's keys and metadata have landed
            if constexpr (ML::kPrefix) {
                if (any) pre[lane] = rank_bases(*reinterpret_cast<const uint4*>((lane < 16 ? rows.km : vm) + (lane & 15) * kMeta));
                __syncwarp();
            }
            if (it > 0) {  // the rotated query of this pass is complete
                if (!mbar_wait(&query_bar, query_phase & 1)) lost = true;
                ++query_phase;
            }
            if (any) {
                const bool okA = g < now.left_x, okB = g < now.left_y;
                const int kidA = min(max(__shfl_sync(0xffffffffu, ids_cur, g), 0), p.ck - 1);
                const int kidB = min(max(__shfl_sync(0xffffffffu, ids_cur, g + 8), 0), p.ck - 1);
                const unsigned char* pk = reinterpret_cast<const unsigned char*>(pre + g);
                const unsigned char *payA = rows.kp + (g) * kRow, *payB = payA + 8 * kRow;
                const unsigned char *metA = rows.km + (g) * kMeta, *metB = metA + 8 * kMeta;
                Field fAl = ML::field(payA, metA, pk, qd, okA), fAh = ML::field(payA, metA, pk, 4 + qd, okA);
                Field fBl = ML::field(payB, metB, pk + 64, qd, okB), fBh = ML::field(payB, metB, pk + 64, 4 + qd, okB);
                const unsigned short kscA = static_cast<unsigned short>(__shfl_sync(0xffffffffu, scl_cur, g));
                const unsigned short kscB = static_cast<unsigned short>(__shfl_sync(0xffffffffu, scl_cur, g + 8));
                // FP32 centroid rows (copy of this lane's parity)
                const float* cA = kc_s + kidA * kCenStride + 8 * qd + 4 * (g & 1);
                const float* cB = kc_s + kidB * kCenStride + 8 * qd + 4 * (g & 1);
                const __half* qbuf = qf + ((it & 1) * 2 * kRows + g) * kQStride + 16 * qd;
                constexpr int kLo = kRows * kQStride, kY = 8 * kQStride;  // offsets of the lo halves, of Y's heads (dual)

                // Two accumulators (hi.hi; hi.lo and lo.hi).  A third one for lo.hi makes the chains of MMAs shorter and costs
                // registers; it pays at every size measured only with one head on tiled rows: 8 x 4000 tokens 46.4 -> 46.1 us,
                // 16 x 8128 140.6 -> 139.5, 300 10.13 -> 10.07.  Elsewhere (us): INT4, 8 x 16320 tokens 100.8 -> 102.0; four heads,
                // tiled 145.4 -> 147.2, bitmap 8 x 65536 419.0 -> 415.6 but 8128 tokens alone 18.2 -> 18.4; one head, bitmap
                // 115.8 -> 117.5, 4:16 223.0 -> 224.4.
                constexpr bool kThird = GQA == 1 && Field::kSlotwise && !ML::kPrefix && ML::kPayloadBytes == 128;
                float sc2[4] = {0.f, 0.f, 0.f, 0.f}, third[kThird ? 4 : 1] = {};
                float (&sc3)[4] = *reinterpret_cast<float (*)[4]>(kThird ? third : sc2);
                float sy[kDual ? 4 : 1] = {}, sy2[kDual ? 4 : 1] = {};
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const int ks = Field::order(kk);
                    // four coordinates 16q + 4ks .. +3 and their partners + 64, both tokens: k = centroid + residual
                    float trig[8];
                    tmem_ld8(tmem + kColTrig + 8 * ks, trig);
                    const float4 al = *reinterpret_cast<const float4*>(cA + 64 * ks), ah = *reinterpret_cast<const float4*>(cA + 64 * ks + 32);
                    const float4 bl = *reinterpret_cast<const float4*>(cB + 64 * ks), bh = *reinterpret_cast<const float4*>(cB + 64 * ks + 32);
                    float kAl[4] = {al.x, al.y, al.z, al.w}, kAh[4] = {ah.x, ah.y, ah.z, ah.w};
                    float kBl[4] = {bl.x, bl.y, bl.z, bl.w}, kBh[4] = {bh.x, bh.y, bh.z, bh.w};
                    if constexpr (Field::kSlotwise) {
                        if constexpr (kWhole) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                fAl.add1(4 * ks + e, kAl[e]);
                                fAh.add1(4 * ks + e, kAh[e]);
                                fBl.add1(4 * ks + e, kBl[e]);
                                fBh.add1(4 * ks + e, kBh[e]);
                            }
                        } else {
                            // one field after the other, four coordinates each: their mask bits are tested together
#pragma unroll
                            for (int e = 0; e < 4; ++e) fAl.add1(4 * ks + e, kAl[e]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) fAh.add1(4 * ks + e, kAh[e]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) fBl.add1(4 * ks + e, kBl[e]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) fBh.add1(4 * ks + e, kBh[e]);
                        }
                    } else {
                        fAl.add4(ks, kAl, kscA);
                        fAh.add4(ks, kAh, kscA);
                        fBl.add4(ks, kBl, kscB);
                        fBh.add4(ks, kBh, kscB);
                    }
                    // rotation by the offset, two frequencies at a time, then hi + lo halves
                    tmem_ld_wait(trig);
                    uint32_t hi_l[4], lo_l[4], hi_h[4], lo_h[4];  // A operands: (X e2 = 0, Y e2 = 0, X e2 = 1, Y e2 = 1)
#pragma unroll
                    for (int e2 = 0; e2 < 2; ++e2) {
                        const uint64_t c = pack_f2(trig[2 * e2], trig[2 * e2 + 1]), s = pack_f2(trig[4 + 2 * e2], trig[5 + 2 * e2]);
#pragma unroll
                        for (int tk = 0; tk < 2; ++tk) {
                            const uint64_t L = tk ? pack_f2(kBl[2 * e2], kBl[2 * e2 + 1]) : pack_f2(kAl[2 * e2], kAl[2 * e2 + 1]);
                            const uint64_t H = tk ? pack_f2(kBh[2 * e2], kBh[2 * e2 + 1]) : pack_f2(kAh[2 * e2], kAh[2 * e2 + 1]);
                            float lc0, lc1, r0, r1;
                            unpack_f2(sub_f2(mul_f2(L, c), mul_f2(H, s)), lc0, lc1);
                            unpack_f2(fma_f2(L, s, mul_f2(H, c)), r0, r1);
                            split_h2(lc0, lc1, hi_l[2 * e2 + tk], lo_l[2 * e2 + tk]);
                            split_h2(r0, r1, hi_h[2 * e2 + tk], lo_h[2 * e2 + tk]);
                        }
                    }
                    // k-steps ks (low half of the head) and ks + 4 (high half)
                    const uint2 qh_l = *reinterpret_cast<const uint2*>(qbuf + 4 * ks), ql_l = *reinterpret_cast<const uint2*>(qbuf + kLo + 4 * ks);
                    mma_16816(sc, hi_l[0], hi_l[1], hi_l[2], hi_l[3], qh_l.x, qh_l.y);
                    mma_16816(sc2, hi_l[0], hi_l[1], hi_l[2], hi_l[3], ql_l.x, ql_l.y);
                    mma_16816(sc3, lo_l[0], lo_l[1], lo_l[2], lo_l[3], qh_l.x, qh_l.y);
                    const uint2 qh_h = *reinterpret_cast<const uint2*>(qbuf + 64 + 4 * ks), ql_h = *reinterpret_cast<const uint2*>(qbuf + kLo + 64 + 4 * ks);
                    mma_16816(sc, hi_h[0], hi_h[1], hi_h[2], hi_h[3], qh_h.x, qh_h.y);
                    mma_16816(sc2, hi_h[0], hi_h[1], hi_h[2], hi_h[3], ql_h.x, ql_h.y);
                    mma_16816(sc3, lo_h[0], lo_h[1], lo_h[2], lo_h[3], qh_h.x, qh_h.y);
                    if constexpr (kDual) {
                        const uint2 yh_l = *reinterpret_cast<const uint2*>(qbuf + kY + 4 * ks), yl_l = *reinterpret_cast<const uint2*>(qbuf + kLo + kY + 4 * ks);
                        mma_16816(sy, hi_l[0], hi_l[1], hi_l[2], hi_l[3], yh_l.x, yh_l.y);
                        mma_16816(sy2, hi_l[0], hi_l[1], hi_l[2], hi_l[3], yl_l.x, yl_l.y);
                        mma_16816(sy2, lo_l[0], lo_l[1], lo_l[2], lo_l[3], yh_l.x, yh_l.y);
                        const uint2 yh_h = *reinterpret_cast<const uint2*>(qbuf + kY + 64 + 4 * ks), yl_h = *reinterpret_cast<const uint2*>(qbuf + kLo + kY + 64 + 4 * ks);
                        mma_16816(sy, hi_h[0], hi_h[1], hi_h[2], hi_h[3], yh_h.x, yh_h.y);
                        mma_16816(sy2, hi_h[0], hi_h[1], hi_h[2], hi_h[3], yl_h.x, yl_h.y);
                        mma_16816(sy2, lo_h[0], lo_h[1], lo_h[2], lo_h[3], yh_h.x, yh_h.y);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) sc[i] += kThird ? sc2[i] + sc3[i] : sc2[i];
                if constexpr (kDual) sc[2] = sy[2] + sy2[2], sc[3] = sy[3] + sy2[3];  // Y's rows
                // with shared columns only X's scores of columns 0..3 (q < 2) and Y's of columns 4..7 mean anything
                if (!(okA && (kDual || qd < 2))) sc[0] = sc[1] = -INFINITY;
                if (!(okB && (kDual || qd >= 2))) sc[2] = sc[3] = -INFINITY;
            }
            __syncwarp();  // the key rows may be rewritten
            issue_keys(it + 1, next);
            // the other query buffer is free: every warp has arrived for this pass, i.e. is past the key phase before it
            if (it + 1 < ntiles) {
                write_query(it + 1, next.sub);
                __syncwarp();
                if (lane == 0) mbar_arrive(&query_bar);
            }
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();  // the values have landed
            if (any) {
                tmem_st_wait();  // last pass's accumulators are in place
                float whole[kWhole ? 32 : 1];
                if constexpr (kWhole) tmem_ld32(tmem + kColAcc, whole);
                // value fields of rows 2q, 2q+1 (X), 2q+8, 2q+9 (Y), coordinates [16g, 16g+16)
                const unsigned char* pv = reinterpret_cast<const unsigned char*>(pre + 16 + 2 * qd);
                const unsigned char *pay = rows.vp + 2 * qd * kRow, *met = vm + 2 * qd * kMeta;
                Field f0 = ML::field(pay, met, pv, g, 2 * qd < now.left_x);
                Field f1 = ML::field(pay + kRow, met + kMeta, pv + 8, g, 2 * qd + 1 < now.left_x);
                Field f2 = ML::field(pay + 8 * kRow, met + 8 * kMeta, pv + 64, g, 2 * qd < now.left_y);
                Field f3 = ML::field(pay + 9 * kRow, met + 9 * kMeta, pv + 72, g, 2 * qd + 1 < now.left_y);
                // ================= softmax (lazy running maximum per column), log2 domain =================
                float mt[2] = {fmaxf(sc[0], sc[2]), fmaxf(sc[1], sc[3])};  // of this lane's tokens
                const bool grow = mt[0] > m_used[0] + kRescaleThreshold || mt[1] > m_used[1] + kRescaleThreshold;
                if (__any_sync(0xffffffffu, grow)) {  // rare: the columns' maxima, and everything summed so far scaled down
#pragma unroll
                    for (int off = 4; off < 32; off <<= 1) {
                        mt[0] = fmaxf(mt[0], __shfl_xor_sync(0xffffffffu, mt[0], off));
                        mt[1] = fmaxf(mt[1], __shfl_xor_sync(0xffffffffu, mt[1], off));
                    }
                    float alpha[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float m_new = fmaxf(m_used[u], mt[u]);
                        alpha[u] = fast_exp2(m_used[u] - m_new);
                        m_used[u] = m_new;
                        l_part[u] *= alpha[u];
                    }
                    if (it > 0) {  // nothing is summed yet in a segment's first pass
                        float beta[4 * BETA];
                        tmem_load_beta<BETA>(tmem + kColBeta, beta);
                        if constexpr (kWhole) {
                            tmem_ld_wait(whole);
#pragma unroll
                            for (int i = 0; i < 32; ++i) whole[i] *= alpha[i & 1];
                        } else {
                            float flat[32];
                            tmem_ld32(tmem + kColAcc, flat);
                            tmem_ld_wait(flat);
#pragma unroll
                            for (int i = 0; i < 32; ++i) flat[i] *= alpha[i & 1];
                            tmem_st32(tmem + kColAcc, flat);
                        }
                        tmem_ld_wait(beta);
#pragma unroll
                        for (int i = 0; i < 4 * BETA; ++i) beta[i] *= alpha[i & 1];
                        tmem_store_beta<BETA>(tmem + kColBeta, beta);
                        tmem_st_wait();
                    }
                }
                float beta[4 * BETA];
                tmem_load_beta<BETA>(tmem + kColBeta, beta);
                __half2 p01, p23;
                if constexpr (kDual) {
                    p01 = __floats2half2_rn(fast_exp2(sc[0] - m_used[0]), fast_exp2(sc[1] - m_used[1]));
                    p23 = __floats2half2_rn(fast_exp2(sc[2] - m_used[0]), fast_exp2(sc[3] - m_used[1]));
                } else {  // one of the two rows counts in this lane: two exponentials
                    const float s0 = qd < 2 ? sc[0] : sc[2], s1 = qd < 2 ? sc[1] : sc[3];
                    const __half2 ph = __floats2half2_rn(fast_exp2(s0 - m_used[0]), fast_exp2(s1 - m_used[1]));
                    const __half2 zero = __float2half2_rn(0.f);
                    p01 = qd < 2 ? ph : zero, p23 = qd < 2 ? zero : ph;
                }
                const float2 p01f = __half22float2(p01), p23f = __half22float2(p23);
                l_part[0] += p01f.x + p23f.x;
                l_part[1] += p01f.y + p23f.y;
                // P as B operand (tokens x columns): transpose the two 8x8 halves
                uint32_t pb0 = movmatrix_trans(as_bits(p01)), pb1 = movmatrix_trans(as_bits(p23));
                {
                    // cluster mass: one-hot rows A[c][t] = (value id of token t == c), built two tokens at a
                    // time by a packed FP16 compare; tokens beyond the end have p = 0
                    const int at = 16 + 2 * qd;
                    const int w0 = __shfl_sync(0xffffffffu, ids_cur, at), w1 = __shfl_sync(0xffffffffu, ids_cur, at + 1);
                    const int w2 = __shfl_sync(0xffffffffu, ids_cur, at + 8), w3 = __shfl_sync(0xffffffffu, ids_cur, at + 9);
                    const __half2 gg = __half2half2(__int2half_rn(g));
                    float (&bacc)[BETA][4] = reinterpret_cast<float(&)[BETA][4]>(beta);
                    const __half2 d01 = __hsub2(__halves2half2(__int2half_rn(w0), __int2half_rn(w1)), gg);
                    const __half2 d23 = __hsub2(__halves2half2(__int2half_rn(w2), __int2half_rn(w3)), gg);
                    tmem_ld_wait(beta);
#pragma unroll
                    for (int mb = 0; mb < BETA; ++mb) {
                        if (16 * mb < p.cv) {
                            const __half2 lo = __float2half2_rn(16.f * mb), hi = __float2half2_rn(16.f * mb + 8.f);
                            mma_16816(bacc[mb], as_bits(__heq2(d01, lo)), as_bits(__heq2(d01, hi)), as_bits(__heq2(d23, lo)),
                                      as_bits(__heq2(d23, hi)), pb0, pb1);
                        }
                    }
                    tmem_store_beta<BETA>(tmem + kColBeta, beta);
                }
                if constexpr (ML::kScale) {
                    // quantised values enter the MMA as integer codes: their per-token scale rides on P
                    const float vsA = h2f_bits(__shfl_sync(0xffffffffu, scl_cur, 16 + g));
                    const float vsB = h2f_bits(__shfl_sync(0xffffffffu, scl_cur, 24 + g));
                    pb0 = movmatrix_trans(as_bits(__floats2half2_rn(p01f.x * vsA, p01f.y * vsA)));
                    pb1 = movmatrix_trans(as_bits(__floats2half2_rn(p23f.x * vsB, p23f.y * vsB)));
                }
                if constexpr (kWhole) {
                    tmem_ld_wait(whole);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint32_t a0 = Field::pair(f0, f1, 2 * i), a2 = Field::pair(f2, f3, 2 * i);
                        const uint32_t a1 = Field::pair(f0, f1, 2 * i + 1), a3 = Field::pair(f2, f3, 2 * i + 1);
                        mma_16816(reinterpret_cast<float(&)[8][4]>(whole)[i], a0, a1, a2, a3, pb0, pb1);
                    }
                    tmem_st32(tmem + kColAcc, whole);
                } else {
                    // O^T += Vres^T . P, two coordinates per MMA; half of the accumulators in registers at a time
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        float flat[16];
                        tmem_ld16(tmem + kColAcc + 16 * half, flat);
                        uint32_t a[4][4];
                        Field::half_block(half, f0, f1, f2, f3, a);
                        tmem_ld_wait(flat);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            mma_16816(reinterpret_cast<float(&)[4][4]>(flat)[i], a[i][0], a[i][1], a[i][2], a[i][3], pb0, pb1);
                        tmem_st16(tmem + kColAcc + 16 * half, flat);
                    }
                }
            }
            __syncwarp();  // the value rows and rank bases may be rewritten
            issue_values(next);
        }

        // ---- the warps' results into one: a warp reads its quarter of the accumulators of the four warps that share its
        // lanes out of tensor memory and weighs them (and X's and Y's columns), so that only four sets meet in shared memory.
        // Every warp's set through shared memory, 16 of them summed behind the barrier: calls of batch 3, 4870 tokens, eight
        // heads 28.4 instead of 26.8 us, batch 1, 8128 tokens 19.7 instead of 19.5, large ones the same.
        tmem_st_wait();
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            l_part[0] += __shfl_xor_sync(0xffffffffu, l_part[0], off);
            l_part[1] += __shfl_xor_sync(0xffffffffu, l_part[1], off);
        }
        const size_t part = static_cast<size_t>(b) * p.nh + hkv * GQA;
        const bool in_range = slot >= 0 && slot < p.splits;
        if constexpr (GQA == 1) {
            // one head: sixteen sets are little to write and to read (8 units x 8000 tokens: 17.5 us, as quarters 18.1)
            float flat[32], beta[4 * BETA];
            tmem_ld32(tmem + kColAcc, flat);
            tmem_load_beta<BETA>(tmem + kColBeta, beta);
            tmem_ld_wait(flat);
            tmem_ld_wait(beta);
            const float m = fmaxf(m_used[0], __shfl_xor_sync(0xffffffffu, m_used[0], 2)), mine = fast_exp2(m_used[0] - m);
            l_part[0] *= mine;
            l_part[0] += __shfl_xor_sync(0xffffffffu, l_part[0], 2);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {  // columns 0 and 4: X's and Y's head
                flat[i] *= mine;
                flat[i] += __shfl_xor_sync(0xffffffffu, flat[i], 2);
            }
#pragma unroll
            for (int i = 0; i < 4 * BETA; i += 2) {
                beta[i] *= mine;
                beta[i] += __shfl_xor_sync(0xffffffffu, beta[i], 2);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();  // every warp is done with its rows: their memory takes the warps' results
            float* red_acc = reinterpret_cast<float*>(smem_raw);    // [warps][kRedAcc]
            float* red_beta = red_acc + kWarpsM * kRedAcc;          // [warps][kRedBeta]
            float* red_ml = red_beta + kWarpsM * kRedBeta;          // [warps][m, l]
            if (qd == 0 && warp < busy_warps) {
                float *dst = red_acc + warp * kRedAcc + g, *bdst = red_beta + warp * kRedBeta + g;
#pragma unroll
                for (int i = 0; i < 8; ++i) dst[9 * Field::first(i)] = flat[4 * i], dst[9 * Field::second(i)] = flat[4 * i + 2];
#pragma unroll
                for (int mb = 0; mb < 4; ++mb) {
                    bdst[16 * mb] = mb < BETA ? beta[mb < BETA ? 4 * mb : 0] : 0.f;
                    bdst[16 * mb + 8] = mb < BETA ? beta[mb < BETA ? 4 * mb + 2 : 0] : 0.f;
                }
                if (g == 0) red_ml[2 * warp] = m, red_ml[2 * warp + 1] = l_part[0];
            }
            __syncthreads();
            if (in_range && tid < 4 * ((kHeadDim + kMaxClusters) / 2)) {  // two values per four threads, four warps' sets each
                const int d = 2 * (tid >> 2), sub = tid & 3;
                const float* src = d < kHeadDim ? red_acc : red_beta;
                const int at0 = d < kHeadDim ? red_pos(d) : d - kHeadDim, at1 = d < kHeadDim ? red_pos(d + 1) : at0 + 1;
                const int stride = d < kHeadDim ? kRedAcc : kRedBeta;
                float2 ml[4];
                float fm = kNoMax, fl = 0.f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int w = sub + 4 * k;
                    ml[k] = w < busy_warps ? *reinterpret_cast<const float2*>(red_ml + 2 * w) : make_float2(kNoMax, 0.f);
                    fm = fmaxf(fm, ml[k].x);
                }
                fm = fmaxf(fm, __shfl_xor_sync(0xffffffffu, fm, 1)), fm = fmaxf(fm, __shfl_xor_sync(0xffffffffu, fm, 2));
                float2 sum = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int w = sub + 4 * k;
                    if (w < busy_warps) {
                        const float weight = fast_exp2(ml[k].x - fm);
                        sum.x = fmaf(src[w * stride + at0], weight, sum.x), sum.y = fmaf(src[w * stride + at1], weight, sum.y);
                        fl = fmaf(ml[k].y, weight, fl);
                    }
                }
#pragma unroll
                for (int off = 1; off < 4; off <<= 1) {
                    sum.x += __shfl_xor_sync(0xffffffffu, sum.x, off), sum.y += __shfl_xor_sync(0xffffffffu, sum.y, off);
                    fl += __shfl_xor_sync(0xffffffffu, fl, off);
                }
                const size_t row = part * p.splits + slot;
                if (sub == 0)
                    *reinterpret_cast<float2*>(d < kHeadDim ? p.ws_delta + row * kHeadDim + d : p.ws_beta + row * kMaxClusters + d - kHeadDim) = sum;
                if (tid == 0) p.ws_m[row] = ntiles > 0 ? fm : -INFINITY, p.ws_l[row] = fl;
            }
        } else {
            // per warp, in its rank bases' place: maximum and sum of the eight columns
            float* stats = reinterpret_cast<float*>(pre);
            const float* all_stats = stats - warp * kStatsWarp;
            if (g == 0) {
                *reinterpret_cast<float2*>(stats + 2 * qd) = make_float2(m_used[0], m_used[1]);
                *reinterpret_cast<float2*>(stats + 8 + 2 * qd) = make_float2(l_part[0], l_part[1]);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            tc_fence_before();
            __syncthreads();  // every warp is done with its rows: their memory takes the quarters' results
            tc_fence_after();
            float* red_acc = reinterpret_cast<float*>(smem_raw);  // [quarters][GQA][kRedAcc]
            float* red_beta = red_acc + 4 * GQA * kRedAcc;        // [quarters][GQA][kRedBeta]
            {
                // lane -> warp lane % 16, four columns (X's or Y's heads, or a half of the eight heads)
                const int from = lane & 15, four = lane >> 4 << 2;
                const float4 ms = from < busy_warps ? *reinterpret_cast<const float4*>(all_stats + from * kStatsWarp + four)
                                                    : make_float4(kNoMax, kNoMax, kNoMax, kNoMax);
                float mx[4] = {ms.x, ms.y, ms.z, ms.w};
#pragma unroll
                for (int off = kDual ? 8 : 16; off > 0; off >>= 1)
#pragma unroll
                    for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], off));
                if (warp == kWarpsM - 1) {  // the heads' maxima and sums
                    const float4 ls = from < busy_warps ? *reinterpret_cast<const float4*>(all_stats + from * kStatsWarp + 8 + four)
                                                        : make_float4(0.f, 0.f, 0.f, 0.f);
                    float sum[4] = {ls.x * fast_exp2(ms.x - mx[0]), ls.y * fast_exp2(ms.y - mx[1]), ls.z * fast_exp2(ms.z - mx[2]),
                                    ls.w * fast_exp2(ms.w - mx[3])};
#pragma unroll
                    for (int off = kDual ? 8 : 16; off > 0; off >>= 1)
#pragma unroll
                        for (int e = 0; e < 4; ++e) sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], off);
                    if (in_range && from == 0 && (kDual || lane == 0)) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const size_t row = (part + four + e) * p.splits + slot;
                            if (four + e < GQA) p.ws_m[row] = ntiles > 0 ? mx[e] : -INFINITY, p.ws_l[row] = sum[e];
                        }
                    }
                }
                if constexpr (kDual) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) mx[e] = __shfl_sync(0xffffffffu, mx[e], qd >> 1 << 4);
                }
                const float m_head[2] = {qd & 1 ? mx[2] : mx[0], qd & 1 ? mx[3] : mx[1]};  // of this lane's columns
                const int quarter = warp % 4, mine = warp / 4;
                const uint32_t quarter_cols = tmem - mine * kColsWarp;
                float acc[8] = {}, bacc[4] = {};  // m-blocks 2 mine, 2 mine + 1; cluster block `mine`
                // two source warps at a time; one without tokens has weight zero and is not read
#pragma unroll 1
                for (int from_warp = quarter; from_warp < busy_warps; from_warp += 8) {
                    const bool two = from_warp + 4 < busy_warps;
                    const uint32_t at = quarter_cols + from_warp / 4 * kColsWarp;
                    float v0[8], v1[8], b0[4], b1[4];
                    tmem_ld8(at + kColAcc + 8 * mine, v0);
                    tmem_ld4(at + kColBeta + 4 * (mine < BETA ? mine : 0), b0);
                    const uint32_t at1 = two ? at + kColsWarp : at;
                    tmem_ld8(at1 + kColAcc + 8 * mine, v1);
                    tmem_ld4(at1 + kColBeta + 4 * (mine < BETA ? mine : 0), b1);
                    const float* st = all_stats + from_warp * kStatsWarp + 2 * qd;
                    const float2 s0 = *reinterpret_cast<const float2*>(st), s1 = *reinterpret_cast<const float2*>(two ? st + 4 * kStatsWarp : st);
                    const float w0[2] = {fast_exp2(s0.x - m_head[0]), fast_exp2(s0.y - m_head[1])};
                    const float w1[2] = {two ? fast_exp2(s1.x - m_head[0]) : 0.f, two ? fast_exp2(s1.y - m_head[1]) : 0.f};
                    tmem_ld_wait(v0), tmem_ld_wait(v1), tmem_ld_wait(b0), tmem_ld_wait(b1);
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[e] = fmaf(v1[e], w1[e & 1], fmaf(v0[e], w0[e & 1], acc[e]));
#pragma unroll
                    for (int e = 0; e < 4; ++e) bacc[e] = fmaf(b1[e], w1[e & 1], fmaf(b0[e], w0[e & 1], bacc[e]));
                }
                if constexpr (!kDual) {  // X's columns and Y's
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 2);
#pragma unroll
                    for (int e = 0; e < 4; ++e) bacc[e] += __shfl_xor_sync(0xffffffffu, bacc[e], 2);
                }
                if (kDual || qd < 2) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int h = 2 * qd + u;
                        if (h < GQA) {
                            float* dst = red_acc + (quarter * GQA + h) * kRedAcc + g;
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                dst[9 * Field::first(2 * mine + i)] = acc[4 * i + u], dst[9 * Field::second(2 * mine + i)] = acc[4 * i + 2 + u];
                            float* bdst = red_beta + (quarter * GQA + h) * kRedBeta + 16 * mine + g;
                            bdst[0] = mine < BETA ? bacc[u] : 0.f, bdst[8] = mine < BETA ? bacc[2 + u] : 0.f;
                        }
                    }
                }
            }
            tc_fence_before();
            __syncthreads();
            tc_fence_after();
            if (in_range) {
#pragma unroll 1
                for (int idx = tid; idx < GQA * ((kHeadDim + kMaxClusters) / 2); idx += kThreadsM) {  // two values per step
                    constexpr int kPer = (kHeadDim + kMaxClusters) / 2;
                    const int h = idx / kPer, d = 2 * (idx % kPer);
                    const float* src = d < kHeadDim ? red_acc + h * kRedAcc : red_beta + h * kRedBeta;
                    const int at0 = d < kHeadDim ? red_pos(d) : d - kHeadDim, at1 = d < kHeadDim ? red_pos(d + 1) : at0 + 1;
                    const int stride = d < kHeadDim ? GQA * kRedAcc : GQA * kRedBeta;
                    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
                    for (int w = 0; w < 4; ++w) sum.x += src[w * stride + at0], sum.y += src[w * stride + at1];
                    const size_t row = (part + h) * p.splits + slot;
                    *reinterpret_cast<float2*>(d < kHeadDim ? p.ws_delta + row * kHeadDim + d : p.ws_beta + row * kMaxClusters + d - kHeadDim) = sum;
                }
            }
        }
        if (in_range) {
            // the segment that ends its unit marks the unit's unused slots as empty
            if (closes_unit) {
                for (int idx = tid; idx < GQA * (p.splits - slot - 1); idx += kThreadsM) {
                    const int h = idx % GQA, s = slot + 1 + idx / GQA;
                    p.ws_m[(part + h) * p.splits + s] = -INFINITY;
                    p.ws_l[(part + h) * p.splits + s] = 0.f;
                }
            }
        } else if (tid == 0) {
            atomicOr(p.status, RESKV_STATUS_STATE_RANGE);
        }
        __syncthreads();  // the next segment's copies go into the memory just read
    }
    if (lost && lane == 0) atomicOr(p.status, RESKV_STATUS_WAIT_TIMEOUT);
    free_tmem();  // every warp is past the last segment's final barrier
}

}  // namespace mma
