// WZP magnitude/sign codec on the GPU.
//
// Stream format (byte-exact with cpu/src/wzp_cpu.cpp:769-867):
//   [u32 LE group offset x groups][u24 LE metadata x chunks][payload]
// 8192 magnitudes per chunk, 16 chunks per directory group. A nonzero chunk
// stores its magnitude bytes (bit-plane transpose + zero/repetition
// elimination, or verbatim when that is not at least 3 bytes smaller) and
// then its compacted sign bits, one per nonzero magnitude, LSB first.
//
// Encoder: one CTA per chunk, chunks taken from a ticket counter so that
// every chunk's predecessors are already resident; the payload offset is
// found by decoupled lookback over per-chunk states and the chunk writes
// straight into the archive. Every wait is bounded: a wait that hits its cap
// records ST_LOOKBACK_TIMEOUT and the kernel still terminates.
// Decoder: one CTA per chunk, fused with dequantisation and the inverse
// Morton scatter into the row-major coefficient array.
#pragma once
#include "common.cuh"
#include "packed.cuh"
#include "quantize.cuh"
#include "scan.cuh"

namespace wb {

constexpr int kWzpThreads = 512;

__device__ __forceinline__ void store_u24(uint8_t* p, uint32_t v) {
    p[0] = uint8_t(v);
    p[1] = uint8_t(v >> 8);
    p[2] = uint8_t(v >> 16);
}
__device__ __forceinline__ uint32_t load_u24(const uint8_t* p) {
    return uint32_t(p[0]) | (uint32_t(p[1]) << 8) | (uint32_t(p[2]) << 16);
}
__device__ __forceinline__ uint32_t load_u32(const uint8_t* p) {
    return load_u24(p) | (uint32_t(p[3]) << 24);
}
__device__ __forceinline__ void store_u32(uint8_t* p, uint32_t v) {
    store_u24(p, v);
    p[3] = uint8_t(v >> 24);
}

// chunk lookback state: bits 62-63 flag, low 62 bits value
constexpr uint64_t kAggregate = 1ull << 62;
constexpr uint64_t kInclusive = 2ull << 62;
constexpr uint64_t kValueMask = (1ull << 62) - 1;

// Bytes of the plane / payload buffer: the 2 * 8192 plane bytes, which the
// zero and repetition elimination overwrite in place with at most
// 16384 + 2048 + 256 + 32 + 4 payload bytes, plus slack for word-wide copies.
constexpr uint32_t kEncBytes = 2 * kChunk + 2048 + 256 + 32 + 4 + 28;

// Bit planes in shared memory: the stream's natural layout puts plane p's
// u16 word b at p * blocks + b, so the 16 lanes that hold the 16 planes of one
// 32-sample group would all hit one bank. Both directions therefore keep the
// planes of a full chunk (512 blocks) at a padded pitch of kEncPitch u32
// words: lane p's word of group g lands in bank (4p + g) mod 32 (two lanes per
// bank instead of sixteen), and a thread's 32 consecutive natural bytes
// (8 words of one plane) stay 16-byte aligned and contiguous at natural word
// 8t plus 4 * (t / 32), so the zero elimination reads them, and the decoder's
// byte spreading writes them, in place. A partial chunk (a field's last)
// keeps the natural layout.
constexpr uint32_t kEncPitch = kChunk / 32 + 4; // u32 words per padded plane, full chunks
static_assert(16 * kEncPitch * 4 <= kEncBytes, "padded encoder planes fit the plane buffer");

struct WzpEncodeSmem {
    uint16_t m[kChunk + 8];            // magnitudes (+ slack for word-wide copies)
    uint8_t planes[kEncBytes];         // bit planes, then the eliminated payload in place
    uint8_t lv[2048 + 256 + 32 + 4 + 4]; // nonzero bitmap and its reductions
    uint32_t sgn[kChunk / 32 + 1];     // compacted sign bits (+ slack)
    uint32_t gcount[kChunk / 32];      // nonzero magnitudes per 32-group
    uint32_t gsign[kChunk / 32];       // per 32-group: sign bits of its nonzero magnitudes, compacted
    uint32_t sel[16];                  // byte_perm selectors: compact the bytes of a 4-bit mask
    uint8_t pack[256];                 // compressed nibbles: entry 16 * mask + value
    uint32_t tmp[2][kWzpThreads / 32]; // totals of the two block scans
    uint32_t chunk, excl, mbytes, raw;
};

struct WzpEncodeArgs {
    uint32_t n;
    uint8_t* out;       // start of the WZP stream
    size_t capacity;    // bytes available from `out`
    uint32_t* ticket;   // zeroed before launch
    uint64_t* state;    // per chunk, zeroed before launch
    uint64_t* sizes;    // per chunk byte count (output)
    uint32_t* status;
    uint32_t spin_cap;  // lookback wait bound (polls of ~0.2 us)
    uint32_t skip_publish; // test hook: this chunk never publishes (0xffffffff = none)
};

// Bit 7 of every byte of the result: the byte of w is not zero (other bits 0).
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {
    return (((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) & 0x80808080u;
}
// Four such flags in the top nibble of a product (the sixteen partial
// products have distinct places, so nothing carries into bits 28..31).
constexpr uint32_t kGatherNibble = 0x00204081u;
// 4-bit mask of the nonzero bytes of w (bit k = byte k).
__device__ __forceinline__ uint32_t nonzero_nibble(uint32_t w) { return (nonzero_bytes(w) * kGatherNibble) >> 28; }
// 4-bit mask of the bytes of w that differ from the byte before them
// (`prev` is the byte preceding w).
__device__ __forceinline__ uint32_t changed_nibble(uint32_t w, uint32_t prev) {
    return nonzero_nibble(w ^ ((w << 8) | (prev & 0xffu)));
}
// 32-bit mask of the nonzero bytes of eight words.
__device__ __forceinline__ uint32_t nonzero_mask(const uint32_t (&w)[8]) {
    uint32_t bits = 0;
#pragma unroll
    for (int k = 7; k >= 0; --k) bits = __funnelshift_l(nonzero_bytes(w[k]) * kGatherNibble, bits, 4);
    return bits;
}
// Appends the bytes of w selected by the 4-bit mask to dst + o; returns how many.
__device__ __forceinline__ uint32_t put_selected(uint8_t* dst, uint32_t o, uint32_t w, uint32_t mask,
                                                 const uint32_t* sel) {
    const uint32_t c = __popc(mask), cw = __byte_perm(w, 0u, sel[mask]);
    if (c > 0) dst[o] = uint8_t(cw);
    if (c > 1) dst[o + 1] = uint8_t(cw >> 8);
    if (c > 2) dst[o + 2] = uint8_t(cw >> 16);
    if (c > 3) dst[o + 3] = uint8_t(cw >> 24);
    return c;
}

// Copies len bytes from 4-byte aligned shared memory to any global address:
// aligned 32-bit stores for whole destination words, byte stores at the two
// ends. src must stay readable 4 bytes past len.
__device__ __forceinline__ void copy_to_global(uint8_t* dst, const uint8_t* src, uint32_t len, int tid, int nthreads) {
    const uint32_t mis = uint32_t(reinterpret_cast<uintptr_t>(dst) & 3u);
    uint32_t* base = reinterpret_cast<uint32_t*>(dst - mis);
    const uint32_t* sw = reinterpret_cast<const uint32_t*>(src);
    const uint32_t total = mis + len, words = (total + 3) / 4;
    for (uint32_t j = tid; j < words; j += nthreads) {
        const int64_t r0 = int64_t(4 * j) - mis; // source offset of the word's first byte
        if (r0 >= 0 && r0 + 4 <= int64_t(len)) {
            base[j] = mis ? __funnelshift_r(sw[j - 1], sw[j], 8 * (4 - mis)) : sw[j];
        } else {
            for (int t = 0; t < 4; ++t) {
                const int64_t r = r0 + t;
                if (r >= 0 && r < int64_t(len)) dst[r] = src[r];
            }
        }
    }
}

// Four consecutive samples through 16-byte accesses (p 16-byte aligned).
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
}
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store4(double* p, const double (&v)[4]) {
    reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}


// ---------------------------------------------------------------------------
// 16-sample blocks. The stream's bit planes are per 16 consecutive Morton
// slots (a "block"): plane p of block b is a u16 whose bit 15-j is bit 15-p
// of the block's magnitude j. In a whole 16 x 16 x bz brick (bz a power of
// two) a block is an aligned 4 x 2 x 2 box when bz = 16 and an aligned
// 4 x 4 x 1 box when bz <= 8 (the recursive octant order of morton_rank), so
// one thread can own a block: load it as four 16-byte rows, hold its 16
// magnitudes in registers and move between magnitudes and planes with one
// 16 x 16 bit transpose.

// 16 x 16 bit transpose, rows packed in pairs (w[i] = row 2i | row 2i+1 << 16,
// bit 15 of a row = column 0): on return row p holds column p. Its own
// inverse. Four block-swap stages (Hacker's Delight 7-3); the stages of
// width 8, 4 and 2 act on both halves of a word pair at once, the stage of
// width 1 inside each word.
__device__ __forceinline__ void bit_transpose16(uint32_t (&w)[8]) {
#pragma unroll
    for (int j = 8; j >= 2; j >>= 1) {
        const uint32_t m = j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : 0x33333333u;
        const int h = j / 2; // word distance of rows k and k + j
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (i & h) continue;
            const uint32_t t = (w[i] ^ (w[i + h] >> j)) & m;
            w[i] ^= t;
            w[i + h] ^= t << j;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t t = (w[i] ^ (w[i] >> 17)) & 0x5555u;
        w[i] ^= t ^ (t << 17);
    }
}

// Element layout of a block: row r (0..3) of the block's four 16-byte rows
// holds magnitudes e0(r), e0(r)+1 (x = 0, 1) and e0(r)+d, e0(r)+d+1 (x = 2, 3);
// its offset from the block origin is dz * plane + dy * nx.
// Tall: bz = 16, 4 x 2 x 2 (rows dy + 2 dz); else 4 x 4 x 1 (rows dy). A
// compile-time shape keeps the packed magnitudes in registers.
template <bool Tall> struct BlockShape {
    static __device__ __forceinline__ constexpr int e0(int r) { return Tall ? 2 * r : ((r & 1) << 1) | ((r >> 1) << 3); }
    static constexpr int d = Tall ? 8 : 4;
    static __device__ __forceinline__ uint32_t row_offset(int r, uint32_t nx, uint32_t plane) {
        return Tall ? uint32_t(r >> 1) * plane + uint32_t(r & 1) * nx : uint32_t(r) * nx;
    }
};

// Origin (x, y, z) inside a 16 x 16 x 2^zb brick of the block holding Morton
// ranks 16k .. 16k+15: the rank's bits come in levels from the bottom, 4 - zb
// levels of (x, y) bits, then zb levels of (x, y, z) bits; the block index
// drops the lowest four bits.
__device__ __forceinline__ void block_origin(uint32_t k, uint32_t zb, uint32_t& x, uint32_t& y, uint32_t& z) {
    uint32_t r = k << 4, bit = 0;
    x = y = z = 0;
    uint32_t zl = 0;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const bool withz = uint32_t(l) >= 4 - zb;
        x |= ((r >> bit) & 1u) << l;
        y |= ((r >> (bit + 1)) & 1u) << l;
        bit += 2;
        if (withz) {
            z |= ((r >> bit) & 1u) << zl;
            ++zl;
            ++bit;
        }
    }
}

// Bit compress and expand of 16 bits by nibbles through 256-entry tables in
// shared memory: about 30 instructions where the shift network of a general
// 16-bit compress takes 85. Entry 16 m + x of `pack` holds the bits of x
// selected by m, moved to bit 0 in order; of `spread`, the low popc(m) bits of
// x moved to the set positions of m.
__device__ __forceinline__ uint32_t pack_entry(uint32_t i) {
    const uint32_t m = i >> 4, x = i & 15u;
    uint32_t v = 0, n = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
        if ((m >> b) & 1u) v |= ((x >> b) & 1u) << n++;
    return v;
}
__device__ __forceinline__ uint32_t spread_entry(uint32_t i) {
    const uint32_t m = i >> 4, x = i & 15u;
    uint32_t v = 0, n = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
        if ((m >> b) & 1u) v |= ((x >> n++) & 1u) << b;
    return v;
}
// The nibbles of a 16-bit value in the low halves of four bytes.
__device__ __forceinline__ uint32_t nibble_bytes(uint32_t x) {
    x = (x | (x << 8)) & 0x00ff00ffu;
    return (x | (x << 4)) & 0x0f0f0f0fu;
}
// Bits of x selected by m, packed towards bit 0 in order.
__device__ __forceinline__ uint32_t compress16(uint32_t x, uint32_t m, const uint8_t* pack) {
    const uint32_t i = nibble_bytes(x) | (nibble_bytes(m) << 4);
    return uint32_t(pack[i & 0xffu]) | (uint32_t(pack[(i >> 8) & 0xffu]) << __popc(m & 0xfu)) |
           (uint32_t(pack[(i >> 16) & 0xffu]) << __popc(m & 0xffu)) | (uint32_t(pack[i >> 24]) << __popc(m & 0xfffu));
}
// The low popc(m) bits of x moved to the set positions of m, in order.
__device__ __forceinline__ uint32_t expand16(uint32_t x, uint32_t m, const uint8_t* spread) {
    const uint32_t h = nibble_bytes(m) << 4;
    return uint32_t(spread[(h & 0xf0u) | (x & 15u)]) |
           (uint32_t(spread[((h >> 8) & 0xf0u) | ((x >> __popc(m & 0xfu)) & 15u)]) << 4) |
           (uint32_t(spread[((h >> 16) & 0xf0u) | ((x >> __popc(m & 0xffu)) & 15u)]) << 8) |
           (uint32_t(spread[(h >> 24) | ((x >> __popc(m & 0xfffu)) & 15u)]) << 12);
}

// Nonzero mask (bit j = magnitude j) of a block from its 16 bit planes.
__device__ __forceinline__ uint32_t planes_nonzero(const uint32_t (&w)[8]) {
    const uint32_t z = (w[0] | w[1] | w[2]) | (w[3] | w[4] | w[5]) | (w[6] | w[7]); // bit 15 - j = magnitude j
    return __brev((z | (z >> 16)) & 0xffffu) >> 16;
}

// One thread per 16-sample block (thread t: Morton slots 16t .. 16t+15 of the
// chunk): stores the block's packed magnitudes w to S.m, its 16 bit planes to
// S.planes (full chunks at the padded pitch, a partial chunk in the natural
// layout, its last count % 16 magnitudes verbatim behind them), and per
// 32-group the nonzero count and the compacted sign bits of its nonzero
// magnitudes (the even thread of each pair). nm: negative mask, bit j = slot j
// (of zero magnitudes: ignored). Slots past the chunk's end hold zero.
__device__ __forceinline__ void emit_block(WzpEncodeSmem& S, uint32_t (&w)[8], uint32_t nm, uint32_t count, uint32_t t) {
    const uint32_t blocks = count >> 4;
    uint4* dm = reinterpret_cast<uint4*>(S.m + 16 * t);
    dm[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dm[1] = make_uint4(w[4], w[5], w[6], w[7]);
    if (t == blocks && (count & 15u)) {
        uint4* tail = reinterpret_cast<uint4*>(S.planes + 32 * t);
        tail[0] = make_uint4(w[0], w[1], w[2], w[3]);
        tail[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
    if ((w[0] | w[1] | w[2] | w[3] | w[4] | w[5] | w[6] | w[7]) != 0) bit_transpose16(w);
    // group statistics: this block's count and compacted signs, merged with
    // the odd neighbour's by the even thread of the pair
    const uint32_t zm = planes_nonzero(w);
    const uint32_t cnt = __popc(zm), cs = nm ? compress16(nm, zm, S.pack) : 0u;
    const uint32_t cnt1 = __shfl_xor_sync(0xffffffffu, cnt, 1), cs1 = __shfl_xor_sync(0xffffffffu, cs, 1);
    if (!(t & 1)) {
        S.gcount[t >> 1] = cnt + cnt1;
        S.gsign[t >> 1] = cs | (cs1 << cnt);
    }
    if (t < blocks) {
        uint16_t* pl = reinterpret_cast<uint16_t*>(S.planes);
        const uint32_t stride = blocks == kChunk / 16 ? 2 * kEncPitch : blocks;
#pragma unroll
        for (int p = 0; p < 16; ++p) pl[p * stride + t] = uint16_t(p & 1 ? w[p >> 1] >> 16 : w[p >> 1]);
    }
}

// Magnitude sources of the encoder: each fills every block of a chunk through
// emit_block.

// Morton-packed u16 magnitudes and a natural sign bitmap in global memory.
struct MagArrays {
    const uint16_t* mag;
    const uint32_t* sign;
    __device__ __forceinline__ void block_planes(WzpEncodeSmem& S, uint32_t first, uint32_t count, int tid) const {
        const uint32_t t = uint32_t(tid), at = 16 * t;
        uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint32_t nm = 0;
        if (at < count) {
            nm = (sign[(first + at) >> 5] >> (at & 16u)) & 0xffffu;
            if (at + 16 <= count) {
                const uint4* src = reinterpret_cast<const uint4*>(mag + first + at);
                const uint4 a = src[0], b = src[1];
                w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w, w[4] = b.x, w[5] = b.y, w[6] = b.z, w[7] = b.w;
            } else {
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j)
                    if (at + j < count) w[j >> 1] |= uint32_t(mag[first + at + j]) << (16 * (j & 1u));
            }
        }
        emit_block(S, w, nm, count, t);
    }
};

// Codes of four samples in the short form: one add of 1.5 * 2^(mantissa
// bits) rounds the scaled value to the nearest integer, ties to even, and the
// sum's bits less the constant's are that integer (as FastRound, without its
// range test). `top` collects the largest |code| as an unsigned value and ends
// above 65535 when a code does not fit 16 bits or its value is outside the
// rounding's range or not finite; the values are then not to be used. v
// receives the dequantised values. Codes of zero give +0, as x - x = +0.
template <class T> struct QuantFast;
template <> struct QuantFast<float> {
    static __device__ __forceinline__ void row(float (&v)[4], float inv, float q, int32_t (&c)[4], uint32_t& top) {
        const f2 q2 = f2_pack(q, q), down = f2_pack(-12582912.0f, -12582912.0f);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            // scalar: a packed product and sum would be contracted (f2_mul)
            const float t0 = __fadd_rn(__fmul_rn(v[2 * h], inv), 12582912.0f),
                        t1 = __fadd_rn(__fmul_rn(v[2 * h + 1], inv), 12582912.0f);
            // an out-of-range sum leaves the constant's binade, so its bits
            // differ by more than 2^22; the caller's maximum sees that
            c[2 * h] = int32_t(__float_as_uint(t0) - 0x4b400000u);
            c[2 * h + 1] = int32_t(__float_as_uint(t1) - 0x4b400000u);
            f2_unpack(f2_mul(f2_add(f2_pack(t0, t1), down), q2), v[2 * h], v[2 * h + 1]);
        }
        (void)top;
    }
};
template <> struct QuantFast<double> {
    static __device__ __forceinline__ void row(double (&v)[4], double inv, double q, int32_t (&c)[4], uint32_t& top) {
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const double t = __dadd_rn(__dmul_rn(v[x], inv), 6755399441055744.0); // 1.5 * 2^52
            c[x] = __double2loint(t);
            // the code fits 32 bits if the high word is the constant's, less
            // one for a negative code
            if (uint32_t(__double2hiint(t)) - uint32_t(c[x] >> 31) != 0x43380000u) top = 0xffffffffu;
            v[x] = __dmul_rn(__dsub_rn(t, 6755399441055744.0), q);
        }
    }
};

// Division by a divisor known to the host: r = reciprocal(d) = floor(2^64 / d)
// + 1 gives floor(x / d) for every 32-bit x and d > 1; d = 1 has r = 0.
inline uint64_t reciprocal(uint32_t d) { return d > 1 ? ~uint64_t(0) / d + 1 : 0; }
__device__ __forceinline__ uint32_t divide(uint32_t x, uint64_t r, uint32_t d) {
    return d > 1 ? uint32_t(__umul64hi(uint64_t(x), r)) : x;
}

// The coefficients themselves, quantised by the encoder (QuantizeOp fused
// in): the chunk is a run of whole 16 x 16 x bz bricks (2^lb samples
// each, the field made of whole bricks only); every brick is read and
// rewritten (dequantised) row by row, its magnitudes and negative flags placed
// at their Morton ranks, and q-outliers recorded as in QuantizeOp.
template <class T> struct QuantBricks {
    T* coeff;
    uint32_t nx, ny, bz, lb;
    uint64_t rnbx, rnby;  // reciprocals of nx / 16 and ny / 16 (reciprocal())
    T q, inv;
    uint32_t* qbits;
    uint32_t* qval;
    uint32_t* status;

    // Quantises block t of the chunk starting at `first` (its dequantised
    // values written back): packed magnitudes w (pairs of Morton slots) and
    // the negative mask (bit j = slot j of the block). Rows whose codes fit 16
    // bits take the short form (QuantFast); the others row_full().
    template <bool Tall>
    __device__ __forceinline__ void quantise_block(uint32_t first, uint32_t t, uint32_t (&w)[8], uint32_t& nm) const {
        using Sh = BlockShape<Tall>;
        const uint32_t plane = nx * ny;
        const uint32_t b = (first >> lb) + ((t << 4) >> lb), k = t & ((1u << (lb - 4)) - 1u);
        const uint32_t nbx = nx / 16, nby = ny / 16;
        const uint32_t tb = divide(b, rnbx, nbx), bxi = b - tb * nbx, slab = divide(tb, rnby, nby), byi = tb - slab * nby;
        uint32_t lx, ly, lz;
        block_origin(k, lb - 8, lx, ly, lz);
        const uint32_t at0 = (slab * bz + lz) * plane + (byi * 16 + ly) * nx + bxi * 16 + lx;
        constexpr int dd = Sh::d;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int e0 = Sh::e0(r), e1 = e0 + dd;
            T* row = coeff + at0 + Sh::row_offset(r, nx, plane);
            T v[4];
            load4(row, v);
            int32_t c[4];
            uint32_t top = 0;
            QuantFast<T>::row(v, inv, q, c, top);
            uint32_t neg = 0; // bit x = sign of sample x
#pragma unroll
            for (int x = 3; x >= 0; --x) neg = __funnelshift_l(uint32_t(c[x]), neg, 1);
            uint32_t m[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                m[x] = c[x] < 0 ? 0u - uint32_t(c[x]) : uint32_t(c[x]);
                top = max(top, m[x]);
            }
            // e0 and e1 are even: each pair fills one packed word
            w[e0 >> 1] = __byte_perm(m[0], m[1], 0x5410);
            w[e1 >> 1] = __byte_perm(m[2], m[3], 0x5410);
            if (top <= 65535u) {
                store4(row, v);
            } else {
                const uint4 full = row_full(row, at0 + Sh::row_offset(r, nx, plane), inv, q, qbits, qval, status);
                w[e0 >> 1] = full.x;
                w[e1 >> 1] = full.y;
                neg = full.z;
            }
            nm |= ((neg & 3u) << e0) | ((neg >> 2) << e1);
        }
    }

    // A row with a code of more than 16 bits or a value that is not finite:
    // sample by sample (`first`: its index in the field). Returns its two
    // packed words and its negative mask.
    static __device__ __noinline__ uint4 row_full(T* row, uint32_t first, T inv, T q, uint32_t* qbits, uint32_t* qval,
                                                  uint32_t* status) {
        uint4 out = make_uint4(0, 0, 0, 0);
        uint32_t bad = 0;
#pragma unroll 1
        for (int x = 0; x < 4; ++x) {
            int32_t m;
            bool neg;
            row[x] = quantize_one<T>(row[x], inv, q, m, neg, bad);
            const uint32_t low = uint32_t(m > 65535 ? 65535 : m) << (16 * (x & 1));
            if (x < 2) out.x |= low;
            else out.y |= low;
            out.z |= uint32_t(neg && m) << x;
            if (m > 65535) {
                const uint32_t at = first + x;
                atomicOr(&qbits[at >> 5], 1u << (at & 31));
                qval[at] = uint32_t(m);
            }
        }
        if (bad) atomicOr(status, ST_QUANT_DOMAIN);
        return out;
    }

    __device__ __forceinline__ void block_planes(WzpEncodeSmem& S, uint32_t first, uint32_t count, int tid) const {
        uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint32_t nm = 0;
        if (uint32_t(tid) < count >> 4) { // whole bricks: count is a multiple of 16
            if (bz == 16) quantise_block<true>(first, uint32_t(tid), w, nm);
            else quantise_block<false>(first, uint32_t(tid), w, nm);
        }
        emit_block(S, w, nm, count, uint32_t(tid));
    }
};

// Bound by the ALU pipe (about 60 instructions per sample, six barriers a
// chunk; four CTAs per SM overlap them). 512^3 f32: 0.41 ms (2.9 TB/s of read,
// rewrite and archive); 0.50 ms with per-sample masks, shift-network compress
// and fourteen barriers a chunk.
template <class Src> struct WzpEncodeOp {
    static constexpr int kThreads = kWzpThreads, kMinBlocks = 4; // 32 registers: four CTAs per SM
    struct Params {
        WzpEncodeArgs A;
        Src src;
    };
    static __device__ __forceinline__ void run(const Params P, uint32_t, uint32_t);
};

template <class Src>
__device__ __forceinline__ void WzpEncodeOp<Src>::run(const Params P, uint32_t, uint32_t) {
    const WzpEncodeArgs& A = P.A;
    const Src& src = P.src;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WzpEncodeSmem& S = *reinterpret_cast<WzpEncodeSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t chunks = wzp_chunks(A.n), groups = wzp_groups(A.n);
    if (tid == 0) S.chunk = atomicAdd(A.ticket, 1u);
    if (tid < 16) {
        uint32_t sel = 0x4444u, k = 0;
        for (int b = 0; b < 4; ++b)
            if ((tid >> b) & 1) {
                sel = (sel & ~(0xfu << (4 * k))) | (uint32_t(b) << (4 * k));
                ++k;
            }
        S.sel[tid] = sel;
    }
    if (tid >= 256) S.pack[tid - 256] = uint8_t(pack_entry(uint32_t(tid) - 256u));
    __syncthreads();
    const uint32_t c = S.chunk;
    if (c >= chunks) return;
    const uint32_t first = c * kChunk;
    const uint32_t count = min(kChunk, A.n - first);
    const uint32_t blocks = count / 16;

    // ---- one thread per 16-sample block: magnitudes, bit planes and group
    // statistics in one pass
    src.block_planes(S, first, count, tid);
    for (int i = tid; i < int(kChunk / 32) + 1; i += kWzpThreads) S.sgn[i] = 0;
    __syncthreads();

    // ---- zero elimination of the plane bytes (thread t owns bytes
    // 32t..32t+31, all of one plane in a warp of a full chunk) and the rank
    // offsets of the 32-groups' signs, from one block scan of both counts
    const uint32_t raw_bytes = 2 * count;
    uint32_t nnz, nzb, c1 = 0;
    {
        const uint32_t b0 = tid * 32;
        uint32_t w[8];
        const uint32_t pad = blocks == kChunk / 16 ? 4 * (kEncPitch - kChunk / 32) * (uint32_t(tid) >> 5) : 0u;
        const uint4* q = reinterpret_cast<const uint4*>(S.planes + b0 + pad);
        const uint4 q0 = q[0], q1 = q[1];
        w[0] = q0.x; w[1] = q0.y; w[2] = q0.z; w[3] = q0.w;
        w[4] = q1.x; w[5] = q1.y; w[6] = q1.z; w[7] = q1.w;
        uint32_t bits = nonzero_mask(w);
        if (b0 + 32 > raw_bytes) bits &= b0 >= raw_bytes ? 0u : ((1u << (raw_bytes - b0)) - 1u);
        const uint32_t gc = tid < int(kChunk / 32) ? S.gcount[tid] : 0u;
        uint32_t sum;
        const uint32_t at = block_excl_scan1<kWzpThreads>((uint32_t(__popc(bits)) << 16) | gc, S.tmp[0], sum);
        nzb = sum >> 16;
        nnz = sum & 0xffffu;
        // signs: each group's packed bits at its rank offset (at most two words)
        if (gc) {
            const uint32_t r = at & 0xffffu, packed = S.gsign[tid], sh = r & 31;
            if (packed) {
                atomicOr(&S.sgn[r >> 5], packed << sh);
                if (sh && (packed >> (32 - sh))) atomicOr(&S.sgn[(r >> 5) + 1], packed >> (32 - sh));
            }
        }
        // the empty high planes leave here warp by warp
        if (__any_sync(0xffffffffu, bits)) {
            uint32_t o = at >> 16;
#pragma unroll
            for (int k = 0; k < 8; ++k) o += put_selected(S.planes, o, w[k], (bits >> (4 * k)) & 15u, S.sel);
        }
        reinterpret_cast<uint32_t*>(S.lv)[tid] = bits; // bitmap bytes 4t..4t+3
    }
    __syncthreads();
    // ---- repetition elimination: 2048 -> 256 -> 32 -> 4 bytes; a byte is
    // kept iff it differs from the byte before it (before the first: 0).
    // Level 1: thread t < 256 owns bitmap bytes 8t..8t+7
    {
        uint32_t flags = 0, w0 = 0, w1 = 0;
        if (tid < 256) {
            const uint32_t* lw = reinterpret_cast<const uint32_t*>(S.lv);
            w0 = lw[2 * tid];
            w1 = lw[2 * tid + 1];
            const uint32_t prev = tid ? (lw[2 * tid - 1] >> 24) : 0u;
            flags = changed_nibble(w0, prev) | (changed_nibble(w1, w0 >> 24) << 4);
            S.lv[2048 + tid] = uint8_t(flags);
        }
        uint32_t o = nzb + block_excl_scan1<kWzpThreads>(__popc(flags), S.tmp[1], c1); // its barrier publishes the flags
        if (flags) {
            o += put_selected(S.planes, o, w0, flags & 15u, S.sel);
            put_selected(S.planes, o, w1, flags >> 4, S.sel);
        }
    }
    // ---- warp 0 alone: levels 2 and 3, the chunk's size and its place, by
    // decoupled lookback over 32 predecessor states per step (the closest
    // inclusive prefix ends the walk; every wait is bounded)
    const uint32_t sbytes = (nnz + 7) / 8;
    if (warp == 0) {
        const uint32_t* l1 = reinterpret_cast<const uint32_t*>(S.lv + 2048);
        const uint32_t v0 = l1[2 * lane], v1 = l1[2 * lane + 1];
        const uint32_t pv = lane ? (l1[2 * lane - 1] >> 24) : 0u;
        const uint32_t f2_ = changed_nibble(v0, pv) | (changed_nibble(v1, v0 >> 24) << 4);
        const uint32_t n2 = __popc(f2_);
        const uint32_t inc = warp_incl_scan(n2);
        const uint32_t c2 = __shfl_sync(0xffffffffu, inc, 31);
        uint32_t o2 = nzb + c1 + inc - n2;
        o2 += put_selected(S.planes, o2, v0, f2_ & 15u, S.sel);
        put_selected(S.planes, o2, v1, f2_ >> 4, S.sel);
        S.lv[2048 + 256 + lane] = uint8_t(f2_);
        __syncwarp();
        const uint32_t* l2 = reinterpret_cast<const uint32_t*>(S.lv + 2048 + 256);
        uint32_t f3 = 0, u0 = 0, u1 = 0;
        if (lane < 4) {
            u0 = l2[2 * lane];
            u1 = l2[2 * lane + 1];
            const uint32_t pu = lane ? (l2[2 * lane - 1] >> 24) : 0u;
            f3 = changed_nibble(u0, pu) | (changed_nibble(u1, u0 >> 24) << 4);
        }
        const uint32_t n3 = __popc(f3);
        const uint32_t inc3 = warp_incl_scan(n3);
        const uint32_t c3 = __shfl_sync(0xffffffffu, inc3, 31);
        if (lane < 4) {
            uint32_t o3 = nzb + c1 + c2 + inc3 - n3;
            o3 += put_selected(S.planes, o3, u0, f3 & 15u, S.sel);
            put_selected(S.planes, o3, u1, f3 >> 4, S.sel);
            S.planes[nzb + c1 + c2 + c3 + lane] = uint8_t(f3);
        }
        const uint32_t rze = nzb ? nzb + c1 + c2 + c3 + 4 : 0;
        const bool raw = rze + 2 >= raw_bytes;
        const uint32_t mbytes = raw ? raw_bytes : rze;
        const uint64_t chunk_bytes = nnz ? uint64_t(mbytes) + sbytes : 0;
        if (lane == 0) {
            S.mbytes = mbytes;
            S.raw = raw;
        }

        const bool publish = c != A.skip_publish;
        if (lane == 0 && publish)
            atomicExch(reinterpret_cast<unsigned long long*>(&A.state[c]),
                       (unsigned long long)((c == 0 ? kInclusive : kAggregate) | chunk_bytes));
        uint64_t excl = 0;
        bool timed_out = false;
        int64_t top = int64_t(c) - 1; // predecessor examined by lane 0
        uint32_t spins = 0;
        while (top >= 0) {
            const int64_t j = top - lane;
            const uint64_t st = j >= 0 ? *reinterpret_cast<volatile uint64_t*>(&A.state[j]) : uint64_t(2ull << 62);
            const uint32_t pub = __ballot_sync(0xffffffffu, (st >> 62) != 0);
            const uint32_t inc = __ballot_sync(0xffffffffu, (st >> 62) == 2);
            const int last = inc ? __ffs(inc) - 1 : 31; // lanes 0..last are needed
            const uint32_t need = last == 31 ? 0xffffffffu : ((2u << last) - 1u);
            if ((pub & need) != need) {
                if (++spins >= A.spin_cap) {
                    timed_out = true;
                    break;
                }
                __nanosleep(200);
                continue;
            }
            uint64_t v = lane <= last ? (st & kValueMask) : 0;
#pragma unroll
            for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            excl += v;
            if (inc) break;
            top -= 32;
        }
        if (lane == 0) {
            if (timed_out) atomicOr(A.status, ST_LOOKBACK_TIMEOUT);
            if (c > 0 && publish)
                atomicExch(reinterpret_cast<unsigned long long*>(&A.state[c]),
                           (unsigned long long)(kInclusive | (excl + chunk_bytes)));
            A.sizes[c] = chunk_bytes;
            S.excl = uint32_t(excl);
            const size_t header = size_t(groups) * 4 + size_t(chunks) * 3;
            if (header + excl + chunk_bytes > A.capacity || excl + chunk_bytes > 0xffffffffull) {
                atomicOr(A.status, ST_CAPACITY);
                S.excl = 0xffffffffu;
            }
            const uint32_t meta = nnz ? ((raw ? kRawCode : mbytes) | ((sbytes == 1024 ? 0u : sbytes) << 14)) : 0u;
            store_u24(A.out + size_t(groups) * 4 + size_t(c) * 3, meta);
        }
    }
    __syncthreads();
    if (!nnz || S.excl == 0xffffffffu) return;
    // ---- payload: magnitude bytes (eliminated, or the raw magnitudes), then
    // the sign bytes, each copied with word-wide stores
    uint8_t* dst = A.out + size_t(groups) * 4 + size_t(chunks) * 3 + S.excl;
    const uint32_t mbytes = S.mbytes;
    copy_to_global(dst, S.raw ? reinterpret_cast<const uint8_t*>(S.m) : S.planes, mbytes, tid, kWzpThreads);
    copy_to_global(dst + mbytes, reinterpret_cast<const uint8_t*>(S.sgn), sbytes, tid, kWzpThreads);
}

// Group directory: payload offset of the first byte of every nonempty group,
// for groups t, t + step, ...
__device__ __forceinline__ void wzp_write_directory(uint8_t* out, uint32_t n, const uint64_t* state,
                                                    const uint64_t* sizes, uint32_t t, uint32_t step) {
    const uint32_t chunks = wzp_chunks(n), groups = wzp_groups(n);
    for (uint32_t g = t; g < groups; g += step) {
        const uint32_t f = g * kGroup, l = min(f + kGroup, chunks) - 1;
        const uint64_t start = (state[f] & kValueMask) - sizes[f];
        const uint64_t end = state[l] & kValueMask;
        store_u32(out + size_t(g) * 4, end > start ? uint32_t(start) : 0u);
    }
}
// Bytes of the whole stream (its header included) once every chunk is done.
__device__ __forceinline__ uint64_t wzp_stream_bytes(uint32_t n, const uint64_t* state) {
    return wzp_header(n) + (state[wzp_chunks(n) - 1] & kValueMask);
}

// The directory of a standalone encode (the compressor writes it with the
// archive's layout).
struct WzpDirectoryOp {
    static constexpr int kThreads = 256, kMinBlocks = 0; // no occupancy floor: the compiler picks the register budget
    struct Params {
        uint8_t* out;
        uint32_t n;
        const uint64_t *state, *sizes;
        uint64_t* total;
    };
    static __device__ __forceinline__ void run(const Params P, uint32_t block, uint32_t blocks) {
        wzp_write_directory(P.out, P.n, P.state, P.sizes, block * kThreads + threadIdx.x, blocks * kThreads);
        if (block == 0 && threadIdx.x == 0) *P.total = wzp_stream_bytes(P.n, P.state);
    }
};

// ------------------------------------------------------------------ decode

// Brick geometry of the Morton-packed stream (bricks of 16 x 16 x bz, raster
// order z, y, x; edge bricks shrink): packed index -> row-major index.
struct BrickMap {
    uint32_t nx, ny, nz, bz;
    const uint16_t* local; // 8 slots x 256*bz: rank -> packed brick-local (x | y << 4 | z << 8)
    // Fast map: every brick whole (16 | nx, 16 | ny, bz | nz) and 256*bz a power
    // of two (lb = its log2), so a chunk is a run of whole bricks.
    bool fast;
    uint32_t lb;
    // Samples of a slab, of a row of bricks (whole / short slab) and of a brick
    // (short y + 2 * short z), and their reciprocals.
    uint32_t slab_sz, row_sz[2], brick_sz[4];
    uint64_t rslab, rrow[2], rbrick[4];
    static BrickMap make(uint32_t nx, uint32_t ny, uint32_t nz, uint32_t bz, const uint16_t* local) {
        BrickMap m{};
        m.nx = nx, m.ny = ny, m.nz = nz, m.bz = bz, m.local = local;
        const uint32_t bsz = 256 * bz;
        if (nx % 16 == 0 && ny % 16 == 0 && nz % bz == 0 && (bsz & (bsz - 1)) == 0 && bsz <= kChunk &&
            kChunk / bsz <= 32) {
            m.fast = true;
            while ((1u << m.lb) < bsz) ++m.lb;
        }
        // sizes beyond 32 bits divide every index to zero, as the largest does
        auto fit = [](uint64_t v) { return uint32_t(v < 1 ? 1 : v > 0xffffffffull ? 0xffffffffull : v); };
        m.slab_sz = fit(uint64_t(nx) * ny * bz);
        m.rslab = reciprocal(m.slab_sz);
        for (uint32_t z = 0; z < 2; ++z) {
            const uint32_t ez = z ? nz % bz : bz;
            m.row_sz[z] = fit(16ull * nx * ez);
            m.rrow[z] = reciprocal(m.row_sz[z]);
            for (uint32_t y = 0; y < 2; ++y) {
                m.brick_sz[y + 2 * z] = fit(16ull * (y ? ny % 16 : 16) * ez);
                m.rbrick[y + 2 * z] = reciprocal(m.brick_sz[y + 2 * z]);
            }
        }
        return m;
    }
    __device__ __forceinline__ uint32_t brick_base(uint32_t b) const {
        const uint32_t nbx = nx / 16, nby = ny / 16;
        const uint32_t bxi = b % nbx, t = b / nbx, byi = t % nby, slab = t / nby;
        return slab * bz * (nx * ny) + byi * 16 * nx + bxi * 16;
    }
    // Every index fits 32 bits: archives hold at most 2^32 - 1 sample bytes.
    // Divisions by the host's reciprocals: the hardware has none for integers,
    // and three per sample were most of this path (181 x 257 x 333 decode of
    // the stream 0.133 -> 0.080 ms with the block form of the magnitudes).
    __device__ __forceinline__ uint32_t rowmajor(uint32_t k) const {
        const uint32_t slab = divide(k, rslab, slab_sz);
        uint32_t r = k - slab * slab_sz;
        const uint32_t ez = min(bz, nz - slab * bz), pz = ez != bz;
        const uint32_t row = divide(r, rrow[pz], row_sz[pz]);
        r -= row * row_sz[pz];
        const uint32_t ey = min(16u, ny - row * 16), py = ey != 16, at = py + 2 * pz;
        const uint32_t bxi = divide(r, rbrick[at], brick_sz[at]);
        const uint32_t rk = r - bxi * brick_sz[at];
        const uint32_t slot = (nx - bxi * 16 < 16) | (at << 1);
        const uint32_t loc = __ldg(local + slot * 256 * bz + rk);
        const uint32_t lx = loc & 15, ly = (loc >> 4) & 15, lz = loc >> 8;
        return ((slab * bz + lz) * ny + row * 16 + ly) * nx + bxi * 16 + lx;
    }
};

// Dequantised samples T(+-m) * q of a block row: magnitudes m in the halves of
// pa (x = 0, 1) and pb (x = 2, 3), signs in bits 0, 1 of sa and sb (never set
// for m = 0). Float: a half under the exponent byte of 2^23 is 2^23 + m, so
// one exact subtraction converts it (two samples at a time).
__device__ __forceinline__ void dequant_row(uint32_t pa, uint32_t pb, uint32_t sa, uint32_t sb, float q, float (&v)[4]) {
    const f2 down = f2_pack(-8388608.0f, -8388608.0f), q2 = f2_pack(q, q);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t p = h ? pb : pa, s = h ? sb : sa;
        const f2 m = f2_pack(__uint_as_float(__byte_perm(p, 0x4b000000u, 0x7410)),
                             __uint_as_float(__byte_perm(p, 0x4b000000u, 0x7432)));
        float x, y;
        f2_unpack(f2_mul(f2_add(m, down), q2), x, y);
        v[2 * h] = __uint_as_float(__float_as_uint(x) ^ (s << 31));
        v[2 * h + 1] = __uint_as_float(__float_as_uint(y) ^ ((s << 30) & 0x80000000u));
    }
}
__device__ __forceinline__ void dequant_row(uint32_t pa, uint32_t pb, uint32_t sa, uint32_t sb, double q,
                                            double (&v)[4]) {
    const uint32_t mg[4] = {pa & 0xffffu, pa >> 16, pb & 0xffffu, pb >> 16};
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const double mag = __dmul_rn(double(mg[x]), q);
        v[x] = (((x < 2 ? sa : sb) >> (x & 1)) & 1u) ? -mag : mag;
    }
}

// Dequantises block t of a chunk (packed magnitudes w, negative mask nm) into
// the row-major coefficients as four 16-byte rows; `brick` is the row-major
// base of the block's brick.
template <class T, bool Tall>
__device__ __forceinline__ void store_block(const BrickMap& map, T* coeff, uint32_t brick, uint32_t t,
                                            const uint32_t (&w)[8], uint32_t nm, T q) {
    using Sh = BlockShape<Tall>;
    const uint32_t plane = map.nx * map.ny;
    uint32_t lx, ly, lz;
    block_origin(t & ((1u << (map.lb - 4)) - 1u), map.lb - 8, lx, ly, lz);
    const uint32_t at0 = brick + lz * plane + ly * map.nx + lx;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        constexpr int dd = Sh::d;
        const int e0 = Sh::e0(r), e1 = e0 + dd;
        T v4[4];
        dequant_row(w[e0 >> 1], w[e1 >> 1], nm >> e0, nm >> e1, q, v4);
        store4(coeff + at0 + Sh::row_offset(r, map.nx, plane), v4);
    }
}

// One word of an expanded repetition level: four entries whose bits in `mask`
// say that a new stream byte starts there; the others repeat the byte before
// (`prev` for the first). `at` is the stream position of the first new byte in
// the staged words `sw`; `rep` the byte_perm selectors of the 16 masks. Sets
// bad where a new byte equals the byte before it.
__device__ __forceinline__ uint32_t repeat_word(const uint32_t* sw, uint32_t at, uint32_t mask, uint32_t prev,
                                                const uint32_t* rep, bool& bad) {
    const uint32_t wi = at >> 2;
    const uint32_t word = __byte_perm(__funnelshift_r(sw[wi], sw[wi + 1], 8 * (at & 3u)), prev, rep[mask]);
    bad |= changed_nibble(word, prev) != mask;
    return word;
}

struct WzpDecodeSmem {
    uint32_t bbase[32];                // row-major base of each whole brick of the chunk (fast map)
    uint16_t m[kChunk + 16];           // staged magnitude bytes, then the decoded magnitudes
    uint8_t sb[1024 + 32];             // staged sign bytes
    uint32_t xsel[16];                 // byte_perm selectors: spread 4-bit-mask bytes into place
    uint32_t rep[16];                  // byte_perm selectors: expand repeated bytes
    uint8_t spread[256];               // expanded nibbles: entry 16 * mask + value
    uint8_t planes[16 * kEncPitch * 4]; // full chunks at pitch kEncPitch; a partial chunk: natural
    uint8_t lv[256];                   // level 1 of the repetition elimination
    uint32_t nsign[kChunk / 32];       // natural sign words of the decoded magnitudes
    uint32_t tmp[40];
    uint32_t tmp1[3][kWzpThreads / 32]; // totals of the block scans
    uint32_t off, mbytes, sbytes, raw, bad, pos;
};

struct WzpChunkInfo {
    uint32_t mbytes, sbytes;
    bool raw, ok;
};
__device__ __forceinline__ WzpChunkInfo wzp_meta(uint32_t meta, uint32_t count) {
    WzpChunkInfo r{0, 0, false, true};
    const uint32_t code = meta & kRawCode, scode = meta >> 14;
    if (!code) {
        r.ok = scode == 0;
        return r;
    }
    r.raw = code == kRawCode;
    if (!r.raw && (code < 4 || code + 2 >= 2 * count)) r.ok = false;
    r.sbytes = scode ? scode : 1024;
    if (r.sbytes > (count + 7) / 8) r.ok = false;
    r.mbytes = r.raw ? 2 * count : code;
    return r;
}

// Directory check by one block of NT threads: group spans must tile the payload
// exactly. This verifies the canonical (increasing) order; ST_DIRECTORY sends
// anything else to the exact host check.
template <int NT>
__device__ __forceinline__ void directory_check(const DecodeJob& J, uint32_t n, uint32_t* status, uint32_t* tmp) {
    const uint8_t* in = J.base + 32;
    const uint64_t payload = J.wzp - wzp_header(n);
    const uint32_t chunks = wzp_chunks(n), groups = wzp_groups(n);
    const uint8_t* meta = in + size_t(groups) * 4;
    uint64_t carry = 0;
    uint32_t st = 0;
    for (uint32_t base = 0; base < groups; base += NT) {
        const uint32_t g = base + threadIdx.x;
        uint32_t len = 0, off = 0;
        if (g < groups) {
            // the group's 16 metadata words are independent loads: all in flight at once
#pragma unroll
            for (uint32_t k = 0; k < kGroup; ++k) {
                const uint32_t c = g * kGroup + k;
                if (c >= chunks) break;
                const WzpChunkInfo ci = wzp_meta(load_u24(meta + size_t(c) * 3), min(kChunk, n - c * kChunk));
                if (!ci.ok) st |= ST_BAD_STREAM;
                len += ci.mbytes + ci.sbytes;
            }
            off = load_u32(in + size_t(g) * 4);
            if (off > payload || len > payload - off || (!len && off)) st |= ST_BAD_STREAM;
        }
        uint32_t sum;
        const uint32_t ex = block_excl_scan<NT>(len, tmp, sum);
        if (g < groups && len && uint64_t(off) != carry + ex) st |= ST_DIRECTORY;
        carry += sum;
    }
    if (threadIdx.x == 0 && carry != payload) st |= ST_DIRECTORY;
    if (st) atomicOr(status, st);
}

// Copies src[0, len) to dst[mis, mis + len), mis = src mod 16 (dst 16-byte
// aligned): 16-byte loads for granules wholly inside the range, bytes at its
// ends. Returns mis.
__device__ __forceinline__ uint32_t stage_bytes(uint8_t* dst, const uint8_t* src, uint32_t len, int tid, int nt) {
    const uint32_t mis = uint32_t(reinterpret_cast<uintptr_t>(src) & 15u);
    const uint8_t* a0 = src - mis;
    const uint32_t n16 = (mis + len + 15) / 16;
    for (uint32_t i = tid; i < n16; i += nt) {
        const uint32_t lo = 16 * i;
        if (lo >= mis && lo + 16 <= mis + len) {
            reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(a0)[i];
        } else {
            for (uint32_t k = 0; k < 16; ++k) {
                const uint32_t r = lo + k;
                if (r >= mis && r < mis + len) dst[r] = a0[r];
            }
        }
    }
    return mis;
}

template <class T> struct WzpDecodeArgs {
    JobRef job;         // archive base, WZP stream length, quantum
    uint32_t n;
    BrickMap map;
    T* coeff;           // row-major dequantised coefficients (output)
    uint32_t* status;
};

// Bound like the encoder (52 instructions per sample, seven barriers). 512^3
// f32: 0.34 ms; 0.46 ms with a block scan and byte loops per repetition level,
// shift-network expand and per-sample conversions.
template <class T> struct WzpDecodeOp {
    static constexpr int kThreads = kWzpThreads, kMinBlocks = 4; // 32 registers: four CTAs per SM
    using Params = WzpDecodeArgs<T>;
    // by reference: the brick map is indexed, which would put a batch's copy of
    // the parameters into local memory
    static __device__ __forceinline__ void run(const Params& A, uint32_t block, uint32_t);
};

template <class T>
__device__ __forceinline__ void WzpDecodeOp<T>::run(const Params& A, uint32_t block, uint32_t) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WzpDecodeSmem& S = *reinterpret_cast<WzpDecodeSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t chunks = wzp_chunks(A.n), groups = wzp_groups(A.n);
    // block 0 checks the directory beside the chunks' blocks (as a launch of
    // its own it took 4.7 us of every decode)
    if (block == 0) {
        directory_check<kWzpThreads>(A.job.get(), A.n, A.status, S.tmp);
        return;
    }
    const uint32_t c = block - 1;
    const uint32_t first = c * kChunk, count = min(kChunk, A.n - first);
    const size_t header = size_t(groups) * 4 + size_t(chunks) * 3;
    const DecodeJob J = A.job.get();
    const uint8_t* in = J.base + 32;
    const T q = T(J.q);
    const uint8_t* meta = in + size_t(groups) * 4;
    const uint8_t* payload = in + header;
    const size_t payload_bytes = J.wzp - header;
    // whole bricks (chunks are runs of them): one thread per 16-sample block
    const bool blockwise = A.map.fast && (reinterpret_cast<uintptr_t>(A.coeff) & 15u) == 0;

    if (warp == 0) {
        // Lane k reads the metadata of the group's chunk k; the chunk's payload
        // offset is the group offset plus its predecessors' lengths.
        const uint32_t g = c / kGroup, k = g * kGroup + lane;
        WzpChunkInfo ci{0, 0, false, true};
        if (lane < int(kGroup) && k <= c) ci = wzp_meta(load_u24(meta + size_t(k) * 3), min(kChunk, A.n - k * kChunk));
        const uint32_t len = (lane < int(kGroup) && k < c) ? ci.mbytes + ci.sbytes : 0u;
        const uint32_t before = __reduce_add_sync(0xffffffffu, len);
        const bool ok_all = __all_sync(0xffffffffu, ci.ok);
        const int me = int(c - g * kGroup);
        const uint32_t mb = __shfl_sync(0xffffffffu, ci.mbytes, me);
        const uint32_t sb = __shfl_sync(0xffffffffu, ci.sbytes, me);
        const bool raw = __shfl_sync(0xffffffffu, ci.raw ? 1u : 0u, me) != 0;
        if (lane == 0) {
            const uint64_t off = uint64_t(load_u32(in + size_t(g) * 4)) + before;
            const bool ok = ok_all && off + mb + sb <= payload_bytes;
            S.off = uint32_t(off);
            S.mbytes = mb;
            S.sbytes = sb;
            S.raw = raw;
            S.bad = !ok;
            if (!ok) atomicOr(A.status, ST_BAD_STREAM);
        }
    }
    __syncthreads();
    if (S.bad) return;
    const uint8_t* gsrc = payload + S.off;
    const uint32_t mbytes = S.mbytes, sbytes = S.sbytes;
    const uint32_t raw_bytes = 2 * count;
    const uint32_t blocks = count / 16;
    bool bad = false;
    // stage the chunk's compressed magnitude bytes and its sign bytes
    uint8_t* mstage = reinterpret_cast<uint8_t*>(S.m);
    uint32_t mis_m = 0, mis_s = 0;
    if (mbytes && !S.raw) mis_m = stage_bytes(mstage, gsrc, mbytes, tid, kWzpThreads);
    if (sbytes) mis_s = stage_bytes(S.sb, gsrc + mbytes, sbytes, tid, kWzpThreads);
    if (tid < 16) {
        uint32_t sel = 0, k = 0;
        for (int b = 0; b < 4; ++b) sel |= (((tid >> b) & 1) ? k++ : 4u) << (4 * b);
        S.xsel[tid] = sel;
        sel = 0, k = 4;
        for (int b = 0; b < 4; ++b) {
            if ((tid >> b) & 1) k = k == 4 ? 0 : k + 1;
            sel |= k << (4 * b);
        }
        S.rep[tid] = sel;
    }
    if (tid >= 256) S.spread[tid - 256] = uint8_t(spread_entry(uint32_t(tid) - 256u));
    if (A.map.fast && tid < int(kChunk >> A.map.lb)) S.bbase[tid] = A.map.brick_base((first >> A.map.lb) + tid);
    __syncthreads();
    const uint8_t* src = mstage + mis_m; // compressed magnitude bytes (RZE chunks)
    const uint8_t* sgn = S.sb + mis_s;

    if (mbytes == 0) {
        // nothing stored: every magnitude is zero
    } else if (S.raw) {
        for (int i = tid; i < int(kChunk); i += kWzpThreads)
            S.m[i] = i < int(count) ? uint16_t(gsrc[2 * i] | (gsrc[2 * i + 1] << 8)) : 0;
    } else {
        // ---- undo repetition elimination from the back of the stream:
        // levels 3 to 1 (4, 32 and 256 bytes) by warp 0
        const uint32_t* sw = reinterpret_cast<const uint32_t*>(mstage);
        if (warp == 0) {
            uint32_t pos = mbytes - 4;
            const uint32_t mark = uint32_t(src[pos]) | (uint32_t(src[pos + 1]) << 8) | (uint32_t(src[pos + 2]) << 16) |
                                  (uint32_t(src[pos + 3]) << 24);
            uint32_t cnt = __popc(mark);
            bool under = cnt > pos;
            uint32_t base = under ? 0 : pos - cnt;
            const uint32_t rank = __popc(mark & ((2u << lane) - 1u)); // inclusive (lane 31 ok: 2u<<31 == 0)
            const uint32_t r = lane == 31 ? cnt : rank;
            uint32_t v = 0; // the lane's byte of level 2
            if (!under && r) v = src[base + r - 1];
            if (!under && ((mark >> lane) & 1u)) {
                const uint32_t prev = r > 1 ? src[base + r - 2] : 0;
                if (v == prev) bad = true;
            }
            bad |= under;
            // level 1: eight entries per lane
            pos = base;
            const uint32_t mine = __popc(v), inc = warp_incl_scan(mine), ex = inc - mine;
            cnt = __shfl_sync(0xffffffffu, inc, 31);
            under = cnt > pos;
            base = under ? 0 : pos - cnt;
            bad |= under;
            const uint32_t prev = ex ? src[base + ex - 1] : 0u;
            const uint32_t a = repeat_word(sw, mis_m + base + ex, v & 15u, prev, S.rep, bad);
            const uint32_t b = repeat_word(sw, mis_m + base + ex + __popc(v & 15u), v >> 4, a >> 24, S.rep, bad);
            reinterpret_cast<uint2*>(S.lv)[lane] = make_uint2(a, b);
            if (lane == 0) S.pos = base;
        }
        __syncthreads();
        uint32_t pos = S.pos;
        // level 0 (2048 bytes): four entries per thread, which are the bitmap
        // word of the thread's 32 plane bytes
        uint32_t bits;
        {
            const uint32_t mask = (uint32_t(S.lv[tid >> 1]) >> (4 * (tid & 1))) & 15u;
            uint32_t cnt;
            const uint32_t ex = block_excl_scan1<kWzpThreads>(__popc(mask), S.tmp1[0], cnt);
            const bool under = cnt > pos;
            const uint32_t base = under ? 0 : pos - cnt;
            bad |= under;
            bits = repeat_word(sw, mis_m + base + ex, mask, ex ? src[base + ex - 1] : 0u, S.rep, bad);
            pos = base;
        }
        // nonzero bytes: 32 per thread
        {
            uint32_t cnt;
            const uint32_t ex = block_excl_scan1<kWzpThreads>(__popc(bits), S.tmp1[1], cnt);
            if (cnt == 0 || cnt != pos) bad = true;
            const uint32_t b0 = tid * 32;
            // bitmap beyond the chunk's bytes must be empty
            if (b0 + 32 > raw_bytes) {
                const uint32_t keep = b0 >= raw_bytes ? 0u : (raw_bytes - b0 >= 32 ? 32u : raw_bytes - b0);
                const uint32_t allowed = keep == 32 ? 0xffffffffu : ((1u << keep) - 1u);
                if (bits & ~allowed) bad = true;
            }
            // spread the next popc(mask) stream bytes over each word's set
            // bytes; every one of them must be nonzero (all lie inside the
            // stream when the counts agree). Empty planes pass warp by warp.
            uint32_t words[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (__any_sync(0xffffffffu, bits)) {
                uint32_t b = mis_m + ex;
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    const uint32_t m4 = (bits >> (4 * w)) & 15u, wi = b >> 2;
                    words[w] = __byte_perm(__funnelshift_r(sw[wi], sw[wi + 1], 8 * (b & 3u)), 0u, S.xsel[m4]);
                    b += __popc(m4);
                }
                if (nonzero_mask(words) != bits) bad = true;
            }
            // full chunks write the padded layout (plane t / 32 at pitch
            // kEncPitch) straight away; a partial chunk writes the natural one
            const uint32_t pad = blocks == kChunk / 16 ? 4 * (kEncPitch - kChunk / 32) * (uint32_t(tid) >> 5) : 0u;
            uint4* out = reinterpret_cast<uint4*>(S.planes + b0 + pad);
            out[0] = make_uint4(words[0], words[1], words[2], words[3]);
            out[1] = make_uint4(words[4], words[5], words[6], words[7]);
        }
    }
    __syncthreads();

    // ---- one thread per 16-sample block: magnitudes from its 16 bit planes
    // (one transpose) or the verbatim ones, nonzero ranks by one block scan,
    // signs spread from the sign stream
    const uint32_t t = uint32_t(tid);
    uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint32_t zm = 0; // bit j: magnitude j is not zero
    if (16 * t < count && mbytes != 0) {
        if (!S.raw && t < blocks) {
            const uint16_t* pl = reinterpret_cast<const uint16_t*>(S.planes);
            const uint32_t stride = blocks == kChunk / 16 ? 2 * kEncPitch : blocks;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                w[i] = uint32_t(pl[2 * i * stride + t]) | (uint32_t(pl[(2 * i + 1) * stride + t]) << 16);
            zm = planes_nonzero(w);
            if (zm) bit_transpose16(w);
        } else {
            // a verbatim chunk, or the last count % 16 magnitudes of a partial
            // one, verbatim behind its planes
            const uint16_t* sm = S.raw ? S.m : reinterpret_cast<const uint16_t*>(S.planes);
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j)
                if (16 * t + j < count) {
                    const uint32_t m = sm[16 * t + j];
                    w[j >> 1] |= m << (16 * (j & 1u));
                    zm |= uint32_t(m != 0) << j;
                }
        }
    }
    const uint32_t cnt = __popc(zm);
    uint32_t nnz;
    const uint32_t base = block_excl_scan1<kWzpThreads>(cnt, S.tmp1[2], nnz);
    if (mbytes != 0) {
        if (nnz == 0 || (nnz + 7) / 8 != sbytes) bad = true;
        else if ((nnz & 7) && (sgn[sbytes - 1] >> (nnz & 7))) bad = true;
    }
    uint32_t nm = 0;
    if (cnt && !bad) {
        const uint32_t by = base >> 3;
        const uint32_t bits = uint32_t(sgn[by]) | (uint32_t(sgn[by + 1]) << 8) | (uint32_t(sgn[by + 2]) << 16);
        nm = expand16(bits >> (base & 7u), zm, S.spread);
    }
    if (bad) atomicOr(A.status, ST_BAD_STREAM);
    if (blockwise) {
        // whole bricks: the dequantised block as four 16-byte rows
        if (t < blocks) {
            const uint32_t brick = S.bbase[(t << 4) >> A.map.lb];
            if (A.map.bz == 16) store_block<T, true>(A.map, A.coeff, brick, t, w, nm, q);
            else store_block<T, false>(A.map, A.coeff, brick, t, w, nm, q);
        }
        return;
    }
    // ---- edge bricks: 32 consecutive magnitudes per warp step (their samples
    // share rows), each scattered to its row-major place
    uint4* dm = reinterpret_cast<uint4*>(S.m + 16 * t);
    dm[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dm[1] = make_uint4(w[4], w[5], w[6], w[7]);
    reinterpret_cast<uint16_t*>(S.nsign)[t] = uint16_t(nm);
    __syncthreads();
#pragma unroll 4
    for (uint32_t e = tid; e < count; e += kWzpThreads) {
        const T mag = Lift<T>::mul(T(uint32_t(S.m[e])), q);
        A.coeff[A.map.rowmajor(first + e)] = ((S.nsign[e >> 5] >> lane) & 1u) ? -mag : mag;
    }
}

} // namespace wb
