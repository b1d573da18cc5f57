// Inverse dyadic level of a float field (synthesis Z, X, Y) as a march along y.
//
// A CTA owns a strip of 32 outputs along x and one canonical Z window of 16,
// and walks the canonical Y windows of 8 of its range. A step stages the four
// new coefficient row pairs of the window by tensor-map copies (eight parity
// boxes of 20 x 4 x 12, as in inverse.cuh), lifts them along Z and X in place
// in shared memory and hands them to the Y pass, whose threads keep the four
// row pairs that a window shares with the next one in registers. Against a
// tile of 32 x 16 x 16 that stages and lifts the y halo again for every 16
// rows (3.4 cells staged per output), a step stages 1.9 cells per output and
// lifts 1.9 along Z and 1.25 along X; the boxes of the next step land in the
// other buffer meanwhile.
//  * The strips start at 28 mod 32, so a footprint's first coefficient is a
//    multiple of 4 (the copy engine's 16-byte rule) without padding columns,
//    and box rows of 20 floats put the eight 16-byte accesses of a quarter
//    warp in distinct banks. X does not fold, so any strip origin gives the
//    same bits.
//  * Z and Y run on pairs of lines with the packed fma.rn.f32x2 / add / mul
//    (two independent correctly rounded operations per instruction, so the
//    bits are those of lift_inverse): Z on two neighbouring columns of a box,
//    Y on the planes z and z + 1 of one column.
//  * Three CTAs of 256 threads share an SM and overlap each other's barriers.
// Bound by issue and by the barriers between the passes (47-53 % of issue
// slots, DRAM 2.9 TB/s; 44 instructions per sample, 76 with the repair test).
// 512^3, finest level: 0.538 ms as tiles of 32 x 16 x 16, 0.31 ms so; with the
// repair test 0.66 and 0.47 ms; 256^3 0.075 ms as two register marches, 0.051.

#pragma once
#include "common.cuh"
#include "inverse.cuh"
#include "packed.cuh"
#include "quantize.cuh"
#include "tma.cuh"

namespace wb {

// Emitters that store at base + z * sz + y * sy + x, with the status word of
// their finiteness check (null: none).
template <class T> struct LinearDst {
    T* p;
    size_t sy, sz;
    uint32_t* status;
};
template <class Out> struct LinearOut {
    static constexpr bool value = false;
};
template <class T> struct LinearOut<StoreOut<T>> {
    static constexpr bool value = true;
    static __device__ __forceinline__ LinearDst<T> get(const StoreOut<T>& o) { return {o.dst, o.sy, o.sz, nullptr}; }
};
template <class T> struct LinearOut<FinalOut<T>> {
    static constexpr bool value = true;
    static __device__ __forceinline__ LinearDst<T> get(const FinalOut<T>& o) { return {o.dst, o.sy, o.sz, o.status}; }
};
template <class T> struct LinearOut<JobOut<T>> {
    static constexpr bool value = true;
    static __device__ __forceinline__ LinearDst<T> get(const JobOut<T>& o) {
        return {reinterpret_cast<T*>(__ldg(reinterpret_cast<const unsigned long long*>(&o.job->out))), o.sy, o.sz,
                o.status};
    }
};

struct InvMarch {
    static constexpr int UX = 32, UZ = 16, UY = 8;    // outputs of a step
    static constexpr int SHIFT = 4;                   // strip b covers x = 32 b - 4 .. 32 b + 27
    static constexpr int HX = UX / 2 + 4, HY = UY / 2, HZ = UZ / 2 + 4;
    static constexpr int BOX = HZ * HY * HX;          // floats per parity box
    static constexpr int STAGE = 8 * BOX;             // floats per step
    static constexpr int FX = 2 * HX, FY = 2 * HY, FZ = 2 * HZ;
    // + alignment, two barriers, the reflection tables
    static constexpr size_t smem = size_t(2) * STAGE * sizeof(float) + 128 + 16 + FZ * sizeof(int) + 8 * sizeof(int2);
    static_assert((BOX * sizeof(float)) % 128 == 0, "parity boxes must stay 128-byte aligned");
};

template <class Out> struct InvMarchOp {
    static constexpr int kThreads = 256, kMinBlocks = 3;
    static constexpr bool kGridConstant = true;
    struct Params {
        CUtensorMap cmap, lmap;
        InvLevel<float> lv;
        uint32_t strips, zwins; // strips of 32 x, Z windows
        uint32_t seg;           // Y windows per CTA
        Out out;
        uint32_t* status;
        uint32_t wait_bound;    // polls of a copy wait
    };
    static __device__ __forceinline__ bool run(const Params& P, uint32_t block, uint32_t);
    static __device__ __forceinline__ void acquire_maps(const Params& P) {
        tensormap_acquire(&P.cmap);
        if (P.lv.low) tensormap_acquire(&P.lmap);
    }
    static constexpr int kBarriers = 2;
    static __device__ __forceinline__ float* staged() { // two steps of eight parity boxes
        extern __shared__ __align__(128) unsigned char march_smem[];
        return reinterpret_cast<float*>(march_smem + ((128 - (smem_u32(march_smem) & 127)) & 127));
    }
    static __device__ __forceinline__ uint64_t* barriers() {
        return reinterpret_cast<uint64_t*>(staged() + 2 * InvMarch::STAGE);
    }
    template <bool Inside>
    static __device__ __forceinline__ void emit_step(const Out& out, f2 (&e)[8], f2 (&o)[8], int x, int y, int z,
                                                     bool live, int rows, int planes, int lane, f2& nonfinite);
};

// Y synthesis and emission of one step: rows y .. y + 7 of the planes z and
// z + 1 at this lane's x. Inside: every sample of the warp lies in the level.
template <class Out>
template <bool Inside>
__device__ __forceinline__ void InvMarchOp<Out>::emit_step(const Out& out, f2 (&e)[8], f2 (&o)[8], int x, int y, int z,
                                                           bool live, int rows, int planes, int lane, f2& nonfinite) {
    auto in = [&](int j, int h) { return Inside || (live && h < planes && j < rows); };
    auto row = [&](int j) { return (j & 1) ? o[2 + j / 2] : e[2 + j / 2]; };
    if constexpr (Out::kPrefetch) {
        // originals first, so their latency overlaps the lifting
        float pre[8][2];
        const float* op = out.orig + size_t(z) * out.sz + size_t(y) * out.sy + x;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            pre[j][0] = in(j, 0) ? __ldg(op) : 0.f;
            pre[j][1] = in(j, 1) ? __ldg(op + out.sz) : 0.f;
            op += out.sy;
        }
        lift_inverse2<8>(e, o);
        const size_t at = size_t(z) * out.sz + size_t(y) * out.sy;
        uint32_t mine = 0; // lane j + 8 h keeps the patched mask of row y + j, plane z + h
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float v[2];
            f2_unpack(row(j), v[0], v[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t m =
                    out.emit_row(v[h], pre[j][h], at + size_t(h) * out.sz + size_t(j) * out.sy + x, in(j, h));
                if (lane == j + 8 * h) mine = m;
            }
        }
        if (mine)
            out.put_row(int64_t(at + size_t(lane >> 3) * out.sz + size_t(lane & 7) * out.sy) + (x - lane), mine);
    } else {
        lift_inverse2<8>(e, o);
        if constexpr (LinearOut<Out>::value) {
            const LinearDst<float> d = LinearOut<Out>::get(out);
            float* q = d.p + size_t(z) * d.sz + size_t(y) * d.sy + x;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float v0, v1;
                f2_unpack(row(j), v0, v1);
                if (in(j, 0)) *q = v0;
                if (in(j, 1)) q[d.sz] = v1;
                if constexpr (Inside) {
                    nonfinite = f2_fma(row(j), 0ull, nonfinite);
                } else if (d.status) {
                    if ((in(j, 0) && !finite_bits(v0)) || (in(j, 1) && !finite_bits(v1)))
                        atomicOr(d.status, ST_NONFINITE_INPUT);
                }
                q += d.sy;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float v0, v1;
                f2_unpack(row(j), v0, v1);
                if (in(j, 0)) out(uint32_t(x), uint32_t(y + j), uint32_t(z), v0);
                if (in(j, 1)) out(uint32_t(x), uint32_t(y + j), uint32_t(z + 1), v1);
            }
        }
    }
}

template <class Out>
__device__ __forceinline__ bool InvMarchOp<Out>::run(const Params& P, uint32_t block, uint32_t) {
    using S = InvMarch;
    const InvLevel<float> lv = P.lv;
    const Out out = P.out;
    float* const stage = staged();
    uint64_t* const bar = barriers();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Dims a = lv.a;
    const uint32_t strip = block % P.strips, zw = (block / P.strips) % P.zwins, sg = block / (P.strips * P.zwins);
    const int ox = int(strip) * S::UX - S::SHIFT, oz = int(zw) * S::UZ;
    const uint32_t wins = (a.y + S::UY - 1) / S::UY;
    const int w0 = int(sg * P.seg), w1 = int(min(wins, sg * P.seg + P.seg));
    const int nw = w1 - w0; // windows; step t = 0 only primes the kept row pairs
    const int hx = int(half_len(a.x)), hy = int(half_len(a.y)), hz = int(half_len(a.z));

    // one thread: the eight boxes of step t (row pairs 4 (w0 + t) - 2 .. + 1)
    auto issue = [&](int t) {
        float* dst = stage + (t & 1) * S::STAGE;
        uint64_t* b = bar + (t & 1);
        mbar_expect_tx(b, uint32_t(S::STAGE * sizeof(float)));
        const int x0 = ox / 2 - 2, y0 = 4 * (w0 + t) - 2, z0 = oz / 2 - 2;
#pragma unroll 1
        for (int k = 0; k < 8; ++k)
            tma_load_3d(dst + k * S::BOX, (k == 0 && lv.low) ? &P.lmap : &P.cmap, x0 + ((k & 1) ? hx : 0),
                        y0 + ((k & 2) ? hy : 0), z0 + ((k & 4) ? hz : 0), b);
    };
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        fence_barrier_init();
        issue(0);
        issue(1);
    }
    __syncthreads(); // the barriers are initialised before any thread polls them

    // Reflections at the level's x and z ends stay inside the footprint. Along
    // z the Z pass reads slot z of a column from ztab[z] (its offset in the
    // buffer for the column's box pair); along x, up to four cells per side of
    // every row are copied after the Z pass (xtab: cell and its source).
    const int fx_lo = min(S::FX, max(0, 4 - ox)), fx_hi = min(S::FX, int(a.x) - ox + 4);
    const int fx_l = min(4, fx_lo), fx_r = min(4, S::FX - fx_hi);
    const int fz_lo = oz < 4 ? 4 - oz : 0, fz_hi = min(S::FZ, int(a.z) - oz + 4);
    const bool edge_x = fx_l | fx_r, edge_z = fz_lo || fz_hi < S::FZ;
    int* const ztab = reinterpret_cast<int*>(bar + 2); // FZ entries
    int2* const xtab = reinterpret_cast<int2*>(ztab + S::FZ); // 8 entries
    if (tid < S::FZ) {
        int f = int(mirror(int64_t(oz) + tid - 4, a.z)) - (oz - 4);
        f = min(max(f, 0), S::FZ - 1); // slots past the needed halo: any
        ztab[tid] = (f & 1) * 4 * S::BOX + (f >> 1) * S::HY * S::HX;
    } else if (tid >= 32 && tid < 40) {
        const int k = tid - 32;
        const int f = k < 4 ? fx_lo - 4 + k : fx_hi + k - 4;
        const bool used = k < 4 ? f >= 0 && fx_l : f < S::FX;
        int m = used ? int(mirror(int64_t(ox) + f - 4, a.x)) - (ox - 4) : 0;
        m = min(max(m, 0), S::FX - 1);
        xtab[k] = used ? make_int2((f & 1) * S::BOX + (f >> 1), (m & 1) * S::BOX + (m >> 1)) : make_int2(-1, 0);
    }
    __syncthreads();

    f2 ke[4], ko[4]; // the Y pass's kept row pairs (lifted along Z and X)
    f2 nonfinite = 0; // interior samples times zero, summed: NaN once one was not finite
#pragma unroll 1
    for (int t = 0; t <= nw; ++t) {
        float* const B = stage + (t & 1) * S::STAGE;
        const int r0 = 8 * (w0 + t) - 4; // first spatial row of the step's pairs
        // the emitter's own operands (the originals, for repairs): one thread
        // per row of the step's outputs asks L2 for its line
        if constexpr (Out::kPrefetch) {
            if (t > 0 && tid < S::UY * S::UZ) {
                const uint32_t gy = uint32_t(r0 - 4 + tid % S::UY), gz = uint32_t(oz + tid / S::UY);
                if (gy < a.y && gz < a.z) out.warm(min(uint32_t(ox + S::SHIFT), a.x - 1), gy, gz); // most of the row
            }
        }
        const bool landed = mbar_wait(bar + (t & 1), uint32_t(t >> 1) & 1u, P.wait_bound);
        // ---- rows outside the level, from their reflections (coefficient
        // mapped): copied from the staged rows when the reflected row is among
        // them, else loaded; cells inside the level along x and z only
        const int fy_lo = max(0, -r0), fy_hi = max(0, min(S::FY, int(a.y) - r0)),
                  fy_end = max(fy_hi, min(S::FY, int(a.y) + 4 - r0));
        if (fy_lo || fy_hi < fy_end) {
            auto cell = [&](int fx, int fy, int fz) -> float* {
                return B + ((fz & 1) * 4 + (fy & 1) * 2 + (fx & 1)) * S::BOX +
                       ((fz >> 1) * S::HY + (fy >> 1)) * S::HX + (fx >> 1);
            };
            const int nx_in = fx_hi - fx_lo, nz_in = fz_hi - fz_lo, ny_out = fy_lo + (fy_end - fy_hi);
            for (int i = tid; i < nx_in * nz_in * ny_out; i += kThreads) {
                const int row = i / nx_in, fx = fx_lo + i - row * nx_in, ks = row / nz_in,
                          fz = fz_lo + row - ks * nz_in, fy = ks < fy_lo ? ks : fy_hi + (ks - fy_lo);
                const uint32_t my = mirror(int64_t(r0) + fy, a.y);
                const int gy = int(my) - r0;
                float v;
                if (gy >= 0 && gy < S::FY) {
                    v = *cell(fx, gy, fz);
                } else {
                    const uint32_t cx = split_of(uint32_t(ox + fx - 4), a.x), cy = split_of(my, a.y),
                                   cz = split_of(uint32_t(oz + fz - 4), a.z);
                    if (lv.low && cx < lv.lo.x && cy < lv.lo.y && cz < lv.lo.z)
                        v = lv.low[(size_t(cz) * lv.lo.y + cy) * lv.lo.x + cx];
                    else
                        v = lv.base[size_t(cz) * lv.sz + size_t(cy) * lv.sy + cx];
                }
                *cell(fx, fy, fz) = v;
            }
            __syncthreads();
        }
        // ---- Z: the canonical window of every footprint column, two
        // neighbouring columns of a box per thread, in place
        constexpr int ZS = S::HY * S::HX; // z-slot stride inside a box
        constexpr int CP = S::HX / 2;     // column pairs of a box row
        if (tid < 4 * S::HY * CP) {
            const int cp = tid % CP, row = tid / CP; // row = k + 4 * (x parity + 2 * y parity)
            float* pe = B + (row >> 2) * S::BOX + (row & 3) * S::HX + 2 * cp;
            float* po = pe + 4 * S::BOX;
            f2 e[S::HZ], o[S::HZ];
            if (edge_z) {
#pragma unroll
                for (int j = 0; j < S::HZ; ++j) {
                    e[j] = *reinterpret_cast<const f2*>(pe + ztab[2 * j]);
                    o[j] = *reinterpret_cast<const f2*>(pe + ztab[2 * j + 1]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < S::HZ; ++j) {
                    e[j] = *reinterpret_cast<const f2*>(pe + j * ZS);
                    o[j] = *reinterpret_cast<const f2*>(po + j * ZS);
                }
            }
            lift_inverse2<S::HZ>(e, o);
#pragma unroll
            for (int j = 2; j < S::HZ - 2; ++j) {
                *reinterpret_cast<f2*>(pe + j * ZS) = e[j];
                *reinterpret_cast<f2*>(po + j * ZS) = o[j];
            }
        }
        fence_proxy_async(); // this thread's accesses to the other buffer precede the copies into it
        if (!__syncthreads_and(landed)) {
            // a copy that did not land: the block stops as a whole, with no
            // further copy issued. Those in flight (this step's, and at the
            // start the next one's) get as long again to end.
            if (tid == 0) {
                atomicOr(P.status, ST_WAIT_TIMEOUT);
                mbar_wait(bar + (t & 1), uint32_t(t >> 1) & 1u, kWaitBound);
                if (t == 0) mbar_wait(bar + 1, 0, kWaitBound);
            }
            return false;
        }
        // every thread has left the previous step: its buffer takes the next one
        if (tid == 0 && t > 0 && t < nw) issue(t + 1);
        if (edge_x) { // both sides of one Z output row per thread pair
            float* r = B + (tid & 3) * 2 * S::BOX + 2 * S::HY * S::HX + ((tid >> 2) & 31) * S::HX;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int2 x = xtab[4 * (tid >> 7) + k];
                if (x.x >= 0) r[x.x] = r[x.y];
            }
            __syncthreads();
        }
        // ---- X: windows of 16 outputs, both windows of a row in one warp;
        // a warp takes 16 rows of one (y, z) parity
        {
            constexpr int PX = 12;
            const int row = 2 * S::HY + 16 * (warp & 1) + (lane & 15), win = lane >> 4; // rows of z slots 2 .. 9
            float* re = B + (warp >> 1) * 2 * S::BOX + row * S::HX + 8 * win;
            float* ro = re + S::BOX;
            float e[PX], o[PX];
#pragma unroll
            for (int q = 0; q < PX / 4; ++q) {
                const float4 ve = reinterpret_cast<const float4*>(re)[q], vo = reinterpret_cast<const float4*>(ro)[q];
                e[4 * q] = ve.x, e[4 * q + 1] = ve.y, e[4 * q + 2] = ve.z, e[4 * q + 3] = ve.w;
                o[4 * q] = vo.x, o[4 * q + 1] = vo.y, o[4 * q + 2] = vo.z, o[4 * q + 3] = vo.w;
            }
            lift_inverse<float, PX, false>(e, o);
            __syncwarp(); // the row's other window has read its cells
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float* r = h ? ro : re;
                const float* v = h ? o : e;
                *reinterpret_cast<float2*>(r + 2) = make_float2(v[2], v[3]);
                *reinterpret_cast<float4*>(r + 4) = make_float4(v[4], v[5], v[6], v[7]);
                *reinterpret_cast<float2*>(r + 8) = make_float2(v[8], v[9]);
            }
        }
        __syncthreads();
        // ---- Y: planes z and z + 1 of one column per thread, the canonical
        // window of 8 from registers
        const float* c = B + (lane & 1) * S::BOX + (2 + warp) * ZS + 2 + (lane >> 1);
        f2 e[8], o[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            e[4 + k] = f2_pack(c[k * S::HX], c[4 * S::BOX + k * S::HX]);
            o[4 + k] = f2_pack(c[2 * S::BOX + k * S::HX], c[6 * S::BOX + k * S::HX]);
        }
        if (t > 0) {
            const int x = ox + lane, z = oz + 2 * warp, y = r0 - 4;
            const bool live = x >= 0 && x < int(a.x);
            const int rows = min(8, int(a.y) - y), planes = int(a.z) - z;
#pragma unroll
            for (int k = 0; k < 4; ++k) e[k] = ke[k], o[k] = ko[k];
#pragma unroll
            for (int k = 0; k < 4; ++k) ke[k] = e[4 + k], ko[k] = o[4 + k];
            // a step wholly inside the level needs no predicate per sample
            // (decided for the whole warp)
            if (ox >= 0 && ox + S::UX <= int(a.x) && rows == 8 && planes >= 2)
                emit_step<true>(out, e, o, x, y, z, true, 8, 2, lane, nonfinite);
            else
                emit_step<false>(out, e, o, x, y, z, live, rows, planes, lane, nonfinite);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) ke[k] = e[4 + k], ko[k] = o[4 + k];
        }
    }
    if constexpr (LinearOut<Out>::value) {
        const LinearDst<float> d = LinearOut<Out>::get(out);
        float n0, n1;
        f2_unpack(nonfinite, n0, n1);
        if (d.status && __any_sync(0xffffffffu, !(n0 == 0.f && n1 == 0.f)) && lane == 0)
            atomicOr(d.status, ST_NONFINITE_INPUT);
    }
    return true;
}

} // namespace wb
