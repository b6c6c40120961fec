// Pair-distance histogram kernel of the form-factor managers: the O(N^2) stage of the Debye hot path
// with one shared-memory atomic per pair.
//
// Replaces the manager lambdas of HistogramManagerMTFFAvg.cpp:214-302, HistogramManagerMTFFExplicit.cpp:
// 233-300 and HistogramManagerMTFFGrid.cpp:68-159 with their SIMD evaluators (CompactCoordinatesXYZFF.h).
//
// What bounds the stage: FP32 and issue slots (the reference's rounding order fixes 17 FP32 operations
// per pair) and the shared-memory pipe (a shared atomic to random bins costs about four wavefronts, the
// bins of 32 lanes being random modulo the 32 banks).  So:
//   * FP32 operations go in pairs through the packed f32x2 instructions (add/mul/fma.rn.f32x2: the same
//     roundings, half the issue slots): a packed operation covers two consecutive inner points, which
//     are staged as quads {x x x x}{y y y y}{z z z z}{i i i i}; the outer point's coordinates are held
//     duplicated in registers;
//   * a pair's count and its 16-bit in-bin offset (pair_residual) are ONE 32-bit shared atomic: the word of
//     (row, bin) holds 2^23 * count + sum of offsets.  The added value 2^23 + offset is the bit pattern
//     of one FMA: coordinates are scaled by 2^-23 when staged, so that r * scale * 2^-149 + (2^23 + 2^15) *
//     2^-149 rounds to a multiple of 2^-149, whose bit pattern is that integer;
//   * a word holds 128 pairs for certain (about 250 in practice), so the words are moved to u16 counts
//     and u32 offset sums every segment of pairs, and every segment is checked: the count fields must
//     add up to the pairs evaluated.  That check is exact.  With C carries out of offset fields and W
//     words that wrapped, the fields add up to N + C - 512 W; a segment has N < 65,536 pairs, hence C <
//     2^16 N / 2^23 < 512, so the sum is N only if C = W = 0.  A segment that fails is taken back (its
//     additions repeated, the same words subtracted) and evaluated again at half the length, or, at the
//     smallest one, with two atomics per pair (count, offset).  The length follows the fullest word, scaled to
//     a full segment (140 to 200 pairs; 110 to 170 measured up to 2 % slower), and a tile is cut into segments of
//     about equal length (a short last one costs a whole drain: 12,000 atoms of one type, 0.25 A, 148 -> 131 us);
//   * with few bins a word is full after few pairs.  Jobs then keep several copies of their words, the lanes of
//     a warp in turn, until a segment lasts 24,576 pairs (pack_copies; 8,192 and 16,384 measured up to 12 %
//     slower at 0.5 A bins, 32,768 up to 2 % at 0.25 A).  Whole calls without and with copies: 12,000 atoms of
//     one type at 1 A 193 -> 143 us, at 2 A 344 -> 154; 25,000 atoms of four types at 1 A 564 -> 463, at 4 A
//     1,573 -> 548; of 13 types at 2 A, whose water pairs have a word per bin, 4,162 -> 537;
//   * rows are the outer point's type only: the inner points of a job share one type, so a CTA keeps T
//     rows instead of T * T and no pair adds a row offset.
// All accumulations are integer, so results do not depend on scheduling; counts and offsets are those of
// pairhist.cu bit for bit (the same roundings up to the power-of-two scale).
//
// Measured on the B200: the inner loop alone (405 bins) 1,702 Gpair/s with the clamp and 1,815 without against
// 1,171 for the scalar two-atomic loop of pairhist.cu; launches of 50,000 atoms + 10,000 waters at 0.25 A bins 1,406
// Gpair/s (16.9 warp instructions per 32 pairs, FMA pipe 67 %, shared-memory wavefronts 76 % of peak) against 1,040,
// of a 264,000-point shell at 3,092 bins 1,286 against 943.  Per-segment drains and checks take about 15 %.
#include <algorithm>
#include <type_traits>

#include "pairhist.cuh"
#include "pairpack.cuh"

namespace ausaxs_b200 {

namespace {

using u64 = unsigned long long;

constexpr unsigned kWaitLimit = 1u << 24;
constexpr u64 kWaitTimedOut = 1ull << 62;
constexpr uint32_t kOffsetMask = (1u << kPackCountShift) - 1u;

__device__ __forceinline__ u64 pack2(float a, float b) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(u64 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// A rounded product that a following sum must not absorb: the assembler contracts mul.rn.f32x2 with
// add.rn.f32x2 into one fma (seen on squared distances one ulp off), but not an fma with a zero
// addend, which is the same value for products that are not negative.  pack_check_kernel makes sure of it: with
// an assembler that folds these too the two-atomic kernel takes over.
__device__ __forceinline__ u64 product2(u64 a, u64 b) { return fma2(a, b, 0ull); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void shared_red_add(uint32_t addr, uint32_t v) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void mbar_init(u64* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(u64* bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, u64* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ bool mbar_wait(u64* bar, unsigned parity) {
    const uint32_t a = smem_addr(bar);
    for (unsigned it = 0; it < kWaitLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

struct Tile {
    int ti;      // outer tile; -1: no tile left
    int j0, jn;  // inner points [j0, j0 + jn)
    int job;
};

// One staged quad of inner points: negated scaled coordinates, and the points' indices.
struct Quad {
    ulonglong2 x, y, z;
    int4 i;
};

// The constants of a job's inner loop (packed pairs of equal values).
struct Consts {
    u64 iw, mg, nmg, nc, sc, off;
    float dmax;  // scaled distance of the overflow column
};

__device__ __forceinline__ Consts constants(float inv_w, float c, float scale, int nb) {
    constexpr float S = 1.0f / 8388608.0f;
    const float iw = inv_w * 8388608.0f, nc = -c * S, sc = scale * 0x1p-126f;
    const float off = __uint_as_float((1u << kPackCountShift) + static_cast<uint32_t>(kResBias));
    Consts K;
    K.iw = pack2(iw, iw);
    K.mg = pack2(kMagic, kMagic);
    K.nmg = pack2(-kMagic, -kMagic);
    K.nc = pack2(nc, nc);
    K.sc = pack2(sc, sc);
    K.off = pack2(off, off);
    K.dmax = static_cast<float>(nb) * c * S;
    return K;
}

// Two inner points (negated) against an outer point (held twice): the bins' magic numbers and the values that
// are added.
template <int NR, bool DSUM, bool CLAMP>
__device__ __forceinline__ void pair_values(u64 ox, u64 oy, u64 oz, u64 bx, u64 by, u64 bz, const Consts& K, float& x0, float& x1,
                                            uint32_t& v0, uint32_t& v1) {
    const u64 dx = add2(ox, bx), dy = add2(oy, by), dz = add2(oz, bz);
    const u64 s = add2(add2(product2(dx, dx), product2(dy, dy)), product2(dz, dz));
    // d = sqrt(s) as pair_sqrt_scaled
    float s0, s1, y0, y1;
    unpack2(s, s0, s1);
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(fmaxf(s0, 1e-36f)));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(fmaxf(s1, 1e-36f)));
    const u64 d0 = mul2(s, pack2(y0, y1));
    const u64 h = pack2(__int_as_float(__float_as_int(y0) - 0x00800000), __int_as_float(__float_as_int(y1) - 0x00800000));
    float d00, d01;
    unpack2(d0, d00, d01);
    u64 d = fma2(pack2(__fmaf_rn(-d00, d00, s0), __fmaf_rn(-d01, d01, s1)), h, d0);
    // distances past the last bin (also NaN and inf) become that of the overflow column's centre,
    // so that every added value is 2^23 + an offset below 2^16.  Launches whose bins cover every
    // distance (PackLaunch::covered) leave that out: one instruction of 17 per pair.
    if (CLAMP) {
        float d1v, d0v;
        unpack2(d, d0v, d1v);
        d = pack2(fminf(d0v, K.dmax), fminf(d1v, K.dmax));
    }
    // bin by the magic number; a power-of-two width (NR == 2) fuses the product
    const u64 xm = NR == 2 ? fma2(d, K.iw, K.mg) : add2(product2(d, K.iw), K.mg);
    unpack2(xm, x0, x1);
    v0 = v1 = 1u << kPackCountShift;
    if (DSUM) {
        const u64 r = fma2(add2(xm, K.nmg), K.nc, d);
        float t0, t1;
        unpack2(fma2(r, K.sc, K.off), t0, t1);
        v0 = __float_as_uint(t0);
        v1 = __float_as_uint(t1);
    }
}

// Four inner points (one quad) against the thread's R outer points.  MASK: only inner positions in
// [p[k], kt) of outer point k are valid; n counts the valid pairs.
template <bool MASK, int R, int NR, bool DSUM, bool CLAMP>
__device__ __forceinline__ void quad_pairs(const Quad* __restrict__ q, int k0, const u64 (&ox)[R], const u64 (&oy)[R],
                                           const u64 (&oz)[R], const uint32_t (&caddr)[R], const int (&p)[R], int kt,
                                           const Consts& K, int& n) {
    const ulonglong2 X = q->x, Y = q->y, Z = q->z;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const u64 bx = u ? X.y : X.x, by = u ? Y.y : Y.x, bz = u ? Z.y : Z.x;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            float x0, x1;
            uint32_t v0, v1;
            pair_values<NR, DSUM, CLAMP>(ox[k], oy[k], oz[k], bx, by, bz, K, x0, x1, v0, v1);
            const uint32_t a0 = caddr[k] + (__float_as_uint(x0) << 2), a1 = caddr[k] + (__float_as_uint(x1) << 2);
            if (MASK) {
                const int j = k0 + 2 * u;
                if (j >= p[k] && j < kt) {
                    shared_red_add(a0, v0);
                    ++n;
                }
                if (j + 1 >= p[k] && j + 1 < kt) {
                    shared_red_add(a1, v1);
                    ++n;
                }
            } else {
                shared_red_add(a0, v0);
                shared_red_add(a1, v1);
            }
        }
    }
}

// Inner positions [k0, k1) one at a time with two atomics per pair (count, offset): the scalar-tail
// partners (contracted form, ties away from zero) and the segments whose words could not hold them.
template <int R, bool DSUM>
__device__ __forceinline__ void slow_pairs(const Quad* s_q, int k0, int k1, const u64 (&ox)[R], const u64 (&oy)[R],
                                           const u64 (&oz)[R], const uint32_t (&row0)[R], uint32_t cnt_addr, uint32_t dacc_addr,
                                           const int (&p)[R], const int (&ts)[R], int b_base, float inv_w, float c, float scale,
                                           int nb) {
    const float limit = pair_bin_limit(nb);
    for (int k = k0; k < k1; ++k) {
        const float* f = reinterpret_cast<const float*>(s_q + (k >> 2)) + (k & 3);
        const float bx = f[0], by = f[4], bz = f[8];
        const int gj = b_base + __float_as_int(f[12]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (k < p[r]) continue;
            float ax, ay, az, same;
            unpack2(ox[r], ax, same);
            unpack2(oy[r], ay, same);
            unpack2(oz[r], az, same);
            const float dx = __fadd_rn(ax, bx), dy = __fadd_rn(ay, by), dz = __fadd_rn(az, bz);
            const bool tail = gj >= ts[r];
            const float s = tail ? __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)))
                                 : __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
            const float d = __fmul_rn(pair_sqrt_scaled(s), 8388608.0f);
            const float x = __fmul_rn(d, inv_w);
            float xm = fminf(__fadd_rn(x, kMagic), limit);
            if (tail && __fsub_rn(x, __fsub_rn(xm, kMagic)) == 0.5f) xm = fminf(__fadd_rn(xm, 1.0f), limit);
            const uint32_t bin = static_cast<uint32_t>(__float_as_int(xm) - kMagicBits);
            const uint32_t cell = row0[r] + bin;
            shared_red_add(cnt_addr + (cell >> 1) * 4u, 1u << ((cell & 1u) * 16u));
            // the overflow column's offsets are of no use (and not bounded)
            if (DSUM && bin < static_cast<uint32_t>(nb)) {
                const float t = __fmaf_rn(__fmaf_rn(-__fsub_rn(xm, kMagic), c, d), scale, kMagic);
                shared_red_add(dacc_addr + bin * 4u, static_cast<uint32_t>(__float_as_int(t) - kMagicBits + kResBias));
            }
        }
    }
}

constexpr int kRoom = 511;  // 511 x 2^23 < 2^32 and 511 x 128 < 2^16

// Shared memory of a CTA: packed words [rows][copies][pad], u32 offset sums [group_sums][pad], u16 counts
// [group_rows][pad], two buffers of tile_j inner points; pad = bins + 1 (the overflow column) rounded up to
// whole quads of bins, an odd number of them: where copies lie a multiple of 32 words apart the lanes of a
// warp, each on its copy, meet in the bank of their bin (50,000 atoms of one type at 4 A, 28 bins: 3,031 us with 32
// words, 1,549 with 36).  Counts and offset sums go to the global accumulators when the CTA moves to another
// group or when they could wrap (kRoom); 16-bit counts keep two CTAs on an SM at the 3,100 bins of a 300 A
// shell.
__host__ __device__ inline int pack_pad(int bins) { return ((bins + 4) & ~3) | 4; }

// Resident CTAs: 16 to 20 warps per SM already reach the pipes' rates (the inner loop alone: 1,688 Gpair/s
// at 16 warps, 1,702 at 32), so up to 102 registers per thread buy a loop without spills.
constexpr int pack_min_blocks(int threads) { return threads >= 512 ? 1 : 640 / threads; }

template <int NT, int G, int NR, bool DSUM, bool CLAMP>
__global__ void __launch_bounds__(NT, pack_min_blocks(NT)) pack_kernel(const PackLaunch L) {
    constexpr int R = 2;
    constexpr int NTG = NT / G;
    constexpr int OUT = NTG * R;
    constexpr int kMaxLen = kPackMaxPairs / (NT * R * 4);  // quads per group of a segment
    static_assert(kMaxLen >= 1, "a segment is at least one quad per group");
    static_assert(kPackMaxTileJ / 4 <= NT, "a thread stages at most one quad");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ u64 s_bar[2];
    __shared__ Tile s_tile[2];
    __shared__ PackJob s_job[2];
    __shared__ int s_diff[2];
    __shared__ unsigned s_fill[2];
    const int pad = pack_pad(L.bins);
    const int tid = threadIdx.x;
    const int group = tid / NTG, tg = tid % NTG, lane = tid & 31;
    uint32_t* const s_pk = reinterpret_cast<uint32_t*>(smem);
    uint32_t* const s_sums = s_pk + L.rows * pad;
    uint16_t* const s_cnts = reinterpret_cast<uint16_t*>(s_sums + L.group_sums * pad);
    const int rows2 = (L.group_rows + 1) & ~1;  // the staging buffers start on 16 bytes
    Quad* const stage0 = reinterpret_cast<Quad*>(s_cnts + rows2 * pad);
    const int stage_quads = L.tile_j / 4;

    // Warp 0: the next tile that holds pairs, its job and the copy of its inner points, into buffer b.  The
    // lanes search the job table together (two rounds cover 1,024 jobs) and copy the job's 8 words.
    auto fetch = [&](int b, long long g) {
        Tile t{-1, 0, 0, 0};
        while (g < L.total_tiles) {
            int lo = 0, n = L.n_jobs;
            while (n > 1) {
                const int step = (n + 31) / 32;
                const int at = lo + lane * step;
                const unsigned le = __ballot_sync(0xffffffffu, lane * step < n && L.jobs[min(at, L.n_jobs - 1)].tile_begin <= g);
                const int hit = 31 - __clz(le);
                lo += hit * step;
                n = min(step, n - hit * step);
            }
            if (lane < static_cast<int>(sizeof(PackJob) / 16))
                reinterpret_cast<uint4*>(&s_job[b])[lane] = reinterpret_cast<const uint4*>(L.jobs + lo)[lane];
            __syncwarp();
            const PackJob& J = s_job[b];
            const long long local = g - J.tile_begin;
            const int ti = static_cast<int>(local / J.tiles_j), tj = static_cast<int>(local - static_cast<long long>(ti) * J.tiles_j);
            // self jobs: the inner points of larger index than the tile's first outer point
            const int base = !J.self ? 0 : (J.indexed ? J.pre[ti * (OUT / kPackPre)] : ti * OUT);
            const int j0 = base + tj * L.tile_j;
            if (j0 < J.nb) {
                t = Tile{ti, j0, min(L.tile_j, J.nb - j0), lo};
                if (lane == 0) bulk_load(stage0 + b * stage_quads, J.B + j0, static_cast<unsigned>(t.jn) * 16u, &s_bar[b]);
                break;
            }
            __syncwarp();  // every lane has read the job before the next one replaces it
            if (lane == 0) g = static_cast<long long>(gridDim.x) + static_cast<long long>(atomicAdd(L.tile_counter, 1ull));
            g = __shfl_sync(0xffffffffu, g, 0);
        }
        if (lane == 0) s_tile[b] = t;
    };
    if (tid < 32) {
        if (lane == 0) {
            mbar_init(&s_bar[0], 1);
            mbar_init(&s_bar[1], 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            s_diff[0] = s_diff[1] = 0;
            s_fill[0] = s_fill[1] = 0;
        }
        __syncwarp();
        fetch(0, blockIdx.x);  // the counter hands out the tiles after the first gridDim.x
    } else {
        const int words = (L.rows * 2 + L.group_sums * 2 + rows2) * pad / 8;
        for (int k = tid - 32; k < words; k += NT - 32) reinterpret_cast<uint4*>(smem)[k] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();

    int cur = -1, cur_group = -1, taken = 0;
    int grp_out = 0, grp_rows = 0, grp_sums = 0, grp_bins = 0, grp_mult = 1;
    int len = 1;         // quads per group of a segment
    int copies = 1;      // of the job's packed words
    int slow_left = 0;   // segments still to be evaluated with two atomics per pair
    int room = kRoom;    // what the u32 offset sums (in 2^23) and u16 counts (in 128) still hold for certain
    int buf = 0, ph = 0;
    unsigned phases = 0u;
    bool failed = false;

    // the group's counts and offset sums -> the global accumulators (coalesced, 32 bins of a row per step)
    auto flush = [&]() {
        __syncthreads();
        const int steps = grp_bins / 32 + 1;  // the overflow column too
        for (int u = tid >> 5; u < (grp_rows + (DSUM ? grp_sums : 0)) * steps; u += NT / 32) {
            const int r = u / steps, b = (u - r * steps) * 32 + lane;
            if (b > grp_bins) continue;
            uint32_t v;
            if (r < grp_rows) {
                v = s_cnts[r * pad + b];
                s_cnts[r * pad + b] = 0;
            } else {
                v = s_sums[(r - grp_rows) * pad + b];
                s_sums[(r - grp_rows) * pad + b] = 0;
            }
            if (v) {
                if (b < grp_bins) atomicAdd(L.out[grp_out + r] + b, static_cast<u64>(v) * grp_mult);
                else if (r < grp_rows) atomicAdd(L.overflow, static_cast<u64>(v));
            }
        }
        room = kRoom;
        __syncthreads();
    };

    while (true) {
        const Tile t = s_tile[buf];
        if (t.ti < 0) break;
        ++taken;
        // the counter's answer is used after the first segment, so its latency is hidden (one asm block: a
        // select after the atomic would wait for it here)
        u64 drawn;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "mov.u64 %0, %3;\n\t"
            "@p atom.global.add.u64 %0, [%2], 1;\n\t}"
            : "=l"(drawn)
            : "r"(static_cast<unsigned>(tid == 0 && (L.max_tiles <= 0 || taken < L.max_tiles))), "l"(L.tile_counter), "l"(L.total_tiles)
            : "memory");

        const PackJob& J = s_job[buf];
        const int rows = J.rows, nb = J.nbins;
        if (t.job != cur) {
            if (J.group != cur_group) {
                if (cur >= 0) flush();
                cur_group = J.group;
                grp_out = J.group_out;
                grp_rows = J.group_rows;
                grp_sums = J.group_sums;
                grp_bins = nb;
                grp_mult = J.mult;
            }
            len = max(1, min(kMaxLen, J.seg_pairs / (NT * R * 4)));
            copies = L.many ? J.copies : 1;  // (known without a load: a shell of 500,000 atoms 122.4 -> 121.4 ms)
            slow_left = 0;
            cur = t.job;
        }
        uint16_t* const s_cnt = s_cnts + J.cnt_row * pad;
        uint32_t* const s_dacc = s_sums + J.sum_slot * pad;

        // Outer points.  Tiles with masked pairs (self tiles that the diagonal crosses, the last outer tile)
        // give a warp consecutive points, so that whole warps drop out of the masked part; the others
        // spread a warp's lanes over the tile (neighbouring points of a chain have similar distances).
        const int i0 = t.ti * OUT;
        const bool ragged = i0 + OUT > J.na;
        const int j_first = J.indexed ? __float_as_int(J.B[t.j0].w) : t.j0;  // the tile's smallest inner index
        const int g_last = J.a_base + min(i0 + OUT, J.na) - 1;               // its largest outer index
        const bool crossed = J.self && J.b_base + j_first <= g_last;
        u64 ox[R], oy[R], oz[R];
        uint32_t caddr[R];
        int p[R], gi[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int o = ragged || crossed ? tg + k * NTG : (lane * (NTG / 32) + (tg >> 5)) + k * NTG;
            const int i = i0 + o;
            const bool on = i < J.na;
            const float4 a = on ? J.A[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            constexpr float S = 1.0f / 8388608.0f;  // 2^-23
            ox[k] = pack2(a.x * S, a.x * S);
            oy[k] = pack2(a.y * S, a.y * S);
            oz[k] = pack2(a.z * S, a.z * S);
            const int row = (rows > 1 ? __float_as_int(a.w) : 0) * copies + (lane & (copies - 1));
            caddr[k] = smem_addr(s_pk) + 4u * static_cast<uint32_t>(row * pad) - 4u * static_cast<uint32_t>(kMagicBits);
            gi[k] = J.a_base + i;
            p[k] = on ? 0 : 0x7fffffff;
        }

        const bool timed_out = !mbar_wait(&s_bar[buf], (phases >> buf) & 1u);
        phases ^= 1u << buf;
        if (__syncthreads_or(timed_out)) {
            failed = true;
            if (tid == 0) atomicOr(L.overflow, kWaitTimedOut);
            break;  // no other copy is in flight: the next tile's is issued below
        }
        // quads in place: {x y z w} x 4 -> {-x}{-y}{-z}{index}, scaled by 2^-23.  Where the order does not
        // matter (no masked pairs, none of the list's last three points, which may be scalar-tail partners and are
        // looked for from the tile's end) a quad takes points a quarter of the tile apart: a segment of quads
        // then spans four stretches of the chain, its distances more bins, and the fullest word takes longer to
        // fill.
        Quad* const s_q = stage0 + buf * stage_quads;
        {
            const int nq = (t.jn + 3) / 4;
            const bool spread = !ragged && !crossed && t.j0 + t.jn + 3 <= J.nb;
            const int first = spread ? tid : 4 * tid, step = spread ? nq : 1;
            float4 v[4];
            if (tid < nq) {
                const float4* f = reinterpret_cast<const float4*>(s_q) + first;
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = f[k * step];
            }
            if (spread) __syncthreads();
            if (tid < nq) {
                float4* const f = reinterpret_cast<float4*>(s_q + tid);
                constexpr float S = -1.0f / 8388608.0f;
                f[0] = make_float4(v[0].x * S, v[1].x * S, v[2].x * S, v[3].x * S);
                f[1] = make_float4(v[0].y * S, v[1].y * S, v[2].y * S, v[3].y * S);
                f[2] = make_float4(v[0].z * S, v[1].z * S, v[2].z * S, v[3].z * S);
                const int j = t.j0 + first;
                f[3] = J.indexed ? make_float4(v[0].w, v[1].w, v[2].w, v[3].w)
                                 : make_float4(__int_as_float(j), __int_as_float(j + step), __int_as_float(j + 2 * step),
                                               __int_as_float(j + 3 * step));
            }
        }
        __syncthreads();
        const int* const s_idx = reinterpret_cast<const int*>(s_q);
        auto index_of = [&](int k) { return s_idx[(k >> 2) * 16 + 12 + (k & 3)]; };
        auto rank_of = [&](int v) {  // inner positions with an index at most v
            int lo = 0, hi = t.jn;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (index_of(mid) <= v) lo = mid + 1;
                else hi = mid;
            }
            return lo;
        };
        // the last three indices of the full set may go through the scalar evaluator
        int kt = t.jn;
        while (kt > 0 && J.b_base + index_of(kt - 1) >= J.tail_end - 3) --kt;
        const int kq = (kt + 3) / 4;
        int mq0 = ragged ? kq : 0;  // quads before mq0 and from mq1 on hold masked pairs
        const int mq1 = kt / 4;
        if (crossed) {
            mq0 = max(mq0, min(kq, (rank_of(g_last - J.b_base) + 3) / 4));
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (p[k] == 0) p[k] = rank_of(gi[k] - J.b_base);
        }
        const int q_warp = __reduce_min_sync(0xffffffffu, min(p[0], p[1])) >> 2;  // first quad the warp needs

        // inner positions [k0, k1) with two atomics per pair; indices from tail_end on cut to whole fours of
        // a row go through the scalar evaluator
        auto slow = [&](int k0, int k1, int tail_end) {
            uint32_t row0[R];
            int ts[R];
#pragma unroll
            for (int k = 0; k < R; ++k) {
                row0[k] = (caddr[k] + 4u * static_cast<uint32_t>(kMagicBits) - smem_addr(s_pk)) / (4u * pad) / copies * pad;
                const int row_begin = J.tail_from_outer ? gi[k] + 1 : 0;
                ts[k] = tail_end == 0x7fffffff ? tail_end : tail_end - ((tail_end - row_begin) & 3);
            }
            slow_pairs<R, DSUM>(s_q, k0, k1, ox, oy, oz, row0, smem_addr(s_cnt), smem_addr(s_dacc), p, ts, J.b_base, J.inv_w, J.c,
                                J.scale, nb);
        };
        bool fetched = false, undo = false;
        for (int s0 = 0; s0 < kq || !fetched;) {
            // what is left of the tile (quads per group) in segments of about equal length, at most len; quotients of
            // numbers below 256 half a unit off the whole ones, so that an approximate division is exact
            const int left = (kq - s0 + G - 1) / G;
            const int parts = max(1, __float2int_rd(__fdividef(left + len - 0.5f, len)));
            const int seg = __float2int_rd(__fdividef(left + parts - 0.5f, parts));
            const int qa = min(kq, s0 + group * seg), qb = min(kq, qa + seg);
            int n = 0;
            if (s0 < kq && slow_left == 0) {
                const Consts K = constants(J.inv_w, J.c, J.scale, nb);
                const int m0 = min(qb, max(qa, mq0)), m1 = max(m0, min(qb, mq1));
                for (int q = max(qa, q_warp); q < m0; ++q)
                    quad_pairs<true, R, NR, DSUM, CLAMP>(s_q + q, 4 * q, ox, oy, oz, caddr, p, kt, K, n);
#pragma unroll 4
                for (int q = m0; q < m1; ++q) quad_pairs<false, R, NR, DSUM, CLAMP>(s_q + q, 0, ox, oy, oz, caddr, p, kt, K, n);
                n += (m1 - m0) * (4 * R);
                for (int q = max(m1, q_warp); q < qb; ++q)
                    quad_pairs<true, R, NR, DSUM, CLAMP>(s_q + q, 4 * q, ox, oy, oz, caddr, p, kt, K, n);
            }
            if (!fetched) {
                // every thread left the other buffer at the previous tile's last barrier
                if (tid < 32) fetch(buf ^ 1, static_cast<long long>(__shfl_sync(0xffffffffu, drawn, 0)) + gridDim.x);
                fetched = true;
            }
            if (s0 >= kq) break;
            if (slow_left == 0) {
                __syncthreads();
                // words -> counts and offset sums (undo: the same words again, taken back)
                // a word holds less than 2^23 of offsets and 512 counts; what a segment adds stays on chip
                // until its check, so that it can be taken back
                const int pk_rows = rows * copies, most = copies * max(rows, 4);
                if (!undo && room < most) flush();
                int sum = -n;
                uint32_t fill = 0;
                // few quads of bins: several threads share a quad's rows (and, with several copies, a quad of counts)
                const int quads = nb / 4 + 1;
                auto drain = [&](auto several) {
                    constexpr bool MANY = decltype(several)::value;
                    const int copy_bits = __ffs(copies) - 1;
                    const int split = quads * 2 <= NT ? min(pk_rows, NT / quads) : 1;
                    const int first = split > 1 ? tid / quads : 0;
                    for (int b = (tid - first * quads) * 4; b <= nb && first < split; b += NT * 4) {
                        uint4 off = make_uint4(0, 0, 0, 0);
                        for (int r = first; r < pk_rows; r += split) {
                            uint4* const pw = reinterpret_cast<uint4*>(s_pk + r * pad + b);
                            uint2* const pc = reinterpret_cast<uint2*>(s_cnt + (MANY ? r >> copy_bits : r) * pad + b);
                            const uint4 w = *pw;
                            const bool shared = MANY && split > 1;
                            uint2 c = shared ? make_uint2(0, 0) : *pc;
                            *pw = make_uint4(0, 0, 0, 0);
                            const uint32_t n0 = w.x >> kPackCountShift, n1 = w.y >> kPackCountShift, n2 = w.z >> kPackCountShift,
                                           n3 = w.w >> kPackCountShift;
                            const uint32_t c0 = n0 | n1 << 16, c1 = n2 | n3 << 16;
                            c = undo ? make_uint2(c.x - c0, c.y - c1) : make_uint2(c.x + c0, c.y + c1);
                            off = make_uint4(off.x + (w.x & kOffsetMask), off.y + (w.y & kOffsetMask), off.z + (w.z & kOffsetMask),
                                             off.w + (w.w & kOffsetMask));
                            if (shared) {
                                if (c.x) shared_red_add(smem_addr(pc), c.x);
                                if (c.y) shared_red_add(smem_addr(pc) + 4, c.y);
                            } else {
                                *pc = c;
                            }
                            sum += static_cast<int>(n0 + n1) + static_cast<int>(n2 + n3);
                            fill = max(max(fill, w.x), w.y);
                            fill = max(max(fill, w.z), w.w);
                        }
                        if (DSUM) {
                            if (undo) off = make_uint4(0u - off.x, 0u - off.y, 0u - off.z, 0u - off.w);
                            if (split > 1) {
                                const uint32_t a = smem_addr(s_dacc + b);
                                if (off.x) shared_red_add(a, off.x);
                                if (off.y) shared_red_add(a + 4, off.y);
                                if (off.z) shared_red_add(a + 8, off.z);
                                if (off.w) shared_red_add(a + 12, off.w);
                            } else {
                                uint4* const pd = reinterpret_cast<uint4*>(s_dacc + b);
                                const uint4 d = *pd;
                                *pd = make_uint4(d.x + off.x, d.y + off.y, d.z + off.z, d.w + off.w);
                            }
                        }
                    }
                };
                if (L.many && copies > 1) drain(std::true_type{});
                else drain(std::false_type{});
                sum = __reduce_add_sync(0xffffffffu, sum);
                fill = __reduce_max_sync(0xffffffffu, fill);
                if (lane == 0) {
                    if (sum) atomicAdd(&s_diff[ph], sum);
                    atomicMax(&s_fill[ph], fill);
                }
                __syncthreads();
                const bool bad = s_diff[ph] != 0;
                const uint32_t full = s_fill[ph] >> kPackCountShift;
                if (tid == 0) {
                    s_diff[ph ^ 1] = 0;
                    s_fill[ph ^ 1] = 0;
                }
                ph ^= 1;
                if (!undo) {
                    if (bad) {
                        undo = true;
                        continue;
                    }
                    // (a count has taken at most the fullest word's of every copy, the offset sums 2^23 of every word)
                    room -= min(most, max(copies * static_cast<int>((full >> 7) + 1), pk_rows));
                    s0 += G * seg;
                    // the fullest word's count decides the next segments' length
                    if (full * len > 200 * seg) len = max(1, len - (len + 3) / 4);
                    else if (full * len < 140 * seg) len = min(kMaxLen, len + (len + 7) / 8);
                    continue;
                }
                undo = false;
                if (seg > 1) {
                    len = seg / 2;
                    continue;
                }
                len = 1;
                slow_left = 64;
            }
            // two atomics per pair: the segments after one whose words could not hold it at the smallest length
            constexpr int kUse = NT * R * 4 / 128;  // one quad per thread and outer point
            if (room < kUse) flush();
            room -= kUse;
            slow(4 * qa, min(kt, 4 * qb), 0x7fffffff);
            s0 += G * seg;
            --slow_left;
        }
        if (kt < t.jn) {
            // scalar-tail candidates: at most three inner points, by the first group
            constexpr int kUse = (3 * OUT + 127) / 128;
            if (room < kUse) flush();
            room -= kUse;
            if (group == 0) slow(kt, t.jn, J.tail_end);
        }
        fence_proxy_async();  // this thread's accesses to the buffer before the next bulk copy into it
        __syncthreads();
        buf ^= 1;
    }
    if (cur >= 0 && !failed) flush();
    if (!failed && tid == 0) {
        mbar_inval(&s_bar[0]);
        mbar_inval(&s_bar[1]);
    }
}

// The packed evaluation against the scalar one, on points of boxes up to the reach of nb bins: pairs whose bin or
// offset differs.
template <int NR>
__global__ void pack_check_kernel(float inv_w, float c, float scale, int nb, u64* mismatches) {
    uint32_t state = (blockIdx.x * blockDim.x + threadIdx.x) * 2654435761u + 12345u;
    const Consts K = constants(inv_w, c, scale, nb);
    constexpr float S = 1.0f / 8388608.0f;
    int bad = 0;
    for (int it = 0; it < 32; ++it) {
        const float box = 0.5f * static_cast<float>(nb) * c / static_cast<float>(1 << (it & 7));
        float v[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            state = state * 1664525u + 1013904223u;
            v[k] = static_cast<float>(state >> 8) * 0x1p-24f * box;
        }
        const u64 ox = pack2(v[0] * S, v[0] * S), oy = pack2(v[1] * S, v[1] * S), oz = pack2(v[2] * S, v[2] * S);
        const u64 bx = pack2(-v[3] * S, -v[6] * S), by = pack2(-v[4] * S, -v[7] * S), bz = pack2(-v[5] * S, -v[8] * S);
        float x[4];
        uint32_t add[4];
        pair_values<NR, true, true>(ox, oy, oz, bx, by, bz, K, x[0], x[1], add[0], add[1]);
        pair_values<NR, true, false>(ox, oy, oz, bx, by, bz, K, x[2], x[3], add[2], add[3]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float* b = v + 3 + 3 * (k & 1);
            const float dx = __fsub_rn(v[0], b[0]), dy = __fsub_rn(v[1], b[1]), dz = __fsub_rn(v[2], b[2]);
            const float d = pair_sqrt_nr(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
            const float xm = __fadd_rn(__fmul_rn(d, inv_w), kMagic);
            const float t = __fmaf_rn(__fmaf_rn(-__fsub_rn(xm, kMagic), c, d), scale, kMagic);
            const uint32_t want = (1u << kPackCountShift) + static_cast<uint32_t>(__float_as_int(t) - kMagicBits + kResBias);
            if (x[k] != xm || add[k] != want) ++bad;
        }
    }
    if (bad) atomicAdd(mismatches, static_cast<u64>(bad));
}

using Kernel = void (*)(const PackLaunch);

template <int NT, int G, bool CLAMP>
Kernel pick(int nr, bool dsum) {
    if (nr == 2) return dsum ? pack_kernel<NT, G, 2, true, CLAMP> : pack_kernel<NT, G, 2, false, CLAMP>;
    return dsum ? pack_kernel<NT, G, 1, true, CLAMP> : pack_kernel<NT, G, 1, false, CLAMP>;
}

template <bool CLAMP>
Kernel pick_shape(int shape, int nr, bool dsum) {
    switch (shape) {
        case 0: return pick<128, 1, CLAMP>(nr, dsum);
        case 1: return pick<256, 1, CLAMP>(nr, dsum);
        case 2: return pick<256, 2, CLAMP>(nr, dsum);
        default: return pick<512, 2, CLAMP>(nr, dsum);
    }
}

}  // namespace

size_t pack_smem_bytes(const PackLaunch& L) {
    const size_t rows2 = (L.group_rows + 1) & ~1;
    return (2 * static_cast<size_t>(L.rows) + 2 * static_cast<size_t>(L.group_sums) + rows2) * pack_pad(L.bins) * 2 +
           2 * static_cast<size_t>(L.tile_j) * 16;
}

int pack_ctas_per_sm(int shape, const PackLaunch& L) {
    const size_t smem = pack_smem_bytes(L);
    if (smem > kPairSmemCap) return 0;
    // what the launch bounds keep resident by registers, and the shared memory (1 KB reserved and the static
    // arrays per CTA); no call into the runtime, since one-shot calls plan every time
    return std::min(pack_min_blocks(kPackShapes[shape].threads), static_cast<int>(233472 / (smem + 1536)));
}

int pack_shape(const PackLaunch& L) {
    for (int s : {0, 1})
        if (pack_ctas_per_sm(s, L) * kPackShapes[s].threads >= 512) return s;
    return pack_ctas_per_sm(3, L) > 0 ? 3 : -1;
}

constexpr int kLongSegment = 24576;  // pairs of a segment that is long enough
constexpr int kCopyWords = 4096;     // words that copies may take: a quarter of a resident CTA's shared memory

int pack_segment_pairs(int bins, double largest_row_share) {
    const double n = 52.0 * bins / std::max(0.01, largest_row_share);
    return static_cast<int>(std::min<double>(n, kPackMaxPairs));
}

int pack_copies(int rows, int bins, int spread, double largest_row_share) {
    int n = 1;
    while (n < 16 && 2 * n * rows * pack_pad(bins) <= kCopyWords &&
           pack_segment_pairs(spread, largest_row_share / n) < kLongSegment)
        n *= 2;
    return n;
}

void pack_check_launch(float inv_w, int bins, bool power_of_two, unsigned long long* mismatches, cudaStream_t s) {
    const float c = static_cast<float>(1.0 / static_cast<double>(inv_w));
    const float scale = static_cast<float>(32768.0 / static_cast<double>(c) * (1.0 - 1.0 / 256));
    if (power_of_two) pack_check_kernel<2><<<148, 256, 0, s>>>(inv_w, c, scale, bins, mismatches);
    else pack_check_kernel<1><<<148, 256, 0, s>>>(inv_w, c, scale, bins, mismatches);
}

void pack_launch(const PackLaunch& L, int shape, int grid, cudaStream_t s) {
    const size_t smem = pack_smem_bytes(L);
    Kernel k = L.covered ? pick_shape<false>(shape, L.nr, L.offsets != 0) : pick_shape<true>(shape, L.nr, L.offsets != 0);
    // the most any launch takes, not this one's: the limit belongs to the process, and another thread's launch may
    // come between the two calls
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPairSmemCap));
    k<<<grid, kPackShapes[shape].threads, smem, s>>>(L);
}

}  // namespace ausaxs_b200
