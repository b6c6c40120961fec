// Point-set preparation: bounding box, form-factor type census and dense-type conversion.
//
// Mirrors CompactCoordinatesFF::setup (include/core/hist/detail/CompactCoordinatesFF.h:21-32):
// every atom's form-factor type is validated (UNKNOWN and out-of-range types are an error) and
// remapped, here to a dense index over the types the structure actually contains, so that the
// on-chip histograms hold T*T rows instead of 15*15.
#include <algorithm>

#include "prep.cuh"

namespace ausaxs_b200 {

namespace {

// float <-> order-preserving uint32 (for atomicMin/atomicMax on floats)
__device__ __forceinline__ unsigned int f2o(float f) {
    unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// first slot of a weight in a table of classes
__device__ __forceinline__ unsigned class_hash(unsigned w) { return (w * 2654435761u) >> 27; }
static_assert(kClassSlots == 32, "one slot per lane, and five hash bits");

// The block's table starts with the weights of its first warp of points, one after the other (lane k keeps slot k):
// with every thread inserting its own, the first round was a string of compare-and-swaps of many lanes to one
// word.
__device__ void class_begin(WeightClasses& t, const float4* p, int n) {  // (a barrier follows)
    const int lane = threadIdx.x;
    if (lane >= 32) return;
    const int i = blockIdx.x * blockDim.x + lane;
    const unsigned w = i < n ? __float_as_uint(p[i].w) : kNoClass;
    unsigned left = __ballot_sync(0xffffffffu, i < n);
    unsigned mine = kNoClass;
    int found = 0;
    bool over = false;
    while (left) {
        const unsigned x = __shfl_sync(0xffffffffu, w, __ffs(left) - 1);
        if (x == kNoClass || ++found > kMaxClasses) {
            over = true;
            break;
        }
        const unsigned h = class_hash(x), empty = __ballot_sync(0xffffffffu, mine == kNoClass);
        if (lane == static_cast<int>((__ffs(__funnelshift_r(empty, empty, h)) - 1 + h) & 31u)) mine = x;
        left &= ~__ballot_sync(0xffffffffu, w == x);
    }
    t.bits[lane] = mine;
    t.count[lane] = 0;
    if (lane == 0) t.over = over;
}

// Slots are never emptied, so a weight is met before the first empty slot after its own.
__device__ void class_add(WeightClasses& t, unsigned w) {
    if (*reinterpret_cast<volatile int*>(&t.over)) return;
    for (unsigned j = 0, k = class_hash(w); w != kNoClass && j < kClassSlots; ++j, k = (k + 1) & 31u) {
        unsigned have = *reinterpret_cast<volatile unsigned*>(t.bits + k);
        if (have == kNoClass) have = atomicCAS(t.bits + k, kNoClass, w);
        if (have == kNoClass || have == w) {
            atomicAdd(t.count + k, 1);
            return;
        }
    }
    t.over = 1;
}

// The block's table into the device's, a thread per slot (a barrier precedes).
__device__ void class_merge(const WeightClasses& t, WeightClasses* out) {
    if (threadIdx.x < kClassSlots && t.bits[threadIdx.x] != kNoClass && !t.over) {
        const unsigned w = t.bits[threadIdx.x];
        unsigned j = 0;
        for (unsigned k = class_hash(w); j < kClassSlots; ++j, k = (k + 1) & 31u) {
            unsigned have = __ldcg(out->bits + k);
            if (have == kNoClass) have = atomicCAS(out->bits + k, kNoClass, w);
            if (have == kNoClass || have == w) {
                atomicAdd(out->count + k, t.count[threadIdx.x]);
                break;
            }
        }
        if (j == kClassSlots) out->over = 1;
    }
    if (threadIdx.x == 0 && t.over) out->over = 1;
}

// classes: also the points' distinct weights, or null
__global__ void census_kernel(const float4* p, int n, int ff_typed, PrepStats* st, WeightClasses* classes) {
    __shared__ WeightClasses s_class;
    if (classes) class_begin(s_class, p, n);
    __shared__ unsigned int s_lo[3], s_hi[3], s_mask, s_bad;
    __shared__ int s_count[kNff];
    if (threadIdx.x < 3) {
        s_lo[threadIdx.x] = 0xffffffffu;
        s_hi[threadIdx.x] = 0u;
    }
    if (threadIdx.x < kNff) s_count[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_mask = 0, s_bad = 0;
    __syncthreads();
    unsigned int lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 v = p[i];
        unsigned int o[3] = {f2o(v.x), f2o(v.y), f2o(v.z)};
        for (int k = 0; k < 3; ++k) {
            lo[k] = min(lo[k], o[k]);
            hi[k] = max(hi[k], o[k]);
        }
        if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) atomicOr(&s_bad, 2u);
        if (ff_typed) {
            int t = __float_as_int(v.w);
            if (t <= kExv || t >= kNff) atomicOr(&s_bad, 1u);
            else {
                atomicOr(&s_mask, 1u << t);
                atomicAdd(&s_count[t], 1);
            }
        }
        if (classes) class_add(s_class, __float_as_uint(v.w));
    }
    for (int k = 0; k < 3; ++k) {
        atomicMin(&s_lo[k], lo[k]);
        atomicMax(&s_hi[k], hi[k]);
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        atomicMin(&st->lo[threadIdx.x], s_lo[threadIdx.x]);
        atomicMax(&st->hi[threadIdx.x], s_hi[threadIdx.x]);
    }
    if (threadIdx.x < kNff && s_count[threadIdx.x]) atomicAdd(&st->count[threadIdx.x], s_count[threadIdx.x]);
    if (threadIdx.x == 0) {
        atomicOr(&st->mask, s_mask);
        atomicOr(&st->bad, s_bad);
    }
    if (classes) class_merge(s_class, classes);
}

__device__ __forceinline__ float o2f(unsigned int o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// max |p - c|^2 in double over the three point sets; non-negative doubles order like their bits
__global__ void radius_kernel(const float4* a, int na, const float4* w, int nw, const float4* x, int nx, PrepStats* st) {
    double c[3];
    for (int k = 0; k < 3; ++k) c[k] = 0.5 * ((double)o2f(st->lo[k]) + (double)o2f(st->hi[k]));
    double r2 = 0;
    const int n = na + nw + nx;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 v = i < na ? a[i] : (i < na + nw ? w[i - na] : x[i - na - nw]);
        const double dx = v.x - c[0], dy = v.y - c[1], dz = v.z - c[2];
        r2 = fmax(r2, dx * dx + dy * dy + dz * dz);
    }
    for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
    if ((threadIdx.x & 31) == 0 && r2 > 0) atomicMax(&st->r2, static_cast<unsigned long long>(__double_as_longlong(r2)));
}

// Dense copy of the points (w = dense type; type map null: w already is), and the points of each
// type in every chunk of kTypedChunk points.
__device__ void dense_count(const float4* in, float4* out, int n, const TypeMap& map, int32_t* counts) {
    __shared__ int s_count[16];
    if (threadIdx.x < 16) s_count[threadIdx.x] = 0;
    __syncthreads();
    const int i = blockIdx.x * kTypedChunk + threadIdx.x;
    if (i < n) {
        float4 v = in[i];
        const int t = __float_as_int(v.w);
        int d = t;
        if (map.classes > 0) {
            d = 0;
            for (int k = 1; k < map.classes; ++k)
                if (map.bits[k] == static_cast<unsigned>(t)) d = k;
        } else if (map.ff_to_type) {
            d = (t > kExv && t < kNff) ? map.ff_to_type[t] : 0;
        }
        v.w = __int_as_float(d);
        if (out) out[i] = v;
        const unsigned same = __match_any_sync(__activemask(), d);
        if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&s_count[d], __popc(same));
    }
    __syncthreads();
    if (threadIdx.x < 16) counts[blockIdx.x * 16 + threadIdx.x] = s_count[threadIdx.x];
}

// The lists of points by type, ascending index (a stable partition): chunk c writes its points after
// those of the earlier chunks.  w of a listed point is its index.
__device__ void typed_scatter(const float4* dense, int n, const TypedOut& o, const int32_t* counts) {
    constexpr int kW = kTypedChunk / 32;
    __shared__ int s_warp[kW + 1][16];  // points of a type in the warps before
    __shared__ int s_base[16];          // ... in the chunks before
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 16 * (kW + 1)) (&s_warp[0][0])[threadIdx.x] = 0;
    __syncthreads();
    const int i = blockIdx.x * kTypedChunk + threadIdx.x;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    int d = 15, rank = 0;
    if (i < n) {
        v = dense[i];
        d = __float_as_int(v.w);
    }
    const unsigned same = __match_any_sync(0xffffffffu, d);
    rank = __popc(same & ((1u << lane) - 1u));
    if (rank == 0) s_warp[warp + 1][d] = __popc(same);
    if (warp < o.types) {  // one warp per type adds up the earlier chunks (kW warps, at most 15 types)
        int b = 0;
        for (int c = lane; c < static_cast<int>(blockIdx.x); c += 32) b += counts[c * 16 + warp];
        b = __reduce_add_sync(0xffffffffu, b);
        if (lane == 0) s_base[warp] = b;
    }
    __syncthreads();
    if (threadIdx.x < o.types)
        for (int w = 1; w <= kW; ++w) s_warp[w][threadIdx.x] += s_warp[w - 1][threadIdx.x];
    __syncthreads();
    if (i < n) {
        const int at = o.start[d] + s_base[d] + s_warp[warp][d] + rank;
        o.pts[at] = make_float4(v.x, v.y, v.z, __int_as_float(i));
        if (o.pos) o.pos[i] = at;
    }
    // points with an index below every multiple of 256 of the chunk (and below n after the last)
    constexpr int kSub = kTypedChunk / kTypedPre;
    for (int k = threadIdx.x; k < kSub * o.types; k += kTypedChunk) {
        const int t = k / kSub, sub = k - t * kSub;
        const int c = blockIdx.x * kSub + sub;
        if (c < o.pre_stride) o.pre[t * o.pre_stride + c] = s_base[t] + s_warp[sub * (kTypedPre / 32)][t];
    }
}

__global__ void __launch_bounds__(kTypedChunk) dense_count_kernel(const float4* in, float4* out, int n, TypeMap map,
                                                                  int32_t* counts) {
    dense_count(in, out, n, map, counts);
}
__global__ void __launch_bounds__(kTypedChunk) typed_scatter_kernel(const float4* dense, int n, TypedOut o, const int32_t* counts) {
    typed_scatter(dense, n, o, counts);
}
// many sets: blockIdx.y selects the set
__global__ void __launch_bounds__(kTypedChunk) dense_count_sets_kernel(const TypedSetJob* sets, TypeMap map) {
    const TypedSetJob& S = sets[blockIdx.y];
    if (static_cast<int>(blockIdx.x) * kTypedChunk < S.n) dense_count(S.in, S.dense, S.n, map, S.counts);
}
__global__ void __launch_bounds__(kTypedChunk) typed_scatter_sets_kernel(const TypedSetJob* sets) {
    const TypedSetJob& S = sets[blockIdx.y];
    if (static_cast<int>(blockIdx.x) * kTypedChunk < S.n) typed_scatter(S.dense, S.n, S.out, S.counts);
}

__global__ void weight_classes_sets_kernel(const TypedSetJob* sets, WeightClasses* out) {
    __shared__ WeightClasses s_class;
    const float4* p = sets[blockIdx.y].in;
    const int n = sets[blockIdx.y].n;
    class_begin(s_class, p, n);
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) class_add(s_class, __float_as_uint(p[i].w));
    __syncthreads();
    class_merge(s_class, out + blockIdx.y);
}

__global__ void set_type_kernel(float4* p, int n, int32_t value) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i].w = __int_as_float(value);
}

}  // namespace

void WeightClasses::clear() {
    std::fill(bits, bits + kClassSlots, kNoClass);
    std::fill(count, count + kClassSlots, 0);
    over = 0;
}

bool WeightClasses::sorted(std::vector<std::pair<unsigned, int>>& out) const {
    out.clear();
    for (int k = 0; k < kClassSlots; ++k)
        if (bits[k] != kNoClass) out.push_back({bits[k], count[k]});
    std::sort(out.begin(), out.end());
    return !over && out.size() <= static_cast<size_t>(kMaxClasses);
}

void census_launch(const float4* p, int n, int ff_typed, PrepStats* st, WeightClasses* classes, int sm_count, cudaStream_t s) {
    if (n <= 0) return;
    int blocks = (n + 255) / 256;
    if (blocks > sm_count * 2) blocks = sm_count * 2;
    census_kernel<<<blocks, 256, 0, s>>>(p, n, ff_typed, st, classes);
}

void radius_launch(const float4* a, int na, const float4* w, int nw, const float4* x, int nx, PrepStats* st,
                   int sm_count, cudaStream_t s) {
    const long long n = (long long)na + nw + nx;
    if (n <= 0) return;
    long long blocks = (n + 255) / 256;
    if (blocks > sm_count * 2) blocks = sm_count * 2;
    radius_kernel<<<(int)blocks, 256, 0, s>>>(a, na, w, nw, x, nx, st);
}

void typed_lists_launch(const float4* in, float4* dense, int n, const TypeMap& map, const TypedOut& o, int32_t* counts,
                        cudaStream_t s) {
    if (n <= 0) return;
    const int chunks = typed_chunks(n);
    dense_count_kernel<<<chunks, kTypedChunk, 0, s>>>(in, dense, n, map, counts);
    typed_scatter_kernel<<<chunks, kTypedChunk, 0, s>>>(dense ? dense : in, n, o, counts);
}

constexpr int kMaxSets = 65535;  // gridDim.y of one launch

void weight_classes_sets_launch(const TypedSetJob* sets_dev, int sets, int max_n, WeightClasses* out, cudaStream_t s) {
    if (max_n <= 0) return;
    for (int at = 0; at < sets; at += kMaxSets)
        weight_classes_sets_kernel<<<dim3(std::min((max_n + 255) / 256, 32), std::min(sets - at, kMaxSets)), 256, 0, s>>>(sets_dev + at,
                                                                                                                   out + at);
}

void typed_sets_launch(const TypedSetJob* sets_dev, int sets, int max_n, const TypeMap& map, cudaStream_t s) {
    if (max_n <= 0) return;
    for (int at = 0; at < sets; at += kMaxSets) {
        const dim3 grid(typed_chunks(max_n), std::min(sets - at, kMaxSets));
        dense_count_sets_kernel<<<grid, kTypedChunk, 0, s>>>(sets_dev + at, map);
        typed_scatter_sets_kernel<<<grid, kTypedChunk, 0, s>>>(sets_dev + at);
    }
}

void set_type_launch(float4* p, int n, int32_t value, int sm_count, cudaStream_t s) {
    if (n <= 0) return;
    int blocks = (n + 255) / 256;
    if (blocks > sm_count * 4) blocks = sm_count * 4;
    set_type_kernel<<<blocks, 256, 0, s>>>(p, n, value);
}

// host-side inverse of f2o
float ordered_to_float(unsigned int o) {
    unsigned int u = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
    float f;
    memcpy(&f, &u, 4);
    return f;
}

}  // namespace ausaxs_b200
