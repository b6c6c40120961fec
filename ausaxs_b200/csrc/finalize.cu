// Manager post-processing on the device: the part of calculate_all() after the pair loops.
//
// From the integer accumulators of the pair kernel this builds, in FP64, what the reference's
// managers return: factors, self-correlation terms, the excluded-volume rows (as marginals of the
// atom-atom rows), the Z_exv scaling, the truncation to max_bin, and the weighted distance axes.
//   HistogramManagerMT.cpp:23-75, SimpleCalculator.h:143-161           (Simple / weights)
//   HistogramManagerMTFFAvg.cpp:304-371                                (FFAvg)
//   HistogramManagerMTFFExplicit.cpp:303-345                           (FFExplicit)
//   HistogramManagerMTFFGrid.cpp:161-233                               (FFGrid)
//   WeightedDistribution1D.cpp:51-58, DistanceHistogram.cpp:30-47     (weighted axis)
#include "finalize.cuh"

namespace ausaxs_b200 {

namespace {

// Sum of factor * d over the pairs of one job in bin b, from its fixed-point offsets:
// d = b*c + r for every pair, r = (acc - n * bias) / scale.
__device__ __forceinline__ double dist_sum(const unsigned long long* ds, const unsigned long long n, int b, float c,
                                           float scale) {
    if (!ds || n == 0) return 0.0;
    long long resid = static_cast<long long>(ds[b]) - static_cast<long long>(n) * kResBias;
    return static_cast<double>(n) * b * static_cast<double>(c) + static_cast<double>(resid) / static_cast<double>(scale);
}

// WeightedDistribution1D::get_weighted_axis for one bin: mean distance, or the bin's lower value when empty.
__device__ __forceinline__ double weighted_bin(double dsum, double count, int b, double width) {
    unsigned int cnt = static_cast<unsigned int>(count);
    double dv = 0 + b * width;
    return (static_cast<double>(dsum == 0) * dv + dsum) / static_cast<double>((cnt == 0) + cnt);
}

// Post-processing takes one launch: the blocks write the rows of their bins and raise max_bin, and the
// block that finishes last forms the distance axes, which depend on it (their bin width is
// (max_bin * width) / max_bin, bins beyond it are zero).  Bound: the latency of one round of loads; a
// thread per (bin, row slice) has all of its loads in flight at once (cold, 5,000 atoms: two launches with
// a thread per bin and serial row loads took 7 + 17 us, this one 10).
constexpr int kFinBins = 32, kFinSlices = 8;

// Whether this block is the last of `blocks` of its structure to get here; what the others wrote is then
// visible (read it past L1).  The counter returns to 0 for the next launch.
__device__ bool last_block(unsigned* done, unsigned blocks) {
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    const bool first = threadIdx.x == 0 && threadIdx.y == 0;
    if (first) {
        const unsigned n = atomicAdd(done, 1u);
        s_last = n + 1 == blocks;
        if (s_last) *done = 0;
    }
    __syncthreads();
    __threadfence();
    return s_last;
}

// max_bin past the warp's last bin in use (lane l holds bin b of the warp's 32 in order), at least the minimum
// size (HistogramManagerMT.cpp:48).  All 32 lanes call it: what they did for their bins may have parted them.
__device__ __forceinline__ void raise_max_bin(int32_t* max_bin, bool in_use, int b) {
    const unsigned at = __ballot_sync(0xffffffffu, in_use);
    if ((threadIdx.x & 31) == 0) atomicMax(max_bin, max(10, at ? b + 32 - __clz(at) : 0));
}

__device__ void ff_finalize_body(const FinalizeFF& F, unsigned blocks) {
    __shared__ unsigned long long s_n[3][kFinSlices][kFinBins];  // aa pairs, aw pairs, ax pairs of the slice's types
    const int T = F.T;
    const size_t nb = F.nb;
    const int lane = threadIdx.x, slice = threadIdx.y;
    const int b = blockIdx.x * kFinBins + lane;
    const bool grid = F.kind == kKindGrid;
    unsigned long long n_aa = 0, n_aw = 0, n_ax = 0;
    if (b < F.nb) {
        for (int ta = slice; ta < T; ta += kFinSlices) {
            // atom-atom rows: factor 2, self terms (ff, ff, 0) += atoms of that type
            unsigned long long of_type = 0;
#pragma unroll 4
            for (int tb = 0; tb < T; ++tb) {
                const unsigned long long c = F.cnt_aa[static_cast<size_t>(ta * T + tb) * nb + b];
                of_type += c;
                double v = 2.0 * static_cast<double>(c);
                if (b == 0 && ta == tb) v += F.type_count[ta];
                F.H[static_cast<size_t>(ta * T + tb) * nb + b] = v;
            }
            n_aa += of_type;
            // [ff][exv] rows: every atom-atom pair also increments (ff_i, exv) with the lower-index
            // atom's type (HistogramManagerMTFFAvg.cpp:27-35), i.e. the marginal over ff_j
            double ax = 0;
            if (F.kind == kKindAvg) {
                ax = 2.0 * static_cast<double>(of_type) * F.z_exv;
            } else if (grid) {
                const unsigned long long c = F.cnt_ax[static_cast<size_t>(ta) * nb + b];
                n_ax += c;
                ax = static_cast<double>(c);
            }
            F.H[static_cast<size_t>(T * T + ta) * nb + b] = ax;
            // atom-water rows (factor 1)
            const unsigned long long c = F.cnt_aw[static_cast<size_t>(ta) * nb + b];
            n_aw += c;
            F.H[static_cast<size_t>(T * T + T + 1 + ta) * nb + b] = static_cast<double>(c);
        }
    }
    s_n[0][slice][lane] = n_aa;
    s_n[1][slice][lane] = n_aw;
    s_n[2][slice][lane] = n_ax;
    __syncthreads();
    bool in_use = false;
    if (slice == 0 && b < F.nb) {
        for (int k = 1; k < kFinSlices; ++k) {
            n_aa += s_n[0][k][lane];
            n_aw += s_n[1][k][lane];
            n_ax += s_n[2][k][lane];
        }
        const unsigned long long n_ww = F.cnt_ww[b];
        const unsigned long long n_xx = grid ? F.cnt_xx[b] : 0, n_wx = grid ? F.cnt_wx[b] : 0;
        double xx = 0, wx = 0;
        // val * (Z * Z): the reference's release build hoists Z*Z (HistogramManagerMTFFAvg.cpp:361-362)
        if (F.kind == kKindAvg) {
            xx = (2.0 * static_cast<double>(n_aa) + (b == 0 ? F.n_a : 0)) * (F.z_exv * F.z_exv);
            wx = static_cast<double>(n_aw) * F.z_exv;
        } else if (grid) {
            xx = 2.0 * static_cast<double>(n_xx) + (b == 0 ? F.n_x : 0);
            wx = static_cast<double>(n_wx);
        }
        F.H[static_cast<size_t>(T * T + T) * nb + b] = xx;
        F.H[static_cast<size_t>(T * T + 2 * T + 1) * nb + b] = wx;
        F.H[static_cast<size_t>(T * T + 2 * T + 2) * nb + b] = 2.0 * static_cast<double>(n_ww) + (b == 0 ? F.n_w : 0);
        unsigned long long tot = 2ull * n_aa + n_aw + 2ull * n_ww;
        if (b == 0) tot += static_cast<unsigned long long>(F.n_a) + F.n_w;
        F.tot[b] = static_cast<double>(tot);
        // the distance sums of the axes, turned into means by the last block
        if (F.weighted)
            F.d_axis[b] = 2.0 * dist_sum(F.ds_aa, n_aa, b, F.c, F.scale) + dist_sum(F.ds_aw, n_aw, b, F.c, F.scale) +
                          2.0 * dist_sum(F.ds_ww, n_ww, b, F.c, F.scale);
        bool used = tot != 0;
        if (grid) {
            F.d_axis_ax[b] = dist_sum(F.ds_ax, n_ax, b, F.c, F.scale) + dist_sum(F.ds_wx, n_wx, b, F.c, F.scale);
            F.d_axis_xx[b] = 2.0 * dist_sum(F.ds_xx, n_xx, b, F.c, F.scale);
            used = used || xx != 0 || n_wx != 0;
        }
        in_use = used && b >= 10;
    }
    if (slice == 0) raise_max_bin(F.max_bin, in_use, b);
    if (!last_block(F.done, blocks)) return;
    const int mb = __ldcg(F.max_bin);
    const double width = (static_cast<double>(mb) * F.bin_width) / mb;  // Axis(0, mb*width, mb).width()
    for (int k = slice * kFinBins + lane; k < F.nb; k += kFinBins * kFinSlices) {
        if (k >= mb) {
            F.d_axis[k] = 0;
            if (F.d_axis_ax) F.d_axis_ax[k] = 0;
            if (F.d_axis_xx) F.d_axis_xx[k] = 0;
            // (atom-dummy pairs do not raise max_bin: the only rows that can hold something here)
            if (grid)
                for (int t = 0; t < T; ++t) F.H[static_cast<size_t>(T * T + t) * nb + k] = 0;
            continue;
        }
        // weighted axis of p_tot = aa(ff >= 1) + aw(ff >= 1) + ww, bin 0 pinned to 0
        if (F.weighted) F.d_axis[k] = k == 0 ? 0.0 : weighted_bin(__ldcg(F.d_axis + k), __ldcg(F.tot + k), k, width);
        else F.d_axis[k] = k * width;
        if (grid) {
            // ax + wx share one axis, xx has its own; neither pins bin 0 (CompositeDistanceHistogramFFGrid.cpp:129-134)
            double n = __ldcg(F.H + static_cast<size_t>(T * T + 2 * T + 1) * nb + k);
            for (int t = 0; t < T; ++t) n += __ldcg(F.H + static_cast<size_t>(T * T + t) * nb + k);
            F.d_axis_ax[k] = weighted_bin(__ldcg(F.d_axis_ax + k), n, k, width);
            F.d_axis_xx[k] = weighted_bin(__ldcg(F.d_axis_xx + k), __ldcg(F.H + static_cast<size_t>(T * T + T) * nb + k), k, width);
        }
    }
}

__global__ void ff_finalize_kernel(FinalizeFF F) { ff_finalize_body(F, gridDim.x); }
// batched: blockIdx.y selects the structure
__global__ void ff_finalize_batch_kernel(const FinalizeFF* Fs) { ff_finalize_body(Fs[blockIdx.y], gridDim.x); }

// Expansion of the compact rows to the reference's [15][15] / [15] layouts, stride max_bin.
__global__ void ff_expand_kernel(FinalizeFF F, double* aa_out, double* aw_out) {
    const int T = F.T;
    const int mb = *F.max_bin;
    const size_t nb = F.nb;
    const int n = kNff * kNff * mb;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
        int row = idx / mb, b = idx - row * mb;
        int f1 = row / kNff, f2 = row - f1 * kNff;
        double v = 0;
        int t1 = F.ff_to_type[f1], t2 = F.ff_to_type[f2];
        if (f1 != kExv && f2 != kExv) {
            if (t1 >= 0 && t2 >= 0) v = F.H[static_cast<size_t>(t1 * T + t2) * nb + b];
        } else if (f1 != kExv && f2 == kExv) {
            if (t1 >= 0 && F.kind != kKindExplicit) v = F.H[static_cast<size_t>(T * T + t1) * nb + b];
        } else if (f1 == kExv && f2 == kExv) {
            if (F.kind != kKindExplicit) v = F.H[static_cast<size_t>(T * T + T) * nb + b];
        }
        aa_out[idx] = v;
    }
    const int n2 = kNff * mb;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n2; idx += gridDim.x * blockDim.x) {
        int f = idx / mb, b = idx - f * mb;
        double v = 0;
        if (f == kExv) {
            if (F.kind != kKindExplicit) v = F.H[static_cast<size_t>(T * T + 2 * T + 1) * nb + b];
        } else if (F.ff_to_type[f] >= 0) {
            v = F.H[static_cast<size_t>(T * T + T + 1 + F.ff_to_type[f]) * nb + b];
        }
        aw_out[idx] = v;
    }
}

// ---- Simple / weighted (HistogramManagerMT) -------------------------------------------------

__global__ void weight_square_sum_kernel(const float4* p, int n, double* out) {
    double s = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float w = p[i].w;
        s += static_cast<double>(__fmul_rn(w, w));  // float product, summed in double (SimpleCalculator.h:146-150)
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

__global__ void weight_scale_kernel(const float4* a, int na, const float4* b, int nb, float* wscale) {
    // largest |w| over both sets; scale 2^k with (max|w|)^2 * 2^k <= 2^30
    __shared__ float s_max[32];
    float m = 0;
    for (int i = threadIdx.x; i < na; i += blockDim.x) m = fmaxf(m, fabsf(a[i].w));
    for (int i = threadIdx.x; i < nb; i += blockDim.x) m = fmaxf(m, fabsf(b[i].w));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float mm = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) mm = fmaxf(mm, s_max[k]);
        double p = static_cast<double>(mm) * mm;
        int e = 0;
        if (p > 0) frexp(p, &e);  // p < 2^e
        int k = 30 - e;
        if (k > 60) k = 60;
        *wscale = ldexpf(1.0f, k);
    }
}

// Pairs and fixed-point weight sum of one job in bin b.  The two-atomic kernel adds rint(w_i w_j * wscale) +
// 2^30 per pair (unsigned, wrapping) and the bias of n pairs is removed; rows by class give the same sum.  rows 0:
// not by class, or no such pairs (one row of zeros).
struct MTSum {
    unsigned long long n;
    long long w;
};
__device__ MTSum mt_sum(const unsigned long long* cnt, const long long* w, int rows, int cols, const float* cr, const float* cc,
                        float wscale, size_t nb, int b) {
    MTSum s{0, 0};
    if (rows == 0) {
        s.n = cnt[b];
        s.w = static_cast<long long>(static_cast<unsigned long long>(w[b]) - s.n * (1ull << 30));
        return s;
    }
    for (int r = 0; r < rows; ++r)
#pragma unroll 4
        for (int k = 0; k < cols; ++k) {
            const unsigned long long n = cnt[static_cast<size_t>(r * cols + k) * nb + b];
            s.n += n;
            s.w += static_cast<long long>(n) * __float2int_rn(__fmul_rn(__fmul_rn(cr[r], cc[k]), wscale));
        }
    return s;
}

__global__ void mt_finalize_kernel(FinalizeMT F) {
    const size_t nb = F.nb;
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    bool in_use = false;
    if (b < F.nb) {
        const float wscale = F.by_class ? F.wscale_v : *F.wscale;
        const double inv = 1.0 / static_cast<double>(wscale);
        const MTSum s_aa = mt_sum(F.c_aa, F.w_aa, F.ta, F.ta, F.class_a, F.class_a, wscale, nb, b);
        const MTSum s_aw = mt_sum(F.c_aw, F.w_aw, F.ta ? F.tw : 0, F.ta, F.class_w, F.class_a, wscale, nb, b);
        const MTSum s_ww = mt_sum(F.c_ww, F.w_ww, F.tw, F.tw, F.class_w, F.class_w, wscale, nb, b);
        double aa = 2.0 * (static_cast<double>(s_aa.w) * inv);
        double aw = 2.0 * (static_cast<double>(s_aw.w) * inv);
        double ww = 2.0 * (static_cast<double>(s_ww.w) * inv);
        F.n32[b] = 2u * static_cast<unsigned>(s_aa.n) + 2u * static_cast<unsigned>(s_ww.n) + 2u * static_cast<unsigned>(s_aw.n);
        if (F.weighted)
            F.d_axis[b] = 2.0 * dist_sum(F.ds_aa, s_aa.n, b, F.c, F.scale) + 2.0 * dist_sum(F.ds_ww, s_ww.n, b, F.c, F.scale) +
                          2.0 * dist_sum(F.ds_aw, s_aw.n, b, F.c, F.scale);
        double v = aa + ww + aw;  // (the order in which bins count as used)
        if (b == 0) {
            const double d_aa = F.by_class ? F.self_v[0] : *F.self_aa, d_ww = F.by_class ? F.self_v[1] : *F.self_ww;
            aa += d_aa;
            ww += d_ww;
            v += d_aa + d_ww;
        }
        F.H[b] = aa;
        F.H[nb + b] = aw;
        F.H[2 * nb + b] = ww;
        F.tot[b] = aa + ww + aw;
        in_use = v != 0 && b >= 10;
    }
    raise_max_bin(F.max_bin, in_use, b);
    if (!last_block(F.done, gridDim.x)) return;
    const int mb = __ldcg(F.max_bin);
    const double width = (static_cast<double>(mb) * F.bin_width) / mb;
    for (int k = threadIdx.x; k < F.nb; k += blockDim.x) {
        if (k >= mb) {
            F.H[k] = F.H[nb + k] = F.H[2 * nb + k] = 0;
            F.tot[k] = 0;
            F.d_axis[k] = 0;
        } else if (F.weighted && k > 0) {
            F.d_axis[k] = weighted_bin(__ldcg(F.d_axis + k), static_cast<double>(static_cast<unsigned>(__ldcg(F.n32 + k))), k, width);
        } else {
            F.d_axis[k] = k == 0 ? 0.0 : k * width;
        }
    }
}

}  // namespace

void ff_finalize_launch(const FinalizeFF& F, cudaStream_t s) {
    ff_finalize_kernel<<<(F.nb + kFinBins - 1) / kFinBins, dim3(kFinBins, kFinSlices), 0, s>>>(F);
}

void ff_finalize_batch_launch(const FinalizeFF* Fs_dev, int n, int max_nb, cudaStream_t s) {
    ff_finalize_batch_kernel<<<dim3((max_nb + kFinBins - 1) / kFinBins, n), dim3(kFinBins, kFinSlices), 0, s>>>(Fs_dev);
}

void ff_expand_launch(const FinalizeFF& F, double* aa_out, double* aw_out, int nb_hint, cudaStream_t s) {
    int threads = 256;
    int blocks = (kNff * kNff * nb_hint + threads - 1) / threads;
    if (blocks > 2048) blocks = 2048;
    ff_expand_kernel<<<blocks, threads, 0, s>>>(F, aa_out, aw_out);
}

void weight_scale_launch(const float4* a, int na, const float4* b, int nb, float* wscale, cudaStream_t s) {
    weight_scale_kernel<<<1, 1024, 0, s>>>(a, na, b, nb, wscale);
}

void weight_square_sum_launch(const float4* p, int n, double* out, cudaStream_t s) {
    int blocks = (n + 255) / 256;
    if (blocks > 148 * 4) blocks = 148 * 4;
    if (blocks < 1) blocks = 1;
    weight_square_sum_kernel<<<blocks, 256, 0, s>>>(p, n, out);
}

void mt_finalize_launch(const FinalizeMT& F, cudaStream_t s) {
    mt_finalize_kernel<<<(F.nb + 127) / 128, 128, 0, s>>>(F);
}

}  // namespace ausaxs_b200
