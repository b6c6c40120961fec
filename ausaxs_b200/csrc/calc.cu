// hist::distance_calculator::SimpleCalculator<weighted_bins = true> on the device
// (include/core/hist/distance_calculator/SimpleCalculator.h:94-330): weighted self and cross jobs with
// an integer scaling factor, accumulated into results keyed by merge id.  SymmetryManagerMT
// (source/core/hist/histogram_manager/SymmetryManagerMT.cpp:37-136) issues its work this way: a
// body's self-distances once with scaling 1 + copies, and one representative of each class of
// equivalent copy pairs with the class size as scaling.
//
// Every job of one run goes into the same persistent pair launches (PairJob::mult carries the
// scaling), each result has its own integer accumulators, and one finalisation kernel turns them
// into the reference's WeightedDistribution1D entries: per bin the weight sum, the count and the
// distance sum, each 2 * scaling times the pair's contribution, plus the self diagonal
// scaling * sum(float(w*w)) in bin 0 (its count: that value truncated to unsigned, per job).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <vector>

#include "engine.cuh"
#include "finalize.cuh"
#include "guard.cuh"
#include "pairhist.cuh"

namespace ausaxs_b200 {
namespace {

struct CalcSlot {
    unsigned long long* cnt;
    unsigned long long* ds;
    long long* ws;
    double diag_value;  // sum over the slot's self jobs of scaling * sum(float(w*w))
    double diag_count;  // sum over them of that value truncated to unsigned
    double* out;        // [3][nb]: value, count, distance sum
};

// Weights of few distinct values: a slot's counts are rows by the two points' classes, [n][n][nb]
struct CalcClasses {
    int n;  // 0: one row, and weight sums
    float w[16];
    float wscale;
};

__device__ __forceinline__ double unbiased_weights(const long long* w, const unsigned long long* n, int b, double inv) {
    const unsigned long long raw = static_cast<unsigned long long>(w[b]) - n[b] * (1ull << 30);
    return static_cast<double>(static_cast<long long>(raw)) * inv;
}

// grid.y = slot; the nb accumulated bins (every later bin is zero)
__global__ void calc_finalize_kernel(const CalcSlot* slots, int nb, const float* wscale, float c, float scale, CalcClasses K) {
    const CalcSlot S = slots[blockIdx.y];
    const double inv = 1.0 / static_cast<double>(K.n ? K.wscale : *wscale);
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        unsigned long long cnt = 0;
        double v;
        if (K.n) {
            // the fixed-point weight product of every class pair times its pairs: the sum the weighted
            // kernel accumulates pair by pair
            long long w = 0;
            for (int i = 0; i < K.n; ++i)
#pragma unroll 4
                for (int j = 0; j < K.n; ++j) {
                    const unsigned long long n = S.cnt[static_cast<size_t>(i * K.n + j) * nb + b];
                    cnt += n;
                    w += static_cast<long long>(n) * __float2int_rn(__fmul_rn(__fmul_rn(K.w[i], K.w[j]), K.wscale));
                }
            v = 2.0 * (static_cast<double>(w) * inv);
        } else {
            cnt = S.cnt[b];
            v = 2.0 * unbiased_weights(S.ws, S.cnt, b, inv);
        }
        double n = 2.0 * static_cast<double>(cnt);
        double d = 0;
        if (cnt) {
            // sum of the pairs' float distances: cnt * b * c + sum of the fixed-point offsets
            const long long resid = static_cast<long long>(S.ds[b]) - static_cast<long long>(cnt) * kResBias;
            d = 2.0 * (static_cast<double>(cnt) * b * static_cast<double>(c) +
                       static_cast<double>(resid) / static_cast<double>(scale));
        }
        if (b == 0) {
            v += S.diag_value;
            n += S.diag_count;
        }
        S.out[b] = v;
        S.out[static_cast<size_t>(nb) + b] = n;
        S.out[2 * static_cast<size_t>(nb) + b] = d;
    }
}

}  // namespace

struct Calculator {
    Ctx* ctx = nullptr;
    double bin_width = 0.25;
    int bin_count = 8000;
    struct Set {
        const float* host;  // the caller's array (must stay valid until run)
        int n;
        size_t off;         // first record in `staged`
    };
    std::vector<Set> sets;
    std::vector<float4> staged;
    struct Job {
        int a, b;  // sets; b < 0: self
        int scaling, slot;
    };
    std::vector<Job> jobs;
    std::map<int, int> ids[2];  // self / cross merge id -> slot
    struct SlotInfo {
        int cross, merge_id;
        int index;  // position among the results of its kind (the reference's res_idx)
    };
    std::vector<SlotInfo> slot_info;
    std::vector<double> results;  // [slots][3][bin_count] of the last run
    std::vector<SlotInfo> result_info;

    int set_of(const float* p, int n) {
        for (size_t k = 0; k < sets.size(); ++k)
            if (sets[k].host == p && sets[k].n == n) return (int)k;
        Set s{p, n, staged.size()};
        staged.resize(staged.size() + n);
        if (n) std::memcpy(staged.data() + s.off, p, (size_t)n * 16);
        sets.push_back(s);
        return (int)sets.size() - 1;
    }

    // SimpleCalculator::enqueue_calculate_self / _cross (SimpleCalculator.h:94-109, 164-181): the
    // result index of the merge id (a new result for a new id; merge id -1: a result of its own,
    // whose id is its index)
    int enqueue(const float* a, int na, const float* b, int nb, int scaling, int merge_id) {
        if (na < 0 || nb < 0 || (na && !a) || (nb && !b)) throw Error{AUSAXS_ERR_ARGUMENT, "invalid point array"};
        if (scaling < 1) throw Error{AUSAXS_ERR_ARGUMENT, "scaling must be positive"};
        const int cross = b != nullptr ? 1 : 0;
        auto& m = ids[cross];
        int slot;
        if (merge_id == -1 || !m.count(merge_id)) {
            const int index = (int)m.size();
            if (merge_id == -1) merge_id = index;
            slot = (int)slot_info.size();
            slot_info.push_back({cross, merge_id, index});
            m[merge_id] = slot;
        } else {
            slot = m[merge_id];
        }
        const int index = slot_info[slot].index;
        jobs.push_back({set_of(a, na), cross ? set_of(b, nb) : -1, scaling, slot});
        return index;
    }

    void run() {
        Ctx& C = *ctx;
        cudaStream_t s = C.stream;
        const int n_slots = (int)slot_info.size();
        results.assign((size_t)n_slots * 3 * bin_count, 0.0);
        result_info = slot_info;
        if (n_slots == 0) return clear();
        // the points, and where it can pay every set's distinct weights, counted while the host finds the largest
        // distance (buffers of the context: a calculator lives for one run, and allocating took longer than the pairs)
        struct Keep {
            Ctx& C;
            ~Keep() {
                for (DevBuf& b : C.calc)
                    if (b.n > Ctx::kCalcKeep) b.release();
            }
        } keep{C};
        DevBuf &in = C.calc[0], &acc = C.calc[1], &out = C.calc[2], &table = C.calc[3];
        const int n_sets = (int)sets.size();
        long long pairs = 0;
        for (const Job& j : jobs) {
            const long long na = sets[j.a].n;
            pairs += j.b < 0 ? na * (na - 1) / 2 : na * sets[j.b].n;
        }
        // Pairs go by class of weight where the rows by class (every result's, cleared and read once) are few against
        // the pairs, and stay within what the context keeps; by value elsewhere.  Measured (6 sets merged into
        // 2 results / 21 results, by class and by value): 300 points each, 15 classes 262 and 256 us / 1,045
        // and 985 us, 8 classes 222 and 256 / 959 and 985; 3,000 points, 15 classes 436 and 431 / 1,347 and 1,357,
        // 4 classes 365 and 431 / 1,221 and 1,357; 50 points (13,700 pairs), 8 classes 217 and 192.
        // A class also costs a pass of its own per job, and what a class saves is a part of the pairs' time: the price
        // of such a pass, in pairs, is from the second list on (40 sets, all pairs of sets: 100 points, 5 and 15 classes
        // 713 and 4,430 us against 260 by value; 300 points, 2 and 5 classes 576 and 931 / 522; 1,000 points, 5
        // classes 1,769 / 1,893; 12 sets of 1,000, 5 and 15 classes 331 and 554 / 345).  Jobs of at least 256 x 256
        // points gain something whatever their number, since they are cut into more tiles (6 sets of 300, 8 classes
        // 172 / 186; 2 of 1,000, 5 classes 166 / 219).
        const long long n_jobs = (long long)jobs.size();
        auto rows_pay = [&](long long classes, long long bins, int least) {
            const long long words = n_slots * classes * classes * bins;
            const long long price = n_jobs * (classes - 1) * (150000 + 15000 * classes);
            return words * 8 <= (long long)Ctx::kCalcKeep && least * words <= pairs &&
                   price <= pairs + (pairs >= 65536 * n_jobs ? 72000000 : 0);
        };
        // by a sample of the points, which costs no launch (its classes and extent are lower bounds); more points
        // than the sample has seldom change the answer, so the exact numbers only bound it
        bool classify = false;
        {
            const int per_set = std::max(8, 256 / std::max(1, n_sets));  // (a cache miss each)
            std::vector<uint32_t> seen;
            double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
            for (int k = 0; k < n_sets && (int)seen.size() <= kMaxClasses; ++k) {
                const float4* q = staged.data() + sets[k].off;
                for (int i = 0; i < sets[k].n && (int)seen.size() <= kMaxClasses; i += 1 + sets[k].n / per_set) {
                    uint32_t w;
                    std::memcpy(&w, &q[i].w, 4);
                    if (std::find(seen.begin(), seen.end(), w) == seen.end()) seen.push_back(w);
                    const double v[3] = {q[i].x, q[i].y, q[i].z};
                    for (int d = 0; d < 3; ++d) lo[d] = std::min(lo[d], v[d]), hi[d] = std::max(hi[d], v[d]);
                }
            }
            const double extent = std::hypot(hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]);
            classify = !seen.empty() && (int)seen.size() <= kMaxClasses &&
                       rows_pay((long long)seen.size(), bin_span(extent, (float)(1.0 / bin_width), bin_count).bins, 6);
        }
        const size_t pts_bytes = align_up(std::max<size_t>(1, staged.size()) * 16, 256);
        size_t list_bytes = 256, jobs_bytes_in = 256, class_bytes = 256;
        if (classify) {
            for (const Set& q : sets) list_bytes += align_up(Structure::typed_bytes(q.n), 256);
            jobs_bytes_in = align_up(sizeof(TypedSetJob) * n_sets, 256);
            class_bytes = align_up(sizeof(WeightClasses) * n_sets, 256);
        }
        const size_t dense_bytes = classify ? pts_bytes : 256;
        in.ensure(pts_bytes + dense_bytes + list_bytes + jobs_bytes_in + class_bytes);
        DevBuf points, dense, lists, set_jobs, classes;
        points.view(in.p, pts_bytes);
        dense.view(in.as<char>(pts_bytes), dense_bytes);
        lists.view(in.as<char>(pts_bytes + dense_bytes), list_bytes);
        set_jobs.view(in.as<char>(pts_bytes + dense_bytes + list_bytes), jobs_bytes_in);
        classes.view(in.as<char>(pts_bytes + dense_bytes + list_bytes + jobs_bytes_in), class_bytes);
        AUSAXS_CUDA(cudaMemcpyAsync(points.p, staged.data(), staged.size() * 16, cudaMemcpyHostToDevice, s));
        const float4* P = points.as<float4>();
        int max_n = 0;
        std::vector<TypedSetJob> sj;
        std::vector<WeightClasses> wc;
        if (classify) {
            sj.resize(n_sets);
            wc.resize(n_sets);
            size_t list_at = 0;
            for (int k = 0; k < n_sets; ++k) {
                const int n = sets[k].n;
                char* mem = lists.as<char>(list_at);
                list_at += align_up(Structure::typed_bytes(n), 256);
                sj[k] = TypedSetJob{};
                sj[k].in = P + sets[k].off;
                sj[k].dense = dense.as<float4>() + sets[k].off;
                sj[k].counts = reinterpret_cast<int32_t*>(mem + typed_off_counts(n));
                sj[k].n = n;
                sj[k].out.pts = reinterpret_cast<float4*>(mem);
                sj[k].out.pre = reinterpret_cast<int32_t*>(mem + typed_off_pre(n));
                sj[k].out.pre_stride = typed_pre_stride(n);
                max_n = std::max(max_n, n);
                wc[k].clear();
            }
            // pageable sources: staged on return
            AUSAXS_CUDA(cudaMemcpyAsync(set_jobs.p, sj.data(), sizeof(TypedSetJob) * n_sets, cudaMemcpyHostToDevice, s));
            AUSAXS_CUDA(cudaMemcpyAsync(classes.p, wc.data(), sizeof(WeightClasses) * n_sets, cudaMemcpyHostToDevice, s));
            weight_classes_sets_launch(set_jobs.as<TypedSetJob>(), n_sets, max_n, classes.as<WeightClasses>(), s);
            C.check_launch("calculator weight classes");
        }
        // the largest pair distance: min(box diagonal, 2 x radius about the box centre) over all points
        double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        std::vector<double> radius(n_sets, 0.0);  // half the largest extent of every set
        for (int k = 0; k < n_sets; ++k) {
            double slo[3] = {INFINITY, INFINITY, INFINITY}, shi[3] = {-INFINITY, -INFINITY, -INFINITY};
            const float4* q = staged.data() + sets[k].off;
            for (int i = 0; i < sets[k].n; ++i) {
                const double v[3] = {q[i].x, q[i].y, q[i].z};
                for (int d = 0; d < 3; ++d) {
                    if (!std::isfinite(v[d])) throw Error{AUSAXS_ERR_ARGUMENT, "non-finite coordinate"};
                    slo[d] = std::min(slo[d], v[d]);
                    shi[d] = std::max(shi[d], v[d]);
                }
            }
            for (int d = 0; d < 3; ++d) {
                lo[d] = std::min(lo[d], slo[d]);
                hi[d] = std::max(hi[d], shi[d]);
                if (sets[k].n) radius[k] = std::max(radius[k], 0.5 * (shi[d] - slo[d]));
            }
        }
        double dmax = 0;
        if (!staged.empty()) {
            double d2 = 0, r2 = 0, c[3];
            for (int d = 0; d < 3; ++d) {
                d2 += (hi[d] - lo[d]) * (hi[d] - lo[d]);
                c[d] = 0.5 * (lo[d] + hi[d]);
            }
            for (const float4& p : staged) {
                const double e[3] = {p.x - c[0], p.y - c[1], p.z - c[2]};
                r2 = std::max(r2, e[0] * e[0] + e[1] * e[1] + e[2] * e[2]);
            }
            dmax = std::min(std::sqrt(d2), 2 * std::sqrt(r2)) * (1 + 1e-6) + 1e-3;
        }
        const float inv_w = (float)(1.0 / bin_width);
        const BinSpan span = bin_span(dmax, inv_w, bin_count);
        const int nb = span.bins;
        const bool covered = span.covered;
        // the classes of all sets together (ascending bit patterns): K.n 0 when there are more than kMaxClasses
        CalcClasses K{};
        TypeMap map;
        std::vector<TypedSet> typed(n_sets);
        if (classify) {
            AUSAXS_CUDA(cudaMemcpyAsync(wc.data(), classes.p, sizeof(WeightClasses) * n_sets, cudaMemcpyDeviceToHost, s));
            AUSAXS_CUDA(cudaStreamSynchronize(s));
            std::map<unsigned, int> found;
            std::vector<std::vector<std::pair<unsigned, int>>> of_set(n_sets);
            bool few = true;
            long long total = 0;
            for (int k = 0; k < n_sets; ++k) {
                few = wc[k].sorted(of_set[k]) && few;
                for (auto& f : of_set[k]) found[f.first] += f.second, total += f.second;
            }
            pair_sqrt_prepare(inv_w, nb);
            PackLaunch fit{};
            fit.nr = pack_sqrt_mode(inv_w, nb);
            fit.rows = fit.group_rows = (int)found.size();
            fit.group_sums = fit.offsets = 1;
            fit.bins = nb;
            fit.tile_j = kPackMaxTileJ;
            if (few && found.size() <= (size_t)kMaxClasses && rows_pay((long long)found.size(), nb, 3) && fit.nr > 0 &&
                pack_shape(fit) >= 0) {
                float m = 0;
                int most = 0;
                for (auto& f : found) {
                    map.bits[K.n] = f.first;
                    std::memcpy(&K.w[K.n], &f.first, 4);
                    m = std::max(m, std::fabs(K.w[K.n]));
                    most = std::max(most, f.second);
                    ++K.n;
                }
                map.classes = K.n;
                class_share = (double)most / total;
                const double p = (double)m * m;  // as weight_scale_launch
                int e = 0;
                if (p > 0) std::frexp(p, &e);
                K.wscale = std::ldexp(1.0f, std::min(60, 30 - e));
                for (int k = 0; k < n_sets; ++k) {
                    TypedSet& t = typed[k];
                    t.pts = sj[k].out.pts;
                    t.pre = sj[k].out.pre;
                    t.pre_stride = sj[k].out.pre_stride;
                    t.types = sj[k].out.types = K.n;
                    for (auto& f : of_set[k]) t.count[std::distance(found.begin(), found.find(f.first))] = f.second;
                    for (int i = 0, at = 0; i < K.n; ++i) {
                        t.start[i] = sj[k].out.start[i] = at;
                        at += t.count[i];
                    }
                }
            }
        }
        const int n_rows = K.n ? K.n * K.n : 1;  // count rows of a slot
        if (pairhist_launch_smem(1, nb, true, 512) > kPairSmemCap)
            throw Error{AUSAXS_ERR_CAPACITY, "too many distance bins for the on-chip histogram"};

        // device layout: per slot [cnt rows | ds | ws] (nb each), outputs, slot table, counters
        const size_t row = align_up((size_t)nb * 8, 256);
        const size_t slot_bytes = align_up((size_t)n_rows * nb * 8, 256) + 2 * row;
        const size_t acc_bytes = (size_t)n_slots * slot_bytes + 1024;
        acc.ensure(acc_bytes);
        AUSAXS_CUDA(cudaMemsetAsync(acc.p, 0, acc_bytes, s));
        char* ab = acc.as<char>();
        unsigned long long* counter = reinterpret_cast<unsigned long long*>(ab + (size_t)n_slots * slot_bytes);
        unsigned long long* overflow = counter + 4;
        float* wscale = reinterpret_cast<float*>(counter + 8);
        out.ensure((size_t)n_slots * 3 * nb * 8);
        if (!K.n) {
            weight_scale_launch(P, (int)staged.size(), P, 0, wscale, s);
            C.check_launch("calculator weight scale");
        }

        Plan plan;  // job-building view
        plan.T = 1;
        plan.nb = nb;
        plan.inv_w = inv_w;
        plan.c = (float)(1.0 / (double)inv_w);
        plan.scale = (float)(32768.0 / (double)plan.c * (1.0 - 1.0 / 256));
        plan.max_group_rows = 1;
        plan.weighted = 1;
        plan.row_share = class_share;
        const float4* D = K.n ? dense.as<float4>() : P;  // outer points carry their class
        auto by_class = [&](JobSpec& sp, int outer, int inner) {
            if (!K.n) return;
            sp.spread_bins = std::max(16, (int)(0.7 * (radius[outer] + radius[inner]) * inv_w));
            sp.rmode = kRowPair;
            sp.rows = n_rows;
            sp.t_out = K.n;
            sp.typed = &typed[inner];
            sp.wsum = nullptr;
        };
        std::vector<CalcSlot> table_h(n_slots);
        for (int k = 0; k < n_slots; ++k) {
            table_h[k].cnt = reinterpret_cast<unsigned long long*>(ab + (size_t)k * slot_bytes);
            table_h[k].ds = reinterpret_cast<unsigned long long*>(ab + (size_t)(k + 1) * slot_bytes - 2 * row);
            table_h[k].ws = reinterpret_cast<long long*>(ab + (size_t)(k + 1) * slot_bytes - row);
            table_h[k].diag_value = table_h[k].diag_count = 0;
            table_h[k].out = out.as<double>() + (size_t)k * 3 * nb;
        }
        int biggest = 0;
        for (const Job& j : jobs) {
            const Set& A = sets[j.a];
            if (j.b < 0) {
                // the diagonal: scaling * sum(float(w*w)) (SimpleCalculator.h:143-161)
                double tw = 0;
                for (int i = 0; i < A.n; ++i) {
                    const float w = staged[A.off + i].w;
                    tw += (double)(float)(w * w);
                }
                tw *= j.scaling;
                table_h[j.slot].diag_value += tw;
                table_h[j.slot].diag_count += (double)(uint32_t)tw;
                if (A.n < 2) continue;
                JobSpec sp{};
                sp.A = D + A.off;
                sp.B = P + A.off;
                sp.na = sp.nbp = A.n;
                sp.self = 1;
                sp.rmode = kRowSingle;
                sp.rows = 1;
                sp.counts = table_h[j.slot].cnt;
                sp.dsum = table_h[j.slot].ds;
                sp.wsum = table_h[j.slot].ws;
                sp.mult = j.scaling;
                by_class(sp, j.a, j.a);
                plan.specs.push_back(sp);
                biggest = std::max(biggest, A.n);
            } else {
                // enqueue_calculate_cross(data_1 = a, data_2 = b): b outer, a inner from 0
                const Set& B = sets[j.b];
                if (A.n == 0 || B.n == 0) continue;
                JobSpec sp{};
                sp.A = D + B.off;
                sp.na = B.n;
                sp.B = P + A.off;
                sp.nbp = A.n;
                sp.self = 0;
                sp.rmode = kRowSingle;
                sp.rows = 1;
                sp.counts = table_h[j.slot].cnt;
                sp.dsum = table_h[j.slot].ds;
                sp.wsum = table_h[j.slot].ws;
                sp.mult = j.scaling;
                by_class(sp, j.b, j.a);
                plan.specs.push_back(sp);
                biggest = std::max({biggest, A.n, B.n});
            }
        }
        const size_t table_bytes = align_up(sizeof(CalcSlot) * n_slots, 256);
        PackLaunch PL{};
        PackTable PT;
        int shape = 0, pack_grid = 0;
        if (K.n && !plan.specs.empty()) {
            AUSAXS_CUDA(cudaMemcpyAsync(set_jobs.p, sj.data(), sizeof(TypedSetJob) * n_sets, cudaMemcpyHostToDevice, s));
            typed_sets_launch(set_jobs.as<TypedSetJob>(), n_sets, max_n, map, s);
            C.check_launch("calculator typed lists");
            C.launches += 1;  // two kernels
            if (!choose_pack(plan, C.sm_count, PL, shape, pack_grid, PT, false))
                throw Error{AUSAXS_ERR_CAPACITY, "too many distance bins for the on-chip histogram"};
            const size_t jobs_bytes = sizeof(PackJob) * PT.jobs.size(), out_bytes = sizeof(void*) * PT.out.size();
            std::vector<char> bytes(table_bytes + jobs_bytes + out_bytes);
            std::memcpy(bytes.data(), table_h.data(), sizeof(CalcSlot) * n_slots);
            std::memcpy(bytes.data() + table_bytes, PT.jobs.data(), jobs_bytes);
            std::memcpy(bytes.data() + table_bytes + jobs_bytes, PT.out.data(), out_bytes);
            table.ensure(bytes.size());
            AUSAXS_CUDA(cudaMemcpyAsync(table.p, bytes.data(), bytes.size(), cudaMemcpyHostToDevice, s));
            PL.jobs = reinterpret_cast<const PackJob*>(table.as<char>(table_bytes));
            PL.out = reinterpret_cast<unsigned long long* const*>(table.as<char>(table_bytes + jobs_bytes));
            PL.tile_counter = counter;
            PL.overflow = overflow;
            PL.covered = covered;
            cudaEvent_t ev;
            C.time_begin(0, &ev);
            pack_launch(PL, shape, pack_grid, s);
            C.check_launch("calculator pairs");
            C.time_end(0, ev);
        } else {
            std::vector<PairJob> pj[3];
            long long tiles[3] = {0, 0, 0};
            int rows[3] = {1, 1, 1};
            const int tile = biggest >= 16384 ? 512 : 256;
            append_pair_jobs(plan, tile, false, pj, tiles, rows);
            table.ensure(table_bytes + align_up(sizeof(PairJob) * std::max<size_t>(1, pj[0].size()), 256));
            AUSAXS_CUDA(cudaMemcpyAsync(table.p, table_h.data(), sizeof(CalcSlot) * n_slots, cudaMemcpyHostToDevice, s));
            PairJob* jobs_dev = reinterpret_cast<PairJob*>(table.as<char>() + table_bytes);
            if (!pj[0].empty()) {
                AUSAXS_CUDA(cudaMemcpyAsync(jobs_dev, pj[0].data(), sizeof(PairJob) * pj[0].size(), cudaMemcpyHostToDevice, s));
                PairLaunch L{};
                L.jobs = jobs_dev;
                L.n_jobs = (int)pj[0].size();
                L.total_tiles = tiles[0];
                L.smem_rows = 1;
                L.smem_bins = nb;
                L.tile_counter = counter;
                L.overflow = overflow;
                L.weighted = 1;
                L.wscale = wscale;
                L.dreg = 0;
                L.inv_w = plan.inv_w;
                pair_sqrt_prepare(plan.inv_w, nb);
                const size_t smem = pairhist_launch_smem(1, nb, true, tile);
                const int per_sm = pairhist_ctas_per_sm(smem, tile, false, true);
                const int grid = (int)std::min<long long>((long long)C.sm_count * per_sm, std::max<long long>(1, tiles[0]));
                L.chunk = (int)std::max<long long>(1, std::min<long long>(8, tiles[0] / ((long long)grid * 8)));
                cudaEvent_t ev;
                C.time_begin(0, &ev);
                pairhist_launch(L, tile, grid, smem, s);
                C.check_launch("calculator pairs");
                C.time_end(0, ev);
            }
        }
        const int threads = 256;
        calc_finalize_kernel<<<dim3((unsigned)((nb + threads - 1) / threads), (unsigned)n_slots), threads, 0, s>>>(
            reinterpret_cast<const CalcSlot*>(table.p), nb, wscale, plan.c, plan.scale, K);
        C.check_launch("calculator finalize");
        unsigned long long of = 0;
        AUSAXS_CUDA(cudaMemcpyAsync(&of, overflow, 8, cudaMemcpyDeviceToHost, s));
        std::vector<double> packed((size_t)n_slots * 3 * nb);
        AUSAXS_CUDA(cudaMemcpyAsync(packed.data(), out.p, packed.size() * 8, cudaMemcpyDeviceToHost, s));
        AUSAXS_CUDA(cudaStreamSynchronize(s));
        for (size_t r = 0; r < (size_t)n_slots * 3; ++r)  // [slot][3][nb] -> [slot][3][bin_count]
            std::memcpy(results.data() + r * bin_count, packed.data() + r * nb, (size_t)nb * 8);
        pairs_last = pairs;
        clear();
        if (of)
            throw Error{AUSAXS_ERR_BIN_OVERFLOW, "pair distances beyond bin_count * bin_width; increase settings::axes::bin_count"};
    }

    // SimpleCalculator::run clears its jobs and merge ids (SimpleCalculator.h:278-282)
    void clear() {
        sets.clear();
        staged.clear();
        jobs.clear();
        ids[0].clear();
        ids[1].clear();
        slot_info.clear();
    }

    long long pairs_last = 0;
    double class_share = 1;
};

}  // namespace ausaxs_b200

using namespace ausaxs_b200;

struct ausaxs_gpu_calculator {
    Calculator impl;
};

extern "C" {

int ausaxs_gpu_calculator_create(ausaxs_gpu_ctx* ctx, double bin_width, int32_t bin_count, ausaxs_gpu_calculator** out) {
    return guarded([&] {
        if (!ctx || !out || !(bin_width > 0) || bin_count <= 0) throw Error{AUSAXS_ERR_ARGUMENT, "invalid argument"};
        *out = nullptr;
        auto* c = new ausaxs_gpu_calculator();
        c->impl.ctx = &ctx->impl;
        c->impl.bin_width = bin_width;
        c->impl.bin_count = bin_count;
        *out = c;
    });
}

int ausaxs_gpu_calculator_destroy(ausaxs_gpu_calculator* c) {
    return guarded([&] {
        if (!c) return;
        cudaStreamSynchronize(c->impl.ctx->stream);
        delete c;
    });
}

int ausaxs_gpu_calculator_enqueue_self(ausaxs_gpu_calculator* c, const float* points, int32_t n, int32_t scaling,
                                       int32_t merge_id, int32_t* result_index) {
    return guarded([&] {
        if (!c) throw Error{AUSAXS_ERR_ARGUMENT, "null calculator"};
        const int r = c->impl.enqueue(points, n, nullptr, 0, scaling, merge_id);
        if (result_index) *result_index = r;
    });
}

int ausaxs_gpu_calculator_enqueue_cross(ausaxs_gpu_calculator* c, const float* points_1, int32_t n_1,
                                        const float* points_2, int32_t n_2, int32_t scaling, int32_t merge_id,
                                        int32_t* result_index) {
    return guarded([&] {
        if (!c || (n_2 > 0 && !points_2)) throw Error{AUSAXS_ERR_ARGUMENT, "invalid argument"};
        // a cross job with an empty second set still creates its (empty) result
        static const float none[4] = {0, 0, 0, 0};
        const int r = c->impl.enqueue(points_1, n_1, points_2 ? points_2 : none, n_2, scaling, merge_id);
        if (result_index) *result_index = r;
    });
}

int ausaxs_gpu_calculator_run(ausaxs_gpu_calculator* c, int32_t* n_self, int32_t* n_cross) {
    return guarded([&] {
        if (!c) throw Error{AUSAXS_ERR_ARGUMENT, "null calculator"};
        AUSAXS_CUDA(cudaSetDevice(c->impl.ctx->device));
        c->impl.run();
        int ns = 0, nc = 0;
        for (auto& r : c->impl.result_info) (r.cross ? nc : ns) += 1;
        if (n_self) *n_self = ns;
        if (n_cross) *n_cross = nc;
    });
}

int ausaxs_gpu_calculator_result_ids(ausaxs_gpu_calculator* c, int32_t cross, int32_t* ids, int32_t capacity, int32_t* n) {
    return guarded([&] {
        if (!c || !n || (capacity > 0 && !ids)) throw Error{AUSAXS_ERR_ARGUMENT, "invalid argument"};
        std::vector<int> v;
        for (auto& r : c->impl.result_info)
            if (r.cross == (cross != 0)) v.push_back(r.merge_id);
        std::sort(v.begin(), v.end());
        *n = (int32_t)v.size();
        for (int k = 0; k < (int)v.size() && k < capacity; ++k) ids[k] = v[k];
    });
}

int ausaxs_gpu_calculator_result(ausaxs_gpu_calculator* c, int32_t cross, int32_t merge_id, double* value, double* count,
                                 double* distance_sum) {
    return guarded([&] {
        if (!c) throw Error{AUSAXS_ERR_ARGUMENT, "null calculator"};
        const auto& I = c->impl.result_info;
        const size_t nb = c->impl.bin_count;
        for (size_t k = 0; k < I.size(); ++k) {
            if (I[k].cross != (cross != 0) || I[k].merge_id != merge_id) continue;
            const double* r = c->impl.results.data() + k * 3 * nb;
            if (value) std::memcpy(value, r, nb * 8);
            if (count) std::memcpy(count, r + nb, nb * 8);
            if (distance_sum) std::memcpy(distance_sum, r + 2 * nb, nb * 8);
            return;
        }
        throw Error{AUSAXS_ERR_NOT_FOUND, "no result with this merge id in the last run"};
    });
}

}  // extern "C"
