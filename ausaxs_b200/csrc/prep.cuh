// Point-set preparation kernels (see prep.cu).
#pragma once
#include <utility>
#include <vector>

#include <string.h>
#include "common.cuh"

namespace ausaxs_b200 {

// The distinct weights of a point set and their points, by bit pattern: a hashed table with open addressing, so
// that blocks meet in few of its slots.  Up to kMaxClasses of them are used; a table of more is of no use.
constexpr int kMaxClasses = 15;
constexpr int kClassSlots = 32;
constexpr unsigned kNoClass = 0xffffffffu;  // an empty slot (a NaN pattern)
struct WeightClasses {
    unsigned bits[kClassSlots];
    int count[kClassSlots];
    int over;  // some block met more than kMaxClasses (or kNoClass itself)
    void clear();
    // the weights in ascending order of their bit patterns, and their points; false: more than kMaxClasses
    bool sorted(std::vector<std::pair<unsigned, int>>& out) const;
};

struct PrepStats {
    unsigned int lo[3];  // order-preserving encodings of the bounding box
    unsigned int hi[3];
    unsigned int mask;   // bit t set: form-factor type t present
    unsigned int bad;    // bit 0: invalid form-factor type, bit 1: non-finite coordinate
    int count[kNff];     // atoms per form-factor type
    unsigned long long r2;  // bits of max |p - c|^2 (double) over every point, c = centre of the box
    WeightClasses weights[2];  // weighted structures: atoms, waters
};

// classes: the points' distinct weights are added to it (cleared before); may be null
void census_launch(const float4* p, int n, int ff_typed, PrepStats* st, WeightClasses* classes, int sm_count, cudaStream_t s);
// After the census launches on the same stream: the radius of the points about the box centre
// (every pair distance is at most twice it).
void radius_launch(const float4* a, int na, const float4* w, int nw, const float4* x, int nx, PrepStats* st,
                   int sm_count, cudaStream_t s);

// Lists of a point set by type: the points of dense type t at pts[start[t] ...] in ascending index, w =
// the index (int bits); pre[t * pre_stride + c] = points of type t with an index below kTypedPre * c.
constexpr int kTypedChunk = 1024;
constexpr int kTypedPre = 256;
struct TypedOut {
    float4* pts;
    int32_t* pre;
    int32_t* pos;        // position of every point in pts, or null
    int32_t types;
    int32_t pre_stride;  // typed_pre_stride(n)
    int32_t start[16];
};
inline int typed_chunks(int n) { return (n + kTypedChunk - 1) / kTypedChunk; }
inline int typed_pre_stride(int n) { return (n + kTypedPre - 1) / kTypedPre; }
// dense (w = dense type through the map; in already dense: no map and null) and the lists, two kernels;
// counts: typed_chunks(n) * 16 ints of scratch
struct TypeMap {
    const int32_t* ff_to_type = nullptr;  // form-factor type -> dense type
    int classes = 0;                      // or the index of w's bit pattern among these
    unsigned bits[16] = {};
};
void typed_lists_launch(const float4* in, float4* dense, int n, const TypeMap& map, const TypedOut& o, int32_t* counts,
                        cudaStream_t s);
// the same for many sets, and their classes (device tables; max_n >= every n)
struct TypedSetJob {
    const float4* in;
    float4* dense;
    int32_t* counts;
    int32_t n;
    TypedOut out;
};
void weight_classes_sets_launch(const TypedSetJob* sets_dev, int sets, int max_n, WeightClasses* out, cudaStream_t s);
void typed_sets_launch(const TypedSetJob* sets_dev, int sets, int max_n, const TypeMap& map, cudaStream_t s);
void set_type_launch(float4* p, int n, int32_t value, int sm_count, cudaStream_t s);
float ordered_to_float(unsigned int o);

}  // namespace ausaxs_b200
