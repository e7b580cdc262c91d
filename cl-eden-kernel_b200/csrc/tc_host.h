// Host side shared by the planners of the tensor-core kernels: tensor maps, and the derivation of the per-column epilogue
// constants from weights, bias and requantisation parameters.
#pragma once
#include <cuda.h>

#include <cstring>
#include <vector>

#include "internal.h"
#include "tc_common.cuh"

namespace enn_b200 {
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline CUtensorMapSwizzle swizzle_of(uint32_t span) {
    return span == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (span == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

inline bool encode_2d(enn_b200_context *ctx, CUtensorMap *map, const void *base, uint64_t inner, uint64_t outer, uint64_t pitch,
                      uint32_t box_inner, uint32_t box_outer) {
    EncodeTiledFn fn = reinterpret_cast<EncodeTiledFn>(ctx->encode_tiled);
    if (!fn) return false;
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {pitch};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_of(box_inner), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

struct QuantHost {   // host copies of what setup_quant uploaded
    std::vector<int32_t> mult, shift, bias;
};

// Per-column facts the epilogue constants follow from: the folded bias bias'[n] and a bound on |accumulator + bias'|.
struct ColumnFold {
    int64_t folded = 0, bound = 0;
};

// wsum / wabs: sum and sum of absolute values of the column's signed weight bytes over its K reduction indices.
inline ColumnFold fold_column(const ConvGeom &g, int64_t bias, int64_t K, int64_t wsum, int64_t wabs, int64_t zw_eff) {
    const int64_t amax = g.a_signed ? 128 : 255;
    ColumnFold f;
    f.folded = bias - static_cast<int64_t>(g.in_zp) * wsum + K * g.in_zp * zw_eff;
    f.bound = amax * wabs + K * amax * (zw_eff < 0 ? -zw_eff : zw_eff) + (f.folded < 0 ? -f.folded : f.folded);
    return f;
}

// The cheapest epilogue mode every column allows (folds[i] belongs to output channel i % N).
inline int32_t column_mode(const enn_b200_context *ctx, const ConvGeom &g, const QuantHost &qh, const std::vector<ColumnFold> &folds, int32_t N,
                           bool allow_relu) {
    const int64_t zo_eff = static_cast<int64_t>(g.out_zp) - g.act_min;
    // ReLU-type outputs (lower clamp == output zero point): can every column use the merged form?
    bool relu_hi = zo_eff == 0 && allow_relu && !ctx->opt("no_relu_mode"), relu_two = relu_hi;
    for (size_t i = 0; i < folds.size() && relu_two; ++i) {
        const size_t n = i % static_cast<size_t>(N);
        const int32_t sh = qh.shift[n];
        const int32_t ls = sh > 0 ? sh : 0, e = sh > 0 ? 0 : -sh;
        const bool in_range = folds[i].folded <= INT32_MAX && folds[i].folded >= INT32_MIN && folds[i].bound < (1ll << 31) && qh.mult[n] >= 0;
        if (!in_range || ls > 30 || e > 31) relu_hi = relu_two = false;
        if (ls > 0 || e < 1) relu_hi = false;
        // two-shift form: the left-shifted accumulator must not wrap (the reference multiplies in int32) and the
        // stage-1 value plus the rounding term must fit 32 bits
        if ((folds[i].bound << ls) + (e >= 1 ? (1ll << (e - 1)) : 0) + 1 >= (1ll << 31)) relu_two = false;
    }
    return relu_hi && !ctx->opt("no_relu_hi") ? kModeReluHi : (relu_two ? kModeReluTwo : kModeNudge);
}

// Constants of one column for `mode`.  Returns false when a two-stage column needs the general code (the operator's mode
// is then kModeGeneral; the constants written stay valid for it).
inline bool column_constants(const ConvGeom &g, int32_t mode, int32_t mult, int32_t shift, const ColumnFold &f, ColParam *c) {
    const int64_t zo_eff = static_cast<int64_t>(g.out_zp) - g.act_min;
    if (mode == kModeReluHi || mode == kModeReluTwo) {
        const int32_t ls = shift > 0 ? shift : 0, e = shift > 0 ? 0 : -shift;
        int64_t cc = f.folded * mult;
        int32_t word;
        if (mode == kModeReluHi) {
            cc += (1ll << 30) + (1ll << (30 + e));
            word = e - 1;
        } else {
            const int32_t s1 = 31 - ls;
            cc += (1ll << (30 - ls)) + (e >= 1 ? (1ll << (e - 1 + s1)) : 0);
            word = s1 | (e << 8);
        }
        c->mult = static_cast<int32_t>(static_cast<uint32_t>(static_cast<uint64_t>(cc) & 0xffffffffu));   // word 0: C low
        c->addend = static_cast<int32_t>(static_cast<uint32_t>(static_cast<uint64_t>(cc) >> 32));            // word 1: C high
        c->esh = mult;                                                                                     // word 2: M0
        c->bias = word;                                                                                    // word 3: shifts
        return true;
    }
    c->mult = mult;
    c->bias = static_cast<int32_t>(f.folded);      // wraps like the reference's int32 accumulation
    const int32_t e = shift > 0 ? -1 : -shift;
    const int64_t addend = e > 0 ? (1ll << (e - 1)) + zo_eff * (1ll << e) : zo_eff;
    if (e < 1 || f.folded > INT32_MAX || f.folded < INT32_MIN || f.bound + 2 + (addend < 0 ? -addend : addend) >= (1ll << 31)) {
        c->addend = shift;                         // general path keeps the raw signed shift
        c->esh = INT32_MIN;
        return false;
    }
    c->addend = static_cast<int32_t>(addend);
    c->esh = e;
    return true;
}

// kModeReluHi whose clamp is the whole unsigned byte: the saturating pack of the epilogue does it (kModeReluSat).
inline bool column_sat_plain(const enn_b200_context *ctx, const ConvGeom &g, int32_t mode) {
    return mode == kModeReluHi && !g.a_signed && g.act_min == 0 && g.act_max >= 255 && !ctx->opt("no_relu_sat");
}

}  // namespace
}  // namespace enn_b200
