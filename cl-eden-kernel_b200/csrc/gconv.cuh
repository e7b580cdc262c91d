// Gather convolution: one launch (transposed convolutions of stride 4 and more: several) for every dense contraction whose A operand cannot be read in place (taps, strides,
// dilation, zero-point borders, rows whose byte pitch is no multiple of 16, the parity classes of a transposed convolution).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"
#include "tc_common.cuh"

namespace enn_b200 {

constexpr int kGcMaxClasses = 9;        // of one launch: strides up to 3

// Quotient by an invariant divisor for dividends below 2^31: q = umulhi(n, mul) >> shift, with mul = ceil(2^(31 + s) / d) and
// shift = s - 1 for s = ceil(log2 d), d > 1 (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994); divisor 1 is mul == 0.
struct FastDiv {
    uint32_t mul = 0, shift = 0;
    __host__ static FastDiv make(uint32_t d) {
        FastDiv f;
        if (d <= 1) return f;
        uint32_t s = 0;
        while ((1ull << s) < d) ++s;
        f.mul = static_cast<uint32_t>(((1ull << (31 + s)) + d - 1) / d);
        f.shift = s - 1;
        return f;
    }
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return mul ? __umulhi(n, mul) >> shift : n; }
};

// One GEMM of the launch: a convolution has one, a transposed convolution one per output parity class.
struct GcClass {
    int32_t unit0;              // first work unit (units of a class: M tiles x N tiles, N fastest)
    int32_t M, tiles_m;
    int32_t k_blocks, ks_last;  // K slices (1, 2 or 4) of the last k-block
    int32_t tab0;               // first entry of the class in the gather table
    int32_t b_tile0;            // resident weights: first (N tile, k-block) of the class
    int32_t oh, ow;             // output grid: row m = (image, oy, ox)
    int32_t y0, x0;             // input position of tap (0, 0) for output (0, 0)
    FastDiv div_ow, div_img;    // by ow and by oh * ow
    int64_t out_base;
};

struct GcParams {
    int32_t n_classes, n_units;
    int32_t N, tiles_n, bn_rows, bn_data;
    int32_t stages;             // pipeline depth
    int32_t n_acc;              // accumulator buffers (1 or 2)
    int32_t tmem_cols;
    int32_t b_res;              // all weights stay in shared memory
    int32_t b_bytes;            // one (N tile, k-block) of weights
    int32_t tab_entries;        // gather table entries (all classes) staged in shared memory, kBK / unit per k-block; 0: read in global memory
    int32_t unit, unit_log2;    // bytes of the reduction per table entry: the largest of 16, 8 and 4 that divides the channels
    int32_t gran;               // bytes per gather copy: unit, or less where the input pointer is not a multiple of it (1: byte by byte)
    int32_t cols_all;           // 1: the constants of every column are staged once
    int32_t need_asum, zw_eff, a_signed, act_min, act_max, out_zp, mode, sat_plain;
    uint32_t idesc;
    int32_t h, w, cin, sy, sx;
    const int2 *tab;            // {byte offset from the row's first position, dy << 16 | dx}
    const ColParam *cols;       // [class][tiles_n][bn_rows]
    const uint8_t *in;
    const uint8_t *fill_src;    // kBK bytes of the input zero point, a line of their own
    uint8_t *out;
    int64_t out_sn, out_sy, out_sx;
    int32_t *err;
    int32_t test_starve;
    int32_t add_on, add_swap;
    AddParams add;
    const uint8_t *add_res;
    GcClass cls[kGcMaxClasses];
};

struct GcPlan {
    GcParams prm{};
    CUtensorMap map_b{};
    void *w_dev = nullptr, *cols_dev = nullptr, *tab_dev = nullptr;
    size_t smem_bytes = 0;
    uint32_t b_res_bytes = 0;   // resident weights
    int grid = 0;
    int per_sm = 2;             // CTAs the shared memory is laid out for
    size_t gather_bytes = 0;    // what the gathered matrix would take: the allocation-free call's limit, which no kernel's choice moves
};

// Geometry of one class for the planner; row m = (image, oy, ox), column k = (ky * kw + kx) * cin + c, input pixel
// iy = oy * sy + ky * dy + y0, ix = ox * sx + kx * dx + x0.
struct GcClassDesc {
    int32_t oh, ow, kh, kw, dy, dx, y0, x0;
    int64_t out_base;
};

constexpr uint32_t kGcSmemLimit = 113 * 1024, kGcSmemAlone = 227 * 1024;      // two CTAs per SM, one
constexpr int kGcMaxStages = 8;

uint32_t gconv_smem_bytes(const GcParams &p, uint32_t b_res_bytes);
cudaError_t gconv_launch(const GcPlan &plan, const GcParams &prm, cudaStream_t stream);      // prm: the plan's, completed by the call
cudaError_t gconv_init(int device);      // with `device` current

}  // namespace enn_b200
