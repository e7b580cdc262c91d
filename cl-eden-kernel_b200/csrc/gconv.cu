// gconv_kernel: gather convolution on the tensor cores, one launch per operator (transposed convolutions of stride 4 and more: one per
// nine parity classes).
//
// Two CTAs per SM, or one (build_gconv says where), each warp-specialised:
//   warps 0..3  epilogue: tcgen05.ld, requantisation, stores (quad form, tc_common.cuh: four rows of the same columns per thread)
//   warps 4..7  gather: the A tile of a k-block (128 output pixels x 128 reduction bytes) is fetched from the NHWC tensor with
//               16-byte asynchronous copies, or 8-, 4- or 1-byte loads, straight into the 128-byte-swizzled operand layout; positions outside
//               the image are stored as the input zero point
//   warp 8      TMEM allocation, MMA issue
//   warp 9      TMA copies of the packed weights (once per CTA when they fit, else per k-block)
//
// Why a gather by ordinary threads and not tensor copies: a tensor copy of an im2col tile costs several cycles per pixel row
// whatever the row's length (a 3x3 layer over 64 channels fetches nine 64-byte rows per output pixel), cannot fill borders
// with a zero point other than 0, and needs rows whose pitch is a multiple of 16 bytes.  The threads address any geometry
// through a table of (offset, dy, dx) per copy, the nine-fold re-reads of a 3x3 window hit the L1, the reduction is
// packed densely (tap-major, no padding per tap) and no zero-point padded or gathered copy of the input is written first.
//
// Every wait is bounded (tc_common.cuh): on expiry an error code reaches the host and all roles fall through to the exit.
#include "gconv.cuh"
#include "per_device.h"

#include <type_traits>

namespace enn_b200 {
namespace {

constexpr int kEpiWarpsGc = 4, kGatherWarps = 4;
constexpr int kGatherThreads = 32 * kGatherWarps;
constexpr int kMmaWarp = kEpiWarpsGc + kGatherWarps, kBWarp = kMmaWarp + 1;
constexpr int kGcThreads = 32 * (kBWarp + 1);
constexpr int kRowTabBytes = kBM * 16;          // {64-bit address, iy, ix} of the 32 rows each gather warp fetches

template <int OFF>
__device__ __forceinline__ void cp_async16(uint32_t dst, const uint8_t *src) {
    asm volatile("cp.async.ca.shared.global [%0 + %2], [%1], 16;" ::"r"(dst), "l"(src), "n"(OFF) : "memory");
}
// Arrives on the barrier (counted in its initial value) once all copies this thread has started so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
template <int OFF>
__device__ __forceinline__ void st_shared(uint32_t dst, const uint2 &v) {
    asm volatile("st.shared.v2.b32 [%0 + %3], {%1, %2};" ::"r"(dst), "r"(v.x), "r"(v.y), "n"(OFF) : "memory");
}
template <int OFF>
__device__ __forceinline__ void st_shared(uint32_t dst, uint32_t v) {
    asm volatile("st.shared.b32 [%0 + %2], %1;" ::"r"(dst), "r"(v), "n"(OFF) : "memory");
}
// One entry of the row table.
__device__ __forceinline__ void load_row(uint32_t addr, const uint8_t *&row, int &iy, int &ix) {
    uint32_t lo, hi;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(lo), "=r"(hi), "=r"(iy), "=r"(ix) : "r"(addr));
    asm("mov.b64 %0, {%1, %2};" : "=l"(row) : "r"(lo), "r"(hi));
}
// f(integral_constant<int, i>) for i = 0 .. N - 1, unrolled.
template <int I, int N, typename F>
__device__ __forceinline__ void static_for(F &&f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(static_cast<F &&>(f));
    }
}

// Shared-memory layout behind the 1024-byte aligned base: weights (resident) | stages (A [, B]) | columns | gather table |
// row table | fused-add tables | barriers.
struct GcSmem {
    uint32_t b_res, stages, cols, tab, rows, add, bars, total;
};
__host__ __device__ inline GcSmem gc_smem(const GcParams &p, uint32_t b_res_bytes, uint32_t col_entries) {
    GcSmem s;
    s.b_res = 0;
    s.stages = b_res_bytes;
    s.cols = s.stages + static_cast<uint32_t>(p.stages) * (kBM * kBK + (p.b_res ? 0u : static_cast<uint32_t>(p.b_bytes)));
    s.tab = s.cols + col_entries * 16;
    s.rows = s.tab + ((static_cast<uint32_t>(p.tab_entries) * 8 + 15) & ~15u);
    s.add = s.rows + kRowTabBytes;
    s.bars = s.add + (p.add_on ? 2048u : 0u);
    s.total = s.bars + (2 * kGcMaxStages + 6) * 8 + 16;
    return s;
}

// Walks the unit numbers of one CTA; (class, M tile, N tile) of the current unit.
struct UnitWalk {
    int unit, c, tm, tn;
    __device__ __forceinline__ void start(int u) {
        unit = u;
        c = 0;
    }
    __device__ __forceinline__ bool locate(const GcParams &p) {
        if (unit >= p.n_units) return false;
        while (c + 1 < p.n_classes && unit >= p.cls[c + 1].unit0) ++c;
        const int t = unit - p.cls[c].unit0;
        if (p.tiles_n == 1) {
            tm = t;
            tn = 0;
        } else {
            tm = t / p.tiles_n;
            tn = t - tm * p.tiles_n;
        }
        return true;
    }
};

// The gather role: this thread's copies of every k-block of every unit.
//   G == 16  asynchronous 16-byte copies that report to the stage's barrier by themselves (every thread is one of its
//            arrivals), so that as many k-blocks are in flight as there are stages.  Border positions copy from a constant
//            block of zero-point bytes, which leaves no branch and no store of the thread's own.  The MMA thread orders
//            the copies before its reads (fence.proxy.async after the barrier): issued here, that fence would wait for
//            every copy in flight (about 1000 cycles per k-block, measured).
//   G < 16   8- or 4-byte loads into registers, all of a k-block in flight, then stores, fence, one arrival per warp.
//            Asynchronous copies of 8 bytes took 27 SM cycles per warp instruction (16 bytes: 10), loads and stores 4 to 6.
//   BYTES    4-byte words put together from single bytes: inputs at odd addresses.
template <int G, bool BYTES = false>
__device__ __forceinline__ void gather_role(const GcParams &p, const GcSmem &L, const uint8_t *sp, uint32_t base, uint32_t full0, uint32_t empty0,
                                            volatile int *abort_flag, bool starve) {
    constexpr int kPerRow = kBK / G;                            // copies per A row and k-block: 8, 16 or 32
    constexpr int kRowsPerPass = kGatherThreads / kPerRow;      // 16, 8 or 4
    constexpr int kPasses = kBM / kRowsPerPass;                 // 8, 16 or 32
    static_assert(kRowsPerPass >= 4, "two swizzle terms per thread at most");
    const int t = static_cast<int>(threadIdx.x) - 32 * kEpiWarpsGc, lane = t & 31;
    const int piece = t % kPerRow, row0 = t / kPerRow;
    // Destination of (row, piece) in the swizzled tile.  Rows of a thread are kRowsPerPass apart: for 16 and 8 of them the
    // swizzle term (row & 7) is one constant, for 4 it alternates between two, and the rest of the address is an immediate.
    const uint32_t chunk16 = static_cast<uint32_t>(piece * G) >> 4, in16 = static_cast<uint32_t>(piece * G) & 15u;
    const uint32_t dst0 = static_cast<uint32_t>(row0) * kBK + ((chunk16 ^ static_cast<uint32_t>(row0 & 7)) << 4) + in16;
    const uint32_t dst1 = static_cast<uint32_t>(row0 + 4) * kBK + ((chunk16 ^ static_cast<uint32_t>((row0 + 4) & 7)) << 4) + in16;
    // A row's lanes copy a border position from the line of zero points each at its own place, as they would an inside one: lanes that
    // all copied the same 16 bytes were served one after another (1x28x28x512 -> 512, whose last M tile has 16 real rows of 128:
    // 31.2 -> 15.1 us; 1x56x56x64 -> 64 5.9 -> 4.6; 256x56x56x64 -> 64 72.3 -> 70.9).
    // A copy smaller than a table entry's unit reads the entry of its unit, a few bytes further on.
    const int unit_log2 = G == 16 ? 4 : p.unit_log2, per_kb = kBK >> unit_log2;
    const int first = (piece * G) >> unit_log2, sub = (piece * G) & ((1 << unit_log2) - 1);
    const uint8_t *fill_src = p.fill_src + piece * G;
    const uint32_t h = static_cast<uint32_t>(p.h), w = static_cast<uint32_t>(p.w);
    const uint32_t stage_bytes = kBM * kBK + (p.b_res ? 0u : static_cast<uint32_t>(p.b_bytes));
    // A warp fetches kRowsPerWarp rows per pass, 32 rows per tile: the lanes work them out and leave them in the warp's table.
    constexpr int kRowsPerWarp = 32 / kPerRow;                  // 4, 2 or 1
    const int wbase = (t >> 5) * kRowsPerWarp;
    const uint32_t rt = base + L.rows + static_cast<uint32_t>(t >> 5) * 512u, rt_lane = rt + static_cast<uint32_t>(lane / kPerRow) * 16;
    const int2 *const tab0 = (p.tab_entries ? reinterpret_cast<const int2 *>(sp + L.tab) : p.tab) + first;
    uint32_t stage = 0, phase = 0;
    bool ok = !starve, waited = false;
    UnitWalk u;
    for (u.start(static_cast<int>(blockIdx.x)); ok && u.locate(p); u.unit += gridDim.x) {
        const GcClass &c = p.cls[u.c];
        __syncwarp();
        {
            const int r = wbase + lane % kRowsPerWarp + kRowsPerPass * (lane / kRowsPerWarp);
            const uint32_t m = static_cast<uint32_t>(u.tm * kBM + r);
            const uint8_t *row = p.in;              // 64-bit: an input may be larger than 4 GiB
            int iy = INT32_MIN / 2, ix = 0;         // rows beyond the class: outside whatever the tap
            if (m < static_cast<uint32_t>(c.M)) {
                const uint32_t img = c.div_img.div(m), rem = m - img * static_cast<uint32_t>(c.oh * c.ow);
                const uint32_t oy = c.div_ow.div(rem), ox = rem - oy * static_cast<uint32_t>(c.ow);
                iy = static_cast<int>(oy) * p.sy + c.y0;
                ix = static_cast<int>(ox) * p.sx + c.x0;
                const int pixel = (static_cast<int>(img) * p.h + iy) * p.w + ix;     // fits (build_gconv)
                row += static_cast<int64_t>(pixel) * p.cin;
            }
            const uint64_t addr = reinterpret_cast<uint64_t>(row);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rt + lane * 16), "r"(static_cast<uint32_t>(addr)), "r"(static_cast<uint32_t>(addr >> 32)), "r"(iy), "r"(ix) : "memory");
        }
        __syncwarp();
        if (!waited) {
            pdl_wait();
            waited = true;
        }
        const uint8_t *rrow[G == 16 ? kPasses : 1];
        int riy[G == 16 ? kPasses : 1], rix[G == 16 ? kPasses : 1];
        if (G == 16) {
#pragma unroll
            for (int i = 0; i < kPasses; ++i) load_row(rt_lane + i * kRowsPerWarp * 16, rrow[i], riy[i], rix[i]);
        }
        const int2 *tab = tab0 + c.tab0;
        for (int kb = 0; kb < c.k_blocks; ++kb) {
            const int2 entry = *tab;        // ahead of the wait, which hides the load (7x7 over 8x14x14x1024, 392 k-blocks: 178 -> 138 us)
            tab += per_kb;
            if (lane == 0) ok = mbar_test_wait(empty0 + 8 * stage, phase ^ 1) || mbar_wait_fast(empty0 + 8 * stage, phase ^ 1, abort_flag, p.err, 1);
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            const int toff = entry.x + sub, tyx = entry.y;
            const int dy = tyx >> 16, dx = static_cast<int16_t>(tyx & 0xffff);
            const uint32_t a0 = base + L.stages + stage * stage_bytes;
            // dy == INT16_MIN: beyond the reduction, meets zero weights whatever it holds
            if constexpr (G == 16) {
                if (dy != INT16_MIN)
                    static_for<0, kPasses>([&](auto tag) {
                        constexpr int i = decltype(tag)::value;
                        const bool inside = static_cast<uint32_t>(riy[i] + dy) < h && static_cast<uint32_t>(rix[i] + dx) < w;
                        cp_async16<i * kRowsPerPass * kBK>(a0 + dst0, inside ? rrow[i] + toff : fill_src);
                    });
                cp_async_arrive(full0 + 8 * stage);
            } else {
                using Word = std::conditional_t<G == 8, uint2, uint32_t>;
                constexpr int kPart = BYTES ? 8 : kPasses;      // loads in flight: all of the k-block, or what the registers hold
                if (dy != INT16_MIN) {
                    if constexpr (BYTES) {
#pragma unroll 1
                        for (int part = 0; part < kPasses; part += kPart) {
                            Word v[kPart];
#pragma unroll
                            for (int i = 0; i < kPart; ++i) {
                                const uint8_t *row;
                                int iy, ix;
                                load_row(rt_lane + (part + i) * kRowsPerWarp * 16, row, iy, ix);
                                const bool inside = static_cast<uint32_t>(iy + dy) < h && static_cast<uint32_t>(ix + dx) < w;
                                const uint8_t *src = inside ? row + toff : fill_src;
                                v[i] = __ldg(src) | __ldg(src + 1) << 8 | __ldg(src + 2) << 16 | static_cast<uint32_t>(__ldg(src + 3)) << 24;
                            }
#pragma unroll
                            for (int i = 0; i < kPart; ++i)
                                st_shared<0>(a0 + (i & 1 ? dst1 : dst0) + static_cast<uint32_t>(part + (i & ~1)) * kRowsPerPass * kBK, v[i]);
                        }
                    } else {
                        Word v[kPasses];
                        static_for<0, kPasses>([&](auto tag) {
                            constexpr int i = decltype(tag)::value;
                            const uint8_t *row;
                            int iy, ix;
                            load_row(rt_lane + i * kRowsPerWarp * 16, row, iy, ix);
                            const bool inside = static_cast<uint32_t>(iy + dy) < h && static_cast<uint32_t>(ix + dx) < w;
                            v[i] = __ldg(reinterpret_cast<const Word *>(inside ? row + toff : fill_src));
                        });
                        static_for<0, kPasses>([&](auto tag) {
                            constexpr int i = decltype(tag)::value;
                            if constexpr (kRowsPerPass == 4) st_shared<(i & ~1) * kRowsPerPass * kBK>(a0 + (i & 1 ? dst1 : dst0), v[i]);
                            else st_shared<i * kRowsPerPass * kBK>(a0 + dst0, v[i]);
                        });
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full0 + 8 * stage);
            }
            if (++stage == static_cast<uint32_t>(p.stages)) { stage = 0; phase ^= 1; }
        }
    }
    if (G == 16) asm volatile("cp.async.wait_all;" ::: "memory");
}

template <bool ASUM, int MODE, bool FADD>
__global__ void __launch_bounds__(kGcThreads, 2) gconv_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ GcParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023) & ~1023u;
    uint8_t *sp = smem_raw + (base - raw);
    uint32_t b_res_bytes = 0;
    if (p.b_res) {
        const GcClass &lc = p.cls[p.n_classes - 1];
        b_res_bytes = static_cast<uint32_t>(lc.b_tile0 + p.tiles_n * lc.k_blocks) * static_cast<uint32_t>(p.b_bytes);
    }
    const uint32_t col_entries = static_cast<uint32_t>(p.cols_all ? p.n_classes * p.tiles_n * p.bn_rows : p.bn_rows);
    const GcSmem L = gc_smem(p, b_res_bytes, col_entries);
    const int nst = p.stages;
    const uint32_t full0 = base + L.bars, empty0 = full0 + 8 * nst, tfull0 = empty0 + 8 * nst, tempty0 = tfull0 + 16, bres_bar = tempty0 + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sp + L.bars + (2 * nst + 5) * 8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool starve = p.test_starve != 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < nst; ++s) {
            mbar_init(full0 + 8 * s, (p.gran == 16 ? kGatherThreads : kGatherWarps) + (p.b_res ? 0 : 1));
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull0 + 8 * b, 1);
            mbar_init(tempty0 + 8 * b, kEpiWarpsGc);
        }
        mbar_init(bres_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) tmem_alloc(smem_u32(tmem_slot), static_cast<uint32_t>(p.tmem_cols));
    if (p.cols_all)
        for (uint32_t i = threadIdx.x; i < col_entries; i += kGcThreads) reinterpret_cast<int4 *>(sp + L.cols)[i] = __ldg(reinterpret_cast<const int4 *>(p.cols) + i);
    for (int i = threadIdx.x; i < p.tab_entries; i += kGcThreads) reinterpret_cast<int2 *>(sp + L.tab)[i] = __ldg(p.tab + i);
    FaddCtx fadd{};
    if (FADD) {
        fadd.lut_u32 = base + L.add;
        fadd.mo = p.add.mo; fadd.so = p.add.so; fadd.out_off = p.add.out_off; fadd.act_min = p.add.act_min; fadd.act_max = p.add.act_max;
        fadd.swap = p.add_swap != 0;
        for (int i = threadIdx.x; i < 512; i += kGcThreads) reinterpret_cast<int32_t *>(sp + L.add)[i] = __ldg(p.add.lut + i);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Weights are constants of the plan: resident ones are fetched ahead of the wait on the kernel before.
    if (p.b_res && warp == kBWarp && lane == 0 && !starve) {
        mbar_expect_tx(bres_bar, b_res_bytes);
        for (int c = 0; c < p.n_classes; ++c)
            for (int tn = 0; tn < p.tiles_n; ++tn)
                for (int kb = 0; kb < p.cls[c].k_blocks; ++kb)
                    tma_load_2d(base + static_cast<uint32_t>(p.cls[c].b_tile0 + tn * p.cls[c].k_blocks + kb) * p.b_bytes, &map_b, bres_bar, kb * kBK,
                                (c * p.tiles_n + tn) * p.bn_rows);
    }
    // The gather warps wait for the kernel before once they have worked out the rows of their first unit (1x56x56x64 -> 64 4.5 -> 4.1 us,
    // 16x28x28x72 -> 200 pointwise 6.15 -> 5.6).
    if (warp < kEpiWarpsGc || warp >= kMmaWarp) {
        pdl_wait();
        pdl_trigger();
    }

    const uint32_t stage_bytes = kBM * kBK + (p.b_res ? 0u : static_cast<uint32_t>(p.b_bytes));
    if (warp >= kEpiWarpsGc && warp < kMmaWarp) {
        if (p.gran == 16) gather_role<16>(p, L, sp, base, full0, empty0, abort_flag, starve);
        else if (p.gran == 8) gather_role<8>(p, L, sp, base, full0, empty0, abort_flag, starve);
        else if (p.gran == 4) gather_role<4>(p, L, sp, base, full0, empty0, abort_flag, starve);
        else gather_role<4, true>(p, L, sp, base, full0, empty0, abort_flag, starve);
    } else if (warp == kBWarp) {
        if (!p.b_res && lane == 0 && !starve) {
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            UnitWalk u;
            for (u.start(static_cast<int>(blockIdx.x)); ok && u.locate(p); u.unit += gridDim.x) {
                const int kbs = p.cls[u.c].k_blocks, row = (u.c * p.tiles_n + u.tn) * p.bn_rows;
                for (int kb = 0; kb < kbs; ++kb) {
                    if (!mbar_test_wait(empty0 + 8 * stage, phase ^ 1) && !mbar_wait_fast(empty0 + 8 * stage, phase ^ 1, abort_flag, p.err, 1)) { ok = false; break; }
                    mbar_expect_tx(full0 + 8 * stage, static_cast<uint32_t>(p.b_bytes));
                    tma_load_2d(base + L.stages + stage * stage_bytes + kBM * kBK, &map_b, full0 + 8 * stage, kb * kBK, row);
                    if (++stage == static_cast<uint32_t>(nst)) { stage = 0; phase ^= 1; }
                }
            }
            if (!ok) drain_stages(full0, nst, stage, phase);
        } else if (p.b_res && lane == 0 && !starve) {
            for (uint32_t i = 0; i < (1u << 12); ++i)        // the MMA role may have given up before they landed
                if (mbar_try_wait(bres_bar, 0)) break;
        }
    } else if (warp == kMmaWarp) {
        if (lane == 0) {
            const uint32_t looks = starve ? 64u : (kSpinLimit >> 7);
            const uint32_t desc_hi = static_cast<uint32_t>(make_smem_desc(0) >> 32);
            uint32_t stage = 0, phase = 0, it = 0;
            bool ok = true;
            if (p.b_res && !mbar_wait_fast(bres_bar, 0, abort_flag, p.err, 5, looks)) ok = false;
            UnitWalk u;
            for (u.start(static_cast<int>(blockIdx.x)); ok && u.locate(p); u.unit += gridDim.x, ++it) {
                const uint32_t ab = p.n_acc == 2 ? (it & 1) : 0, use = p.n_acc == 2 ? (it >> 1) : it;
                if (!mbar_wait_fast(tempty0 + 8 * ab, (use & 1) ^ 1, abort_flag, p.err, 2, looks)) { ok = false; break; }
                tc_fence_after();
                const GcClass &c = p.cls[u.c];
                const uint32_t d = tmem_base + ab * p.bn_rows;
                uint32_t lo_res = (base + static_cast<uint32_t>(c.b_tile0 + u.tn * c.k_blocks) * p.b_bytes) >> 4;
                for (int kb = 0; kb < c.k_blocks; ++kb) {
                    if (!mbar_test_wait(full0 + 8 * stage, phase) && !mbar_wait_fast(full0 + 8 * stage, phase, abort_flag, p.err, 3, looks)) { ok = false; break; }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    tc_fence_after();
                    const uint32_t lo = (base + L.stages + stage * stage_bytes) >> 4;
                    const uint32_t lo_b = p.b_res ? lo_res : lo + ((kBM * kBK) >> 4);
                    lo_res += static_cast<uint32_t>(p.b_bytes) >> 4;
                    const int ks = kb + 1 == c.k_blocks ? c.ks_last : 4;
                    if (ks == 4) umma_i8_run<false, 4>(d, desc_hi, lo, lo_b, p.idesc, kb != 0);
                    else if (ks == 2) umma_i8_run<false, 2>(d, desc_hi, lo, lo_b, p.idesc, kb != 0);
                    else umma_i8_run<false, 1>(d, desc_hi, lo, lo_b, p.idesc, kb != 0);
                    umma_commit(empty0 + 8 * stage);
                    if (++stage == static_cast<uint32_t>(nst)) { stage = 0; phase ^= 1; }
                }
                if (ok) umma_commit(tfull0 + 8 * ab);
            }
        }
    } else {
        // ---------------- epilogue ----------------
        int64_t st_bits = p.out_sn | p.out_sy | p.out_sx | p.bn_data | static_cast<int64_t>(reinterpret_cast<uintptr_t>(p.out));
        for (int c = 0; c < p.n_classes; ++c) st_bits |= p.cls[c].out_base;
        const EpiArgs e = epi_args(p, st_bits, FADD ? p.add_res - p.out : 0, fadd);
        EpiTile t;
        int loaded = -1;
        uint32_t it = 0;
        bool ok = true;
        UnitWalk u;
        for (u.start(static_cast<int>(blockIdx.x)); u.locate(p) && (ok || !p.cols_all); u.unit += gridDim.x, ++it) {
            const GcClass &c = p.cls[u.c];
            const uint32_t ab = p.n_acc == 2 ? (it & 1) : 0, use = p.n_acc == 2 ? (it >> 1) : it;
            const int ct = u.c * p.tiles_n + u.tn;
            if (!p.cols_all && ct != loaded) {
                // Also where the four warps agree to go on: a warp whose wait ran out reports it here, so that none of the
                // others is left at the barrier.
                uint32_t all_ok;
                asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.red.and.pred q, 2, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                             : "=r"(all_ok) : "r"(ok ? 1 : 0), "n"(32 * kEpiWarpsGc) : "memory");
                if (!all_ok) break;
                for (int i = threadIdx.x; i < p.bn_rows; i += 32 * kEpiWarpsGc)
                    reinterpret_cast<int4 *>(sp + L.cols)[i] = __ldg(reinterpret_cast<const int4 *>(p.cols) + static_cast<size_t>(ct) * p.bn_rows + i);
                asm volatile("bar.sync 2, %0;" ::"n"(32 * kEpiWarpsGc) : "memory");
                loaded = ct;
            }
            const uint8_t *cols = sp + L.cols + (p.cols_all ? ct * p.bn_rows * 16 : 0);
            // Lane l works out where row l of the warp's quarter starts; a thread then takes its four rows from the lanes.
            const int n_base = u.tn * p.bn_data;
            t.n_left = min(p.bn_data, p.N - n_base);
            {
                const uint32_t m = static_cast<uint32_t>(u.tm * kBM + warp * 32 + lane);
                int64_t off = -1;
                if (m < static_cast<uint32_t>(c.M)) {
                    const uint32_t img = c.div_img.div(m), rem = m - img * static_cast<uint32_t>(c.oh * c.ow);
                    const uint32_t oy = c.div_ow.div(rem), ox = rem - oy * static_cast<uint32_t>(c.ow);
                    off = c.out_base + n_base + img * p.out_sn + oy * p.out_sy + ox * p.out_sx;
                }
                t.live = 0;
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int64_t o = __shfl_sync(0xffffffffu, off, (lane >> 2) + 8 * h);
                    t.live |= o >= 0 ? 1u << h : 0u;
                    t.row[h] = p.out + o;
                }
            }
            if (ok) ok = mbar_wait(tfull0 + 8 * ab, use & 1, abort_flag, p.err, 4);
            if (!ok) continue;
            tc_fence_after();
            const uint32_t t_row = tmem_base + ab * p.bn_rows + (static_cast<uint32_t>(warp * 32) << 16);
            if (ASUM) epi_asum(t_row, p.bn_data, p.zw_eff, lane, t.asum);
            epi_tile<MODE, ASUM, FADD>(t_row, 0, 1, p.bn_data, t, lane, e, [&](int) { return cols; });
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty0 + 8 * ab);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kMmaWarp) tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
}

template <bool ASUM, int MODE, bool FADD = false>
cudaError_t launch_one(const GcPlan &plan, const GcParams &p, cudaStream_t s) {
    return launch_pdl(gconv_kernel<ASUM, MODE, FADD>, dim3(static_cast<unsigned>(plan.grid)), dim3(kGcThreads), plan.smem_bytes, s, plan.map_b, p);
}
template <bool ASUM>
cudaError_t launch_mode(const GcPlan &plan, const GcParams &p, cudaStream_t s) {
    if (p.add_on) return p.mode == kModeNudge ? launch_one<ASUM, kModeNudge, true>(plan, p, s) : launch_one<ASUM, kModeGeneral, true>(plan, p, s);
    switch (p.mode) {
        case kModeNudge: return launch_one<ASUM, kModeNudge>(plan, p, s);
        case kModeGeneral: return launch_one<ASUM, kModeGeneral>(plan, p, s);
        case kModeReluHi: return p.sat_plain ? launch_one<ASUM, kModeReluSat>(plan, p, s) : launch_one<ASUM, kModeReluHi>(plan, p, s);
        default: return launch_one<ASUM, kModeReluTwo>(plan, p, s);
    }
}
template <bool ASUM, int MODE, bool FADD = false>
cudaError_t set_attr() {
    return cudaFuncSetAttribute(gconv_kernel<ASUM, MODE, FADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGcSmemAlone);
}
template <bool ASUM>
cudaError_t set_attrs() {
    cudaError_t e = set_attr<ASUM, kModeNudge>();
    if (e == cudaSuccess) e = set_attr<ASUM, kModeGeneral>();
    if (e == cudaSuccess) e = set_attr<ASUM, kModeReluHi>();
    if (e == cudaSuccess) e = set_attr<ASUM, kModeReluTwo>();
    if (e == cudaSuccess) e = set_attr<ASUM, kModeReluSat>();
    if (e == cudaSuccess) e = set_attr<ASUM, kModeNudge, true>();
    if (e == cudaSuccess) e = set_attr<ASUM, kModeGeneral, true>();
    return e;
}

}  // namespace

uint32_t gconv_smem_bytes(const GcParams &p, uint32_t b_res_bytes) {
    const uint32_t cols = static_cast<uint32_t>(p.cols_all ? p.n_classes * p.tiles_n * p.bn_rows : p.bn_rows);
    return gc_smem(p, b_res_bytes, cols).total + 1024;       // 1024: alignment of the tiles
}

cudaError_t gconv_init(int device) {
    static PerDeviceInit once;
    return once.run(device, [] {
        const cudaError_t e = set_attrs<false>();
        return e == cudaSuccess ? set_attrs<true>() : e;
    });
}

cudaError_t gconv_launch(const GcPlan &plan, const GcParams &p, cudaStream_t s) { return p.need_asum ? launch_mode<true>(plan, p, s) : launch_mode<false>(plan, p, s); }

}  // namespace enn_b200
