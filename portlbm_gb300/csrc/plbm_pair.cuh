// plbm_pair.cuh — two timesteps of the two-lattice algorithms in one pass over memory, for the shifted
// forms (FP32 arithmetic) and F64_Q60, whose single steps of a large domain are bound by HBM and of a
// small one by the latency of a launch.
//
// A warp owns a strip of 30 columns and marches up `rows` rows of it.  At row r it pulls the first step's
// populations of its 32 columns from memory (the outermost two only feed their neighbours), collides
// them, and then has what the second step needs at row r - 1: directions 0-2 come from row r, 3-5 from
// row r - 1, 6-8 from row r - 2, the columns beside by shuffle, a bounced direction from the node's own
// values.  Only the second step's populations are written.  A lane keeps 12 values of the rows behind
// it, nothing goes through shared memory and no barrier is needed; the price is the first step of 2
// columns in 32 and of 2 rows a strip done twice.  The values are those of two single steps: each
// population is rounded to its storage type in between.
//
// Bound by instruction issue with HBM half busy: 48 registers for ten blocks of 128 (eight in the record
// layout, five for Q60) hide the loads better than fetching the next row ahead with 64 or 80 registers
// (f32 8192 x 8192: 143 k and 126 k MLUPS against 156 k).  Edge nodes share the interior's loads and
// take their ghost constants afterwards: with pull_one's gather of its own for them the f32 kernel
// spilled and took 84 us instead of 60 a step at 4000 x 1999.  Measured, single steps -> two-step
// launches, us a step: 8192 x 8192 f32 stream 708 -> 429, bundle 776 -> 413, records 764 -> 664, f16s
// 462 -> 391, bf16s 468 -> 391, f16c 645 -> 565, f64_q60 1414 -> 1222 (bundle 1465 -> 1223);
// 4000 x 1999 f32 93 -> 60, f16s 70 -> 59; 4096 x 4096 porous f32 267 -> 160, f16s 144 -> 128 (lptl
// records 248 -> 131), f16c 198 -> 180, f64_q60 433 -> 373.  Two nodes a lane with packed FP32
// instructions (64 columns a warp, every neighbour by shuffle) took 549 instructions a row instead of
// 315 for half the columns, and was slower.
#pragma once

#include "plbm_kernels.cuh"

namespace plbm {

constexpr int PAIR_WARPS = 4;        // warps of a block, each with a strip of its own
constexpr int PAIR_COLUMNS = 30;     // columns a warp writes

// The value a lane's population takes in memory between two steps (a rounding for 2-byte storage).
template <int PREC> __device__ __forceinline__ CT<PREC> stored_value(CT<PREC> v, const StepParams &p)
{
    if constexpr (PREC == F16S) return __half2float(__float2half_rn(v));
    else if constexpr (PREC == BF16S) return __bfloat162float(__float2bfloat16_rn(v));
    else if constexpr (PREC == F16C) {
        bool over;
        const unsigned b = f16c_bits(v, over);
        if (over) atomicOr(p.status, 1);
        return f16c_value(b);
    } else return v;
}

// What the outlet of the next step takes of this step's jy in column W - 2 (write_observables' jy_next):
// for F64_Q60 the value itself, for the shifted forms half of it in the form's own scale, an exact product
// as half_jy's.
__device__ __forceinline__ double outlet_jy(const Moments &m, const StepParams &p)
{
    const double v = q_to_double(__double_as_longlong(m.jy));
    return p.nan_protection ? nan_guard(v) : v;
}
__device__ __forceinline__ float outlet_jy(const MomentsF &m, const StepParams &p)
{
    const bool drop = p.nan_protection && !(m.jy <= 3.40282347e38f);   // NaN or above FLT_MAX
    return drop ? 0.0f : 0.5f * m.jy;
}

// Byte offsets in a lattice, all below 2^32 (the launch checks): node n's entry of direction d lies at
// n * STRIDE + plane(d) values.
template <int PREC, int L> struct PairIndex {
    static constexpr bool WIDE = sizeof(typename Store<PREC>::T) == 8;   // 8-byte storage: offsets in values
    static constexpr unsigned SIZE = WIDE ? 1u : sizeof(typename Store<PREC>::T);
    static constexpr unsigned STRIDE = SIZE * (L == COLLISION ? 9 : L == STREAM ? 1 : 3);
    __device__ static __forceinline__ unsigned plane(int d, unsigned N)
    {
        return SIZE * (L == COLLISION ? (unsigned)d : L == STREAM ? N * d : 3u * (d / 3) * N + d % 3);
    }
};

template <int PREC>
__device__ __forceinline__ CT<PREC> pair_load(const void *lattice, unsigned at, const StepParams &p)
{
    using T = typename Store<PREC>::T;
    constexpr bool wide = sizeof(T) == 8;
    if (!in_range(wide ? at : at / sizeof(T), p.lat_elems, p)) return CT<PREC>(0);
    const T v = wide ? static_cast<const T *>(lattice)[at]
                     : *reinterpret_cast<const T *>(static_cast<const char *>(lattice) + at);
    if constexpr (PREC == F16S) return __half2float(v);
    else if constexpr (PREC == BF16S) return __bfloat162float(v);
    else if constexpr (PREC == F16C) return f16c_value(v);
    else return v;
}

// Directions (bits) whose source lies beyond a domain edge: below / above, and left / right.
__device__ __forceinline__ unsigned ghosts_y(int y, const StepParams &p)
{
    return (y == 0 ? 0x1C0u : 0u) | (y == p.H - 1 ? 0x007u : 0u);
}
__device__ __forceinline__ unsigned ghosts_x(int x, const StepParams &p)
{
    return (x == 0 ? 0x124u : 0u) | (x == p.W - 1 ? 0x049u : 0u);
}
// Puts pull_one's ghost constants into an edge node's populations.
template <int PREC>
__device__ __forceinline__ void fill_ghosts(CT<PREC> f[9], int x, int y, const StepParams &p)
{
    const unsigned gy = ghosts_y(y, p), gx = ghosts_x(x, p);
#pragma unroll
    for (int d = 0; d < 9; ++d) {
        if (d == 4) continue;
        if constexpr (shifted<PREC>()) {
            if ((gy >> d) & 1u) f[d] = p.weightf[d] + p.shift_wg[d] * (float)x;
        } else {
            if ((gy >> d) & 1u) f[d] = g_weight<PREC>(p, d);
        }
        if (!((gy >> d) & 1u) && ((gx >> d) & 1u)) f[d] = x == 0 && cxd(d) == 1 ? g_in<PREC>(p, d) : g_out<PREC>(p, d);
    }
}

// The incoming populations of fluid node (xi, yi) from memory, re-referenced (at: the byte offset of its
// direction-0 entry without plane(0)).
template <int PREC, int L>
__device__ __forceinline__ void pair_gather(CT<PREC> g[9], unsigned at, int xi, int yi, uint16_t lk, const StepParams &p)
{
    using I = PairIndex<PREC, L>;
    const unsigned N = (unsigned)p.N, P = (unsigned)p.P;
    auto from = [&](int d) {
        const unsigned neighbour = at + (I::plane(d, N) - I::STRIDE * (unsigned)(cxd(d) + cyd(d) * (int)P));
        return d != 4 && ((lk >> d) & 1u) ? at + I::plane(8 - d, N) : neighbour;
    };
    if (!(lk & LINK_EDGE)) {
#pragma unroll
        for (int d = 0; d < 9; ++d) g[d] = pair_load<PREC>(p.lat0, from(d), p);
    } else {
        const unsigned ghost = ghosts_y(yi, p) | ghosts_x(xi, p);
#pragma unroll
        for (int d = 0; d < 9; ++d)
            if (!((ghost >> d) & 1u)) g[d] = pair_load<PREC>(p.lat0, from(d), p);
    }
    if constexpr (shifted<PREC>()) {
#pragma unroll
        for (int d = 0; d < 9; ++d)
            if (cxd(d) != 0 && !((lk >> d) & 1u)) g[d] += p.shift_cx[d];
    }
    if (lk & LINK_EDGE) fill_ghosts<PREC>(g, xi, yi, p);
}

// One warp's rows [ya, yb) of strip `strip` (at least one column of it in the domain).
template <int PREC, int L>
__device__ __forceinline__ void march_two_steps(const StepParams &p, int strip, int ya, int yb)
{
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x;
    const int xi = strip * PAIR_COLUMNS - 1 + lane;
    const bool inx = xi >= 0 && xi < p.W;
    const bool writes = inx && lane >= 1 && lane <= PAIR_COLUMNS;
    auto link = [&](int y) -> uint16_t {
        return inx && y >= 0 && y < p.H ? link_at(p, (unsigned)(xi + y * p.P)) : (uint16_t)0;
    };
    using I = PairIndex<PREC, L>;
    const unsigned row_bytes = I::STRIDE * (unsigned)p.P;
    unsigned at = I::STRIDE * (unsigned)(xi + (ya - 1) * p.P);     // of row r; wraps where nothing is read
    uint16_t lk_next = link(ya - 1), lk_prev = 0;
    step_begin();
    CT<PREC> b[9] = {}, c[3] = {};
    using J = typename std::conditional<PREC == F64_Q60, double, float>::type;
    J jyb = 0;
#pragma unroll 1
    for (int r = ya - 1; r <= yb; ++r, at += row_bytes) {
        CT<PREC> a[9] = {};
        const uint16_t lk = lk_next;
        lk_next = link(r + 1);
        // the first step's node (xi, r)
        J jya = 0;
        if (lk & LINK_FLUID) {
            pair_gather<PREC, L>(a, at, xi, r, lk, p);
            if (is_outlet_row(xi, r, p)) outlet_fill<PREC>(a, jy_prev_at(p, r), p);
            const auto m = collide<PREC>(a, p);
#pragma unroll
            for (int d = 0; d < 9; ++d) a[d] = stored_value<PREC>(a[d], p);
            if (PREC != F64_Q60 || xi == p.W - 2) jya = outlet_jy(m, p);
        }
        // the second step's node (xi, r - 1): its sources are rows r - 2 (c), r - 1 (b) and r (a)
        const int y = r - 1;
        if (y >= ya) {
            CT<PREC> f[9];
            f[0] = __shfl_down_sync(ALL, a[0], 1);
            f[1] = a[1];
            f[2] = __shfl_up_sync(ALL, a[2], 1);
            f[3] = __shfl_down_sync(ALL, b[3], 1);
            f[4] = b[4];
            f[5] = __shfl_up_sync(ALL, b[5], 1);
            f[6] = __shfl_down_sync(ALL, c[0], 1);
            f[7] = c[1];
            f[8] = __shfl_up_sync(ALL, c[2], 1);
            const J hy = __shfl_up_sync(ALL, jyb, 1);   // of column W - 2, where xi is the outlet
            if (writes && (lk_prev & LINK_FLUID)) {
                if constexpr (shifted<PREC>()) {
#pragma unroll
                    for (int d = 0; d < 9; ++d)
                        if (cxd(d) != 0) f[d] += p.shift_cx[d];
                }
                if (lk_prev != LINK_FLUID) {
#pragma unroll
                    for (int d = 0; d < 9; ++d)
                        if (d != 4 && ((lk_prev >> d) & 1u)) f[d] = b[8 - d];
                    if (lk_prev & LINK_EDGE) {
                        fill_ghosts<PREC>(f, xi, y, p);
                        if (is_outlet_row(xi, y, p)) {
                            if constexpr (PREC == F64_Q60) outlet_fill<PREC>(f, hy, p);
                            else outlet_fill_float(f, hy, p);
                        }
                    }
                }
                const auto m = collide<PREC>(f, p);
#pragma unroll
                for (int d = 0; d < 9; ++d) {
                    using T = typename Store<PREC>::T;
                    const unsigned to = at - row_bytes;
                    if (!in_range((I::plane(d, (unsigned)p.N) + (unsigned long long)to) / I::SIZE, p.lat_elems, p)) continue;
                    if constexpr (I::WIDE) static_cast<T *>(p.lat1)[I::plane(d, (unsigned)p.N) + to] = f[d];
                    else {
                        char *plane = static_cast<char *>(p.lat1) + I::plane(d, (unsigned)p.N);
                        *reinterpret_cast<T *>(plane + to) = encode_value<PREC>(f[d], p);
                    }
                }
                emit_observables<PREC>(m, xi, y, p);
            }
        }
        c[0] = b[6]; c[1] = b[7]; c[2] = b[8];
#pragma unroll
        for (int d = 0; d < 9; ++d) b[d] = a[d];
        lk_prev = lk;
        jyb = jya;
    }
}

// Launch bounds (blocks an SM) of the two-step kernels.
template <int PREC, int L> struct PairBlocks { static constexpr int value = PREC == F64_Q60 ? 5 : L == COLLISION ? 8 : 10; };

template <int PREC, int L>
__global__ void __launch_bounds__(32 * PAIR_WARPS, PairBlocks<PREC, L>::value) k_two_steps(StepParams p, int rows)
{
    const int strip = blockIdx.x * PAIR_WARPS + threadIdx.y;
    if (strip * PAIR_COLUMNS >= p.W) return;   // warp-uniform
    const int ya = blockIdx.y * rows;
    march_two_steps<PREC, L>(p, strip, ya, min(ya + rows, p.H));
}

}  // namespace plbm
