// runtime.cu -- aether_runtime_eval: the runtime-typed strided evaluator.
//
// Follows eval/Runtime.h:73-300 of the reference: out = op(a, b, scalar) for
// every element of out's logical shape (rank <= 6, double or float), each
// operand addressed through its own element strides, the flat element index
// running row-major over out's extents. Ops: Assign (copy or double<->float
// cast), Add, Sub, Scale (s*a), AddScaled (a + s*b), SubScaled (a - s*b); the
// scalar is rounded to the input type first (Runtime.h:221). Every add and
// multiply rounds on its own (no contraction), so results equal the
// reference's host loop bit for bit.
//
// Three kernels per (op, input type, output type):
//  * contiguous: all operands row-major with no gaps -> flat indices,
//    four elements per thread with 128-bit accesses when every base is
//    16-byte aligned;
//  * tiled: any other strides with rows long enough. x is the axis along which
//    out is densest, so stores coalesce; an input that is dense along another
//    axis y (a transpose) is read along y and turned in shared memory;
//  * strided: short rows. Each thread decodes its first flat index into a
//    multi-index with invariant-divisor division (ag_fastdiv.cuh), then walks
//    four consecutive elements by carrying the multi-index.
// All are grid-stride loops; the flat ones run a few CTAs per SM, the tiled one a
// CTA per tile.

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>

#include "aether_gb300.h"
#include "ag_fastdiv.cuh"

int ag_internal_fail(const char* message);

namespace {

constexpr int kRun = 4;        // elements per thread per step
constexpr int kBlock = 256;

struct RtDesc {
    const void* a;
    const void* b;
    void* o;
    int rank;
    uint32_t total;
    AgFastDiv ext[AETHER_RT_RANK_CAP];
    int64_t sa[AETHER_RT_RANK_CAP], sb[AETHER_RT_RANK_CAP], so[AETHER_RT_RANK_CAP];
    double scalar;
};

__device__ __forceinline__ double rt_add(double x, double y) { return __dadd_rn(x, y); }
__device__ __forceinline__ float rt_add(float x, float y) { return __fadd_rn(x, y); }
__device__ __forceinline__ double rt_sub(double x, double y) { return __dsub_rn(x, y); }
__device__ __forceinline__ float rt_sub(float x, float y) { return __fsub_rn(x, y); }
__device__ __forceinline__ double rt_mul(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ float rt_mul(float x, float y) { return __fmul_rn(x, y); }
template <class TO>
__device__ __forceinline__ TO rt_cast(double x);
template <>
__device__ __forceinline__ double rt_cast<double>(double x) { return x; }
template <>
__device__ __forceinline__ float rt_cast<float>(double x) { return __double2float_rn(x); }
template <class TO>
__device__ __forceinline__ TO rt_cast(float x) { return TO(x); }

template <int OP, class TI, class TO>
__device__ __forceinline__ TO rt_apply(TI a, TI b, TI s) {
    if (OP == AETHER_RT_ASSIGN) return rt_cast<TO>(a);
    if (OP == AETHER_RT_ADD) return TO(rt_add(a, b));
    if (OP == AETHER_RT_SUB) return TO(rt_sub(a, b));
    if (OP == AETHER_RT_SCALE) return TO(rt_mul(s, a));
    if (OP == AETHER_RT_ADD_SCALED) return TO(rt_add(a, rt_mul(s, b)));
    return TO(rt_sub(a, rt_mul(s, b)));
}

__host__ __device__ constexpr bool uses_b(int op) {
    return op == AETHER_RT_ADD || op == AETHER_RT_SUB || op == AETHER_RT_ADD_SCALED || op == AETHER_RT_SUB_SCALED;
}

// 4 consecutive elements at 16-byte aligned addresses.
template <class T>
struct Quad;
template <>
struct Quad<double> {
    static __device__ __forceinline__ void load(const double* p, double v[4]) {
        const double2 x = __ldcs(reinterpret_cast<const double2*>(p));
        const double2 y = __ldcs(reinterpret_cast<const double2*>(p) + 1);
        v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
    }
    static __device__ __forceinline__ void store(double* p, const double v[4]) {
        __stcs(reinterpret_cast<double2*>(p), make_double2(v[0], v[1]));
        __stcs(reinterpret_cast<double2*>(p) + 1, make_double2(v[2], v[3]));
    }
};
template <>
struct Quad<float> {
    static __device__ __forceinline__ void load(const float* p, float v[4]) {
        const float4 x = __ldcs(reinterpret_cast<const float4*>(p));
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    }
    static __device__ __forceinline__ void store(float* p, const float v[4]) {
        __stcs(reinterpret_cast<float4*>(p), make_float4(v[0], v[1], v[2], v[3]));
    }
};

template <int OP, class TI, class TO, bool VEC>
__global__ void __launch_bounds__(kBlock) rt_contiguous(RtDesc d) {
    const TI* A = static_cast<const TI*>(d.a);
    const TI* B = static_cast<const TI*>(d.b);
    TO* O = static_cast<TO*>(d.o);
    const TI s = TI(d.scalar);
    const uint64_t total = d.total;
    const uint64_t step = uint64_t(gridDim.x) * kBlock * kRun;
    for (uint64_t base = (uint64_t(blockIdx.x) * kBlock + threadIdx.x) * kRun; base < total; base += step) {
        if (VEC && base + kRun <= total) {
            TI va[4], vb[4] = {TI(0), TI(0), TI(0), TI(0)};
            TO vo[4];
            Quad<TI>::load(A + base, va);
            if (uses_b(OP)) Quad<TI>::load(B + base, vb);
#pragma unroll
            for (int j = 0; j < 4; ++j) vo[j] = rt_apply<OP, TI, TO>(va[j], vb[j], s);
            Quad<TO>::store(O + base, vo);
        } else {
            for (int j = 0; j < kRun && base + j < total; ++j) {
                const TI x = A[base + j];
                const TI y = uses_b(OP) ? B[base + j] : TI(0);
                O[base + j] = rt_apply<OP, TI, TO>(x, y, s);
            }
        }
    }
}

template <int OP, class TI, class TO>
__global__ void __launch_bounds__(kBlock) rt_strided(RtDesc d) {
    const TI* A = static_cast<const TI*>(d.a);
    const TI* B = static_cast<const TI*>(d.b);
    TO* O = static_cast<TO*>(d.o);
    const TI s = TI(d.scalar);
    const int rank = d.rank;
    const uint64_t total = d.total;
    const uint64_t step = uint64_t(gridDim.x) * kBlock * kRun;
    for (uint64_t base = (uint64_t(blockIdx.x) * kBlock + threadIdx.x) * kRun; base < total; base += step) {
        uint32_t idx[AETHER_RT_RANK_CAP];
        int64_t oa = 0, ob = 0, oo = 0;
        uint32_t rem = uint32_t(base);
        for (int k = rank - 1; k >= 0; --k) {
            uint32_t q, r;
            ag_fastdiv_divmod(rem, d.ext[k], q, r);
            idx[k] = r;
            rem = q;
            oa += int64_t(r) * d.sa[k];
            if (uses_b(OP)) ob += int64_t(r) * d.sb[k];
            oo += int64_t(r) * d.so[k];
        }
        for (int j = 0; j < kRun && base + j < total; ++j) {
            const TI x = A[oa];
            const TI y = uses_b(OP) ? B[ob] : TI(0);
            O[oo] = rt_apply<OP, TI, TO>(x, y, s);
            // next flat index: carry the multi-index
            for (int k = rank - 1; k >= 0; --k) {
                oa += d.sa[k];
                if (uses_b(OP)) ob += d.sb[k];
                oo += d.so[k];
                if (++idx[k] < d.ext[k].d) break;
                idx[k] = 0;
                oa -= int64_t(d.ext[k].d) * d.sa[k];
                if (uses_b(OP)) ob -= int64_t(d.ext[k].d) * d.sb[k];
                oo -= int64_t(d.ext[k].d) * d.so[k];
            }
        }
    }
}

// One tile of x and y at a time, the other axes decoded once per tile. Bound by
// HBM: 24 bytes an element for f64 with two inputs. Without a turned input a
// tile is 8 rows of 128, each warp one row, or one row of 1024; with one it is
// 32 x 32, 33 words a row in shared memory so that neither the row nor the
// column access conflicts.
// Reads keep their lines in L2 (a row's last sector is the next tile's first):
// 135 us against 142 with evict-first reads. Measured, a + s b over 96 x 509 x
// 515 f64 with b's axes permuted: 275 us in the strided kernel (every read of
// b a sector of its own), 111 here, 5.5 TB/s. Tiles of 64 rows took 128.
struct RtTile {
    const void* a;
    const void* b;
    void* o;
    uint32_t nx, ny;                 // extents of x and y
    int64_t xa, xb, xo, ya, yb, yo;  // element strides along them
    AgFastDiv tx, ty;                // tiles along x, along y
    uint32_t tiles;
    int flat;                        // a tile is one row of 1024: the warps follow one another along x
    int rest;                        // the other axes, innermost first
    AgFastDiv ext[AETHER_RT_RANK_CAP];
    int64_t sa[AETHER_RT_RANK_CAP], sb[AETHER_RT_RANK_CAP], so[AETHER_RT_RANK_CAP];
    double scalar;
};

template <class T, bool TURN, int TX>
__device__ __forceinline__ void rt_fetch(const T* p, int64_t sx, int64_t sy, uint32_t x0, uint32_t y0,
                                         uint32_t nx, uint32_t ny, int lane, int warp, int row, T* buf, T v[4]) {
    if (TURN) {   // lanes along y; element (x, y) of the tile goes to buf[33 x + y]
        const uint32_t y = y0 + lane;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t x = x0 + warp + 8 * j;
            if (x < nx && y < ny) buf[33 * (warp + 8 * j) + lane] = __ldg(p + int64_t(x) * sx + int64_t(y) * sy);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t x = x0 + lane + (TX == 128 ? 32 * j : 0), y = y0 + row + (TX == 128 ? 0 : 8 * j);
            v[j] = x < nx && y < ny ? __ldg(p + int64_t(x) * sx + int64_t(y) * sy) : T(0);
        }
    }
}

template <int OP, class TI, class TO, bool TA, bool TB>
__global__ void __launch_bounds__(kBlock) rt_tiled(RtTile d) {
    constexpr int TX = TA || TB ? 32 : 128, TY = TA || TB ? 32 : 8;
    __shared__ TI ba[TA ? 32 * 33 : 1], bb[TB ? 32 * 33 : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const TI s = TI(d.scalar);
    for (uint32_t t = blockIdx.x; t < d.tiles; t += gridDim.x) {
        uint32_t q, ix, iy;
        ag_fastdiv_divmod(t, d.tx, q, ix);
        ag_fastdiv_divmod(q, d.ty, q, iy);
        int64_t oa = 0, ob = 0, oo = 0;
        for (int k = 0; k < d.rest; ++k) {
            uint32_t r;
            ag_fastdiv_divmod(q, d.ext[k], q, r);
            oa += int64_t(r) * d.sa[k];
            if (uses_b(OP)) ob += int64_t(r) * d.sb[k];
            oo += int64_t(r) * d.so[k];
        }
        const bool flat = TX == 128 && d.flat;
        const uint32_t x0 = flat ? ix * 1024 + warp * 128 : ix * TX, y0 = iy * TY;
        const int row = flat ? 0 : warp;
        TI va[4], vb[4] = {TI(0), TI(0), TI(0), TI(0)};
        rt_fetch<TI, TA, TX>(static_cast<const TI*>(d.a) + oa, d.xa, d.ya, x0, y0, d.nx, d.ny, lane, warp, row, ba, va);
        if (uses_b(OP))
            rt_fetch<TI, TB, TX>(static_cast<const TI*>(d.b) + ob, d.xb, d.yb, x0, y0, d.nx, d.ny, lane, warp, row, bb, vb);
        if (TA || TB) {
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (TA) va[j] = ba[33 * lane + row + 8 * j];
                if (TB) vb[j] = bb[33 * lane + row + 8 * j];
            }
        }
        TO* O = static_cast<TO*>(d.o) + oo;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t x = x0 + lane + (TX == 128 ? 32 * j : 0), y = y0 + row + (TX == 128 ? 0 : 8 * j);
            if (x < d.nx && y < d.ny) __stcs(O + int64_t(x) * d.xo + int64_t(y) * d.yo, rt_apply<OP, TI, TO>(va[j], vb[j], s));
        }
        if (TA || TB) __syncthreads();   // the buffers are filled again
    }
}

// The axes of a tiled evaluation, or false where the strided kernel is the
// better one: where fewer than a quarter of a tile's lanes would have an
// element (the strided kernel gives every lane four), or rows along x are
// shorter than half a warp.
constexpr uint32_t kTileRow = 16;

bool rt_plan_tiles(const RtDesc& d, bool ub, RtTile& t, bool& turn_a, bool& turn_b) {
    // axes of extent 1 say nothing; from the outermost of out inwards,
    // neighbours that every operand walks as one axis become one
    int order[AETHER_RT_RANK_CAP], m = 0;
    for (int k = 0; k < d.rank; ++k) {
        if (d.ext[k].d == 1) continue;
        int i = m++;
        for (; i > 0 && d.so[order[i - 1]] < d.so[k]; --i) order[i] = order[i - 1];
        order[i] = k;
    }
    uint32_t ext[AETHER_RT_RANK_CAP];
    int64_t sa[AETHER_RT_RANK_CAP], sb[AETHER_RT_RANK_CAP], so[AETHER_RT_RANK_CAP];
    int n = 0;
    for (int i = 0; i < m; ++i) {
        const int k = order[i];
        const uint32_t e = d.ext[k].d;
        if (n && sa[n - 1] == d.sa[k] * int64_t(e) && so[n - 1] == d.so[k] * int64_t(e) &&
            (!ub || sb[n - 1] == d.sb[k] * int64_t(e))) {
            ext[n - 1] *= e, sa[n - 1] = d.sa[k], sb[n - 1] = d.sb[k], so[n - 1] = d.so[k];
            continue;
        }
        ext[n] = e, sa[n] = d.sa[k], sb[n] = d.sb[k], so[n] = d.so[k], ++n;
    }
    if (n == 0) return false;
    // the axis along which an operand is densest (stride 0 repeats an element)
    auto densest = [&](const int64_t* s) {
        int best = n - 1;
        for (int k = n - 1; k >= 0; --k)
            if (s[k] > 0 && (s[best] <= 0 || s[k] < s[best])) best = k;
        return best;
    };
    const int x = densest(so);
    if (ext[x] < kTileRow) return false;
    auto turned = [&](const int64_t* s) {   // the axis to read along instead of x, or -1
        const int k = densest(s);
        return k != x && s[k] > 0 && s[x] > s[k] && ext[k] >= kTileRow ? k : -1;
    };
    auto filled = [](uint32_t e, uint32_t tile) {   // share of the tiles' lanes with an element
        return double(e) / (double((uint64_t(e) + tile - 1) / tile) * tile);
    };
    const int ya = turned(sa), yb = ub ? turned(sb) : -1;
    int y = ya >= 0 ? ya : yb;
    turn_a = ya >= 0;
    turn_b = yb >= 0 && yb == y;
    const bool turn = turn_a || turn_b;
    double share = turn ? filled(ext[x], 32) * filled(ext[y], 32) : filled(ext[x], 1024);
    t.flat = turn ? 0 : 1;
    for (int k = n - 1; !turn && k >= 0; --k) {
        if (k == x || filled(ext[x], 128) * filled(ext[k], 8) <= share) continue;
        share = filled(ext[x], 128) * filled(ext[k], 8);
        y = k;
        t.flat = 0;
    }
    if (share < 0.25) return false;
    const uint32_t TX = turn ? 32 : t.flat ? 1024 : 128, TY = turn ? 32 : 8;
    t.a = d.a, t.b = d.b, t.o = d.o, t.scalar = d.scalar;
    t.nx = ext[x], t.xa = sa[x], t.xb = sb[x], t.xo = so[x];
    t.ny = 1, t.ya = t.yb = t.yo = 0;
    if (y >= 0) t.ny = ext[y], t.ya = sa[y], t.yb = sb[y], t.yo = so[y];
    if (t.nx > 0xFFFFF000u || t.ny > 0xFFFFF000u) return false;   // x0 + 1023 must not wrap
    const uint32_t tx = (t.nx - 1) / TX + 1, ty = (t.ny - 1) / TY + 1;
    uint64_t tiles = uint64_t(tx) * ty;
    t.rest = 0;
    for (int k = n - 1; k >= 0; --k) {
        if (k == x || k == y) continue;
        t.ext[t.rest] = ag_fastdiv_make(ext[k]);
        t.sa[t.rest] = sa[k], t.sb[t.rest] = sb[k], t.so[t.rest] = so[k];
        ++t.rest;
        tiles *= ext[k];
    }
    if (tiles > 0xFFFF0000ull) return false;   // t += gridDim.x must not wrap
    t.tx = ag_fastdiv_make(tx), t.ty = ag_fastdiv_make(ty);
    t.tiles = uint32_t(tiles);
    return true;
}

template <int OP, class TI, class TO>
cudaError_t rt_launch_tiled(const RtTile& t, bool turn_a, bool turn_b, cudaStream_t s) {
    // a CTA per tile: 111 us where a grid of 8 CTAs per SM, whose warps wait for
    // one another at each tile, took 135 (96 x 509 x 515 f64, one input turned)
    constexpr unsigned cap = 1u << 30;
    const unsigned grid = t.tiles < cap ? t.tiles : cap;
    if (turn_a && turn_b) rt_tiled<OP, TI, TO, true, true><<<grid, kBlock, 0, s>>>(t);
    else if (turn_a) rt_tiled<OP, TI, TO, true, false><<<grid, kBlock, 0, s>>>(t);
    else if (turn_b) rt_tiled<OP, TI, TO, false, true><<<grid, kBlock, 0, s>>>(t);
    else rt_tiled<OP, TI, TO, false, false><<<grid, kBlock, 0, s>>>(t);
    return cudaGetLastError();
}

template <int OP, class TI, class TO>
cudaError_t rt_launch(const RtDesc& d, bool contiguous, bool vec, cudaStream_t s) {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (!contiguous) {
        RtTile t;
        bool turn_a = false, turn_b = false;
        if (rt_plan_tiles(d, uses_b(OP), t, turn_a, turn_b)) return rt_launch_tiled<OP, TI, TO>(t, turn_a, turn_b, s);
    }
    const uint64_t threads = (uint64_t(d.total) + kRun - 1) / kRun;
    const uint64_t want = (threads + kBlock - 1) / kBlock;
    const unsigned grid = unsigned(want < uint64_t(sms) * 8 ? (want ? want : 1) : uint64_t(sms) * 8);
    if (contiguous && vec) rt_contiguous<OP, TI, TO, true><<<grid, kBlock, 0, s>>>(d);
    else if (contiguous) rt_contiguous<OP, TI, TO, false><<<grid, kBlock, 0, s>>>(d);
    else rt_strided<OP, TI, TO><<<grid, kBlock, 0, s>>>(d);
    return cudaGetLastError();
}

template <class TI, class TO>
cudaError_t rt_dispatch_op(int op, const RtDesc& d, bool contiguous, bool vec, cudaStream_t s) {
    switch (op) {
    case AETHER_RT_ASSIGN: return rt_launch<AETHER_RT_ASSIGN, TI, TO>(d, contiguous, vec, s);
    case AETHER_RT_ADD: return rt_launch<AETHER_RT_ADD, TI, TO>(d, contiguous, vec, s);
    case AETHER_RT_SUB: return rt_launch<AETHER_RT_SUB, TI, TO>(d, contiguous, vec, s);
    case AETHER_RT_SCALE: return rt_launch<AETHER_RT_SCALE, TI, TO>(d, contiguous, vec, s);
    case AETHER_RT_ADD_SCALED: return rt_launch<AETHER_RT_ADD_SCALED, TI, TO>(d, contiguous, vec, s);
    default: return rt_launch<AETHER_RT_SUB_SCALED, TI, TO>(d, contiguous, vec, s);
    }
}

bool is_f64(const AetherRuntimeView& v) { return v.dtype_code == 2 && v.dtype_bits == 64 && v.dtype_lanes == 1; }
bool is_f32(const AetherRuntimeView& v) { return v.dtype_code == 2 && v.dtype_bits == 32 && v.dtype_lanes == 1; }
bool same_dtype(const AetherRuntimeView& x, const AetherRuntimeView& y) {
    return x.dtype_code == y.dtype_code && x.dtype_bits == y.dtype_bits && x.dtype_lanes == y.dtype_lanes;
}
bool same_shape(const AetherRuntimeView& x, const AetherRuntimeView& y) {
    if (x.rank != y.rank) return false;
    for (int k = 0; k < x.rank; ++k)
        if (x.extents[k] != y.extents[k]) return false;
    return true;
}
bool row_major(const AetherRuntimeView& v) {
    int64_t want = 1;
    for (int k = v.rank - 1; k >= 0; --k) {
        if (v.extents[k] != 1 && v.strides[k] != want) return false;
        want *= v.extents[k];
    }
    return true;
}
bool on_device(const void* p) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

int rt_fail(uint64_t size, const std::string& detail) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
    const std::string m = "aether::eval::runtimeEval failed on cuda:" + std::to_string(dev) + ", size=" +
                          std::to_string(size) + " bytes (" + detail + ")";
    return ag_internal_fail(m.c_str());
}

}  // namespace

extern "C" __attribute__((visibility("default"))) int aether_runtime_eval(int op, const AetherRuntimeView* a,
                                                                         const AetherRuntimeView* b,
                                                                         const AetherRuntimeView* out, double scalar,
                                                                         void* stream) {
    if (op < AETHER_RT_ASSIGN || op > AETHER_RT_SUB_SCALED) return rt_fail(0, "unknown op");
    if (!a || !out) return rt_fail(0, "null view");
    const bool ub = uses_b(op);
    if (ub && !b) return rt_fail(0, "the op reads b but b is null");
    for (const AetherRuntimeView* v : {a, ub ? b : a, out})
        if (v->rank < 0 || v->rank > AETHER_RT_RANK_CAP) return rt_fail(0, "rank above the cap of 6");
    if (!same_shape(*a, *out)) return rt_fail(0, "shape mismatch: a vs out");
    if (ub && !same_shape(*b, *out)) return rt_fail(0, "shape mismatch: b vs out");
    if (!is_f32(*a) && !is_f64(*a)) return rt_fail(0, "unsupported input dtype (v1: double/float only)");
    if (!is_f32(*out) && !is_f64(*out)) return rt_fail(0, "unsupported output dtype (v1: double/float only)");
    if (op != AETHER_RT_ASSIGN) {
        if (!same_dtype(*a, *out)) return rt_fail(0, "dtype mismatch: a vs out (only Assign performs a cast)");
        if (ub && !same_dtype(*b, *out)) return rt_fail(0, "dtype mismatch: b vs out");
    }
    uint64_t total = 1;
    for (int k = 0; k < out->rank; ++k) {
        if (out->extents[k] < 0) return rt_fail(0, "negative extent");
        total *= uint64_t(out->extents[k]);
        if (total > 0xFFFFFFFFull) break;
    }
    for (const AetherRuntimeView* v : {a, ub ? b : a, out})
        for (int k = 0; k < v->rank; ++k)
            if (v->strides[k] < 0) return rt_fail(0, "negative strides are not addressable");
    if (total == 0) return AETHER_OK;
    if (total > 0xFFFFFFFFull) return rt_fail(total, "flat element count exceeds the offset_t addressable maximum");
    if (!a->data || !out->data || (ub && !b->data)) return rt_fail(0, "null data pointer");
    if (!on_device(a->data) || !on_device(out->data) || (ub && !on_device(b->data)))
        return rt_fail(0, "operands must be device memory (this engine has no host path)");

    RtDesc d{};
    d.a = a->data;
    d.b = ub ? b->data : nullptr;
    d.o = out->data;
    d.rank = out->rank;
    d.total = uint32_t(total);
    d.scalar = scalar;
    for (int k = 0; k < d.rank; ++k) {
        d.ext[k] = ag_fastdiv_make(uint32_t(out->extents[k]));
        d.sa[k] = a->strides[k];
        d.sb[k] = ub ? b->strides[k] : 0;
        d.so[k] = out->strides[k];
    }
    const bool contiguous = row_major(*a) && row_major(*out) && (!ub || row_major(*b));
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const bool vec = contiguous && aligned(d.a) && aligned(d.o) && (!ub || aligned(d.b));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    if (is_f64(*a) && is_f64(*out)) e = rt_dispatch_op<double, double>(op, d, contiguous, vec, s);
    else if (is_f32(*a) && is_f32(*out)) e = rt_dispatch_op<float, float>(op, d, contiguous, vec, s);
    else if (is_f64(*a)) e = rt_launch<AETHER_RT_ASSIGN, double, float>(d, contiguous, vec, s);
    else e = rt_launch<AETHER_RT_ASSIGN, float, double>(d, contiguous, vec, s);
    if (e != cudaSuccess) return rt_fail(total, std::string("launch: ") + cudaGetErrorString(e));
    return AETHER_OK;
}
