// Block-Jacobi preconditioner Phi^-1 = blockdiag(S_kk^-1), built on the GPU.
//
// The reference takes Phi^-1 from its caller (include/interface.cuh:24-32) and
// its documented pcg_solve(S, gamma, lambda, ...) (README.md:42) has no Phi^-1
// argument; this kernel supplies it.  The diagonal blocks S_kk (the middle block
// of a cbtd block row) are inverted in registers, a group of 8, 16 or 32 lanes a
// block (gauss_jordan.cuh), padded with the identity to NP x NP (NP in {8, 12,
// 16, 24, 32}, the smallest that holds n).  A shared-memory transpose symmetrises
// the inverse, written either as a cbtd block row [0 | S_kk^-1 | 0] or compactly
// (n^2 per knot, column-major), column by column.
//
// A warp takes `per` consecutive knots of the batch (the knot-prefix array maps
// them to systems) and inverts as many at once as their n allows.
//
// Two kernels.  FP32 batches with 8192 knots or more of a block-size class take
// four rows a lane (block_jacobi_quad_kernel): 16 to 4 blocks a warp share the
// search for their system, the divisions and the barriers.  Everything else takes
// one row a lane: few knots, because one block then has the shorter chain and
// runs beside the others (one system of n=14, 60 knots: 6.9 us against 9.1 with
// two a warp), and FP64, whose pipe (two lanes a clock per SM) bounds it: there
// two blocks of n <= 16 a warp instead of one halve the instructions (1024
// systems of n=14, 1634 -> 823 us), and n = 24 gains 2%.
//
// Measured, FP32, us, one block a warp with a scaled pivot row / one row a lane /
// four: 2048 systems of 16 to 128 knots, n=14 302 / 143 / 108, n=6 173 / 57 / 34,
// n in {6, 12, 14, 24} 317 / 225 / 182; 1024 of n=24 269 / 250 / 181; 512 of n=32
// 223 / 287 / 181.  What bounds four rows a lane is the fetch of its long
// straight-line code by two or three warps a scheduler (n=24: 990 instructions a
// block, issued at 37%).  TI: element type of S, TO: of Phi^-1, CT: arithmetic (double S
// with float Phi^-1 serves the FP32-inner refinement).
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <type_traits>

#include "gauss_jordan.cuh"
#include "pcg_types.h"

namespace gbdpcg {

constexpr int kPrecWarps = 4;  // warps per CTA
constexpr int kPrecMaxN = 32;
// elements of the transposes of a warp's blocks: 32 rows of 33, or two of 16 x 17,
// or four of 8 x 9
constexpr int kPrecX = kPrecMaxN * (kPrecMaxN + 1);

// The classes of block sizes: NP = 8, 12, 16, 24, 32; -1 outside.
__host__ __device__ constexpr int np_class(uint32_t n) {
    return n == 0 ? -1 : (n <= 8 ? 0 : (n <= 12 ? 1 : (n <= 16 ? 2 : (n <= 24 ? 3 : (n <= (uint32_t)kPrecMaxN ? 4 : -1)))));
}

// The last s in [0, nsys) with knot_prefix[s] <= gk, by a whole warp: 32 probes a
// round (three rounds of loads for 32768 systems where a binary search pays 15
// one after another).
__device__ __forceinline__ uint32_t find_system(const uint64_t *__restrict__ knot_prefix, uint32_t nsys, uint64_t gk,
                                                uint32_t lane) {
    uint32_t lo = 0, len = nsys;
    while (len > 1) {
        const uint32_t step = (len + 31) / 32, i = lane * step;
        const uint32_t below = __popc(__ballot_sync(0xffffffffu, i < len && knot_prefix[lo + i] <= gk));
        lo += (below - 1) * step;  // (the first probe always holds)
        len = min(step, len - (below - 1) * step);
    }
    return lo;
}

// Inverts `cnt` blocks of one system at once (cnt <= 32 / GL): block g's S_kk at
// Sk + g strideS, its row of Phi^-1 at row + g strideP.  Groups from cnt on run on
// the identity and write nothing.  Whether this lane's block is inverted (gj_inverse).
template <typename TI, typename TO, typename CT, int NP>
__device__ __forceinline__ bool invert_knots(const TI *Sk, TO *row, uint32_t n, uint32_t cnt, int tri_layout, CT *s, CT *X,
                                             uint32_t lane) {
    constexpr int GL = gj_lanes(NP), LD = GL + 1;
    const uint32_t g = lane / GL, r = lane % GL;
    const bool mine = g < cnt && r < n;
    Sk += (size_t)g * 3 * n * n;
    row += (size_t)g * (tri_layout ? 3 : 1) * n * n;
    // row r of S_kk (column-major: (r, c) at c*n + r; coalesced over lanes),
    // identity beyond n
    CT a[NP];
#pragma unroll
    for (int c = 0; c < NP; ++c)
        a[c] = (mine && (uint32_t)c < n) ? CT(Sk[(size_t)c * n + r]) : ((uint32_t)c == r ? CT(1) : CT(0));
    const CT diag = mine ? CT(Sk[(size_t)r * n + r]) : CT(1);
    s += g * 3 * GL;
    X += g * GL * LD;
    bool ok;
    const CT h = CT(0.5) * gj_inverse<CT, NP, GL>(a, diag, mine, s, r, ok);  // (lanes without a row: 0, not used)
    const CT *D = s + 2 * GL;
    // symmetrise through a shared-memory transpose: X[r][c] = a[c] of lane r
    if (r < (uint32_t)NP) {
#pragma unroll
        for (int c = 0; c < NP; ++c) X[r * LD + c] = a[c];
    }
    __syncwarp();
    // column by column, lane = row: coalesced stores, no index division
    const uint32_t nn = n * n, mid = tri_layout ? nn : 0;
    if (mine) {
#pragma unroll
        for (int c = 0; c < NP; ++c) {
            if ((uint32_t)c < n) {
                row[mid + c * n + r] = TO(mul_pow2(a[c] + X[c * LD + r], h, D[c]));
                if (tri_layout) {
                    row[c * n + r] = TO(0);
                    row[2 * nn + c * n + r] = TO(0);
                }
            }
        }
    }
    __syncwarp();
    return ok;
}

// Inverts knots [gk, end) of the batch again, one after another (gj_invert_any): for
// a warp that met a block that is not definite.  sys: the systems in the order of
// knot_prefix (null: 0, 1, ..); descs null: `one`.  s: 32 elements, X: 32 x 32.
template <typename TI, typename TO, typename CT>
__device__ __noinline__ void invert_range_any(const SysDesc *descs, const uint32_t *sys, const uint64_t *knot_prefix,
                                              uint32_t nsys, uint64_t gk, uint64_t end, int tri_layout, const SysDesc *one,
                                              CT *s, CT *X) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = descs ? find_system(knot_prefix, nsys, gk, lane) : 0u;
    for (; gk < end; ++gk) {
        while (descs && lo + 1 < nsys && knot_prefix[lo + 1] <= gk) ++lo;
        const SysDesc *d = descs ? descs + (sys ? sys[lo] : lo) : one;
        const uint32_t n = d->n, nn = n * n, k = (uint32_t)(descs ? gk - knot_prefix[lo] : gk);
        if (np_class(n) < 0) continue;
        const TI *Sk = static_cast<const TI *>(d->S) + (size_t)k * 3 * nn + nn;
        TO *row = static_cast<TO *>(const_cast<void *>(d->P)) + (size_t)k * (tri_layout ? 3 : 1) * nn + (tri_layout ? nn : 0);
        for (uint32_t e = lane; e < nn; e += 32) X[e] = CT(Sk[e]);
        gj_invert_any<CT, TO>(X, n, row, tri_layout, n, s, lane);
    }
}

template <typename TI, typename TO, typename CT>
__global__ void __launch_bounds__(kPrecWarps * 32, sizeof(CT) == 4 ? 5 : 4)
    block_jacobi_kernel(const SysDesc *__restrict__ descs, const uint32_t *__restrict__ sys,
                        const uint64_t *__restrict__ knot_prefix, uint32_t nsys, uint64_t first_knot, uint64_t end_knot,
                        uint32_t per, int tri_layout, const __grid_constant__ SysDesc one) {
    __shared__ CT sX[kPrecWarps][kPrecX];
    __shared__ __align__(16) CT sR[kPrecWarps][kGjElems];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t start = first_knot + ((uint64_t)blockIdx.x * kPrecWarps + warp) * per;
    if (start >= end_knot) return;  // warp-uniform; no CTA-wide barrier below
    uint64_t gk = start;
    const uint64_t end = min(gk + per, end_knot);
    // system owning global knot gk: last s with knot_prefix[s] <= gk (or the
    // one system passed by value)
    uint32_t lo = descs ? find_system(knot_prefix, nsys, gk, lane) : 0u;
    CT *s = sR[warp], *X = sX[warp];
    bool ok = true;
    while (gk < end) {
        const SysDesc *d = descs ? descs + (sys ? sys[lo] : lo) : nullptr;
        const uint32_t n = d ? d->n : one.n, N = d ? d->N : one.N;
        const void *dS = d ? d->S : one.S, *dP = d ? d->P : one.P;
        const uint32_t k = (uint32_t)(descs ? gk - knot_prefix[lo] : gk);
        const uint32_t left = (uint32_t)min(end - gk, (uint64_t)(N - k));  // knots of this system in the range
        uint32_t cnt = left;
        if (np_class(n) >= 0) {
            cnt = min(left, n <= 8 ? 4u : (n <= 16 ? 2u : 1u));
            const TI *Sk = static_cast<const TI *>(dS) + (size_t)k * 3 * n * n + (size_t)n * n;
            TO *row = static_cast<TO *>(const_cast<void *>(dP)) + (size_t)k * (tri_layout ? 3 : 1) * n * n;
            if (n <= 8) ok &= invert_knots<TI, TO, CT, 8>(Sk, row, n, cnt, tri_layout, s, X, lane);
            else if (n <= 12) ok &= invert_knots<TI, TO, CT, 12>(Sk, row, n, cnt, tri_layout, s, X, lane);
            else if (n <= 16) ok &= invert_knots<TI, TO, CT, 16>(Sk, row, n, cnt, tri_layout, s, X, lane);
            else if (n <= 24) ok &= invert_knots<TI, TO, CT, 24>(Sk, row, n, cnt, tri_layout, s, X, lane);
            else ok &= invert_knots<TI, TO, CT, 32>(Sk, row, n, cnt, tri_layout, s, X, lane);
        }
        if (cnt == left) ++lo;  // the next knots are the next system's
        gk += cnt;
    }
    if (!__all_sync(0xffffffffu, ok)) {
        invert_range_any<TI, TO, CT>(descs, sys, knot_prefix, nsys, start, end, tri_layout, &one, s, X);
    }
}

// ---- FP32 batches: four rows a lane (gj_inverse_quad)

constexpr int kQuadWarps = 2;
// batches from this many knots on take it
constexpr uint64_t kQuadFrom = 8192;
// words of a warp's scratch: three rows of every block, and their transposes
template <int NP>
__host__ __device__ constexpr int quad_words() { return 3 * GjQuad<NP>::SCRATCH + GjQuad<NP>::BLOCKS * (NP * (NP + 1) + 1); }

// Inverts `cnt` blocks of one system at once (cnt <= GjQuad::BLOCKS); whether this
// lane's block is inverted.  vw: rows of
// an access (4 or 2 where n is a multiple and the addresses allow, else 1).
template <int NP>
__device__ __forceinline__ bool invert_quads(const float *Sk, float *row, uint32_t n, uint32_t cnt, int tri_layout, uint32_t vw,
                                             float *s, uint32_t lane) {
    using G = GjQuad<NP>;
    constexpr int P = NP / 2, LD = NP + 1, KX = NP * LD + 1;
    const uint32_t g0 = lane / G::LANES, g = g0 < (uint32_t)G::BLOCKS ? g0 : 0u;
    const uint32_t r = g0 < (uint32_t)G::BLOCKS ? lane % G::LANES : (uint32_t)G::LANES;
    const uint32_t i0 = 4 * r, nn = n * n;
    const bool mine = r < (uint32_t)G::LANES && g < cnt;
    Sk += (size_t)g * 3 * nn + i0;
    row += (size_t)g * (tri_layout ? 3 : 1) * nn + (tri_layout ? nn : 0) + i0;
    bool in[4];  // rows of the block
#pragma unroll
    for (int t = 0; t < 4; ++t) in[t] = mine && i0 + t < n;
    auto load4 = [&](const float *p, float (&v)[4], uint32_t c) {  // rows i0.. of column c; identity outside
#pragma unroll
        for (int t = 0; t < 4; ++t) v[t] = (c == i0 + t) ? 1.f : 0.f;
        if (c >= n) return;
        if (vw == 4) {
            if (in[0]) {
                const float4 x = __ldg(reinterpret_cast<const float4 *>(p));
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
            }
        } else if (vw == 2) {
#pragma unroll
            for (int t = 0; t < 4; t += 2)
                if (in[t]) {
                    const float2 x = __ldg(reinterpret_cast<const float2 *>(p + t));
                    v[t] = x.x; v[t + 1] = x.y;
                }
        } else {
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (in[t]) v[t] = __ldg(p + t);
        }
    };
    unsigned long long A[4][P];
    float diag[4], scale[4];
#pragma unroll
    for (int p = 0; p < P; ++p) {
        float x[4], y[4];
        load4(Sk + (size_t)(2 * p) * n, x, 2 * p);
        load4(Sk + (size_t)(2 * p + 1) * n, y, 2 * p + 1);
#pragma unroll
        for (int t = 0; t < 4; ++t) A[t][p] = pack2(x[t], y[t]);
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) diag[t] = in[t] ? __ldg(Sk + (size_t)(i0 + t) * n + t) : 1.f;
    float *buf = s + g * G::KS;
    const bool negative = __shfl_sync(0xffffffffu, diag[0], g * G::LANES) < 0.f;
    const bool ok = gj_inverse_quad<NP>(A, diag, in, negative, scale, buf, r);
    // symmetrise: X[c][row] of every block, and back transposed
    float *X = s + 3 * G::SCRATCH + g * KX;
    const float *D = buf + 2 * G::SCRATCH;
    if (r < (uint32_t)G::LANES) {
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                X[(2 * p) * LD + i0 + t] = lo2(A[t][p]);
                X[(2 * p + 1) * LD + i0 + t] = hi2(A[t][p]);
            }
    }
    __syncwarp();
    if (mine && i0 < n) {
#pragma unroll
        for (int c = 0; c < NP; ++c) {
            if ((uint32_t)c >= n) continue;
            const float dc = D[c];
            float v[4];
#pragma unroll
            for (int t = 0; t < 4; ++t)
                v[t] = (((c & 1) ? hi2(A[t][c / 2]) : lo2(A[t][c / 2])) + X[(i0 + t) * LD + c]) * (0.5f * scale[t] * dc);
            float *o = row + (size_t)c * n;
            if (vw == 4) {
                *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
            } else if (vw == 2) {
                *reinterpret_cast<float2 *>(o) = make_float2(v[0], v[1]);
                if (in[2]) *reinterpret_cast<float2 *>(o + 2) = make_float2(v[2], v[3]);
            } else {
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (in[t]) o[t] = v[t];
            }
            if (tri_layout) {
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (in[t]) {
                        o[(int64_t)t - (int64_t)nn] = 0.f;
                        o[t + nn] = 0.f;
                    }
            }
        }
    }
    __syncwarp();
    return ok;
}

// One launch per block-size class, so that an SM runs one class's code and a
// narrow block does not pay for the registers of a wide one (all classes in one
// kernel: 312 us where these take 182, 2048 systems of n in {6, 12, 14, 24}).
// sys, knot_prefix: the class's systems and the knots before each, whose knots are
// [first_knot, end_knot); null: `one`.
template <int NP>
__global__ void __launch_bounds__(kQuadWarps * 32, NP <= 8 ? 12 : (NP <= 12 ? 9 : (NP <= 16 ? 8 : (NP <= 24 ? 6 : 4))))
    block_jacobi_quad_kernel(const SysDesc *__restrict__ descs, const uint32_t *__restrict__ sys,
                             const uint64_t *__restrict__ knot_prefix, uint32_t nsys, uint64_t first_knot, uint64_t end_knot,
                             uint32_t per, int tri_layout, const __grid_constant__ SysDesc one) {
    __shared__ __align__(16) float scratch[kQuadWarps][(quad_words<NP>() + 3) / 4 * 4];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t start = first_knot + ((uint64_t)blockIdx.x * kQuadWarps + warp) * per;
    if (start >= end_knot) return;  // warp-uniform; no CTA-wide barrier below
    uint64_t gk = start;
    const uint64_t end = min(gk + per, end_knot);
    uint32_t lo = sys ? find_system(knot_prefix, nsys, gk, lane) : 0u;
    bool ok = true;
    while (gk < end) {
        const SysDesc *d = sys ? descs + sys[lo] : nullptr;
        const uint32_t n = d ? d->n : one.n, N = d ? d->N : one.N;
        const float *S = static_cast<const float *>(d ? d->S : one.S);
        float *P = static_cast<float *>(const_cast<void *>(d ? d->P : one.P));
        const uint32_t k = (uint32_t)(sys ? gk - knot_prefix[lo] : gk);
        const uint32_t left = (uint32_t)min(end - gk, (uint64_t)(N - k));  // knots of this system in the range
        const uint32_t cnt = min(left, (uint32_t)GjQuad<NP>::BLOCKS);
        const uintptr_t at = reinterpret_cast<uintptr_t>(S) | reinterpret_cast<uintptr_t>(P);
        const uint32_t vw = (n % 4 == 0 && (at & 15u) == 0) ? 4u : ((n % 2 == 0 && (at & 7u) == 0) ? 2u : 1u);
        ok &= invert_quads<NP>(S + (size_t)k * 3 * n * n + (size_t)n * n, P + (size_t)k * (tri_layout ? 3 : 1) * n * n, n, cnt,
                               tri_layout, vw, scratch[warp], lane);
        if (cnt == left) ++lo;  // the next knots are the next system's
        gk += cnt;
    }
    if (!__all_sync(0xffffffffu, ok)) {
        static_assert(quad_words<NP>() >= 32 + NP * NP, "scratch of the other inverse");
        invert_range_any<float, float, float>(sys ? descs : nullptr, sys, knot_prefix, nsys, start, end, tri_layout, &one,
                                              scratch[warp], scratch[warp] + 32);
    }
}

// kind: 0 float S -> float Phi^-1 (float arithmetic); 1 double -> double;
// 2 double S -> float Phi^-1 (double arithmetic, for the refinement's inner solve)
// d_descs == nullptr: the single system *one (total_knots = its N), passed to
// the kernel by value (no descriptor upload).
// cls: the batch by block-size class (null for a single system).
int jacobi_class(uint32_t n) { return np_class(n); }

cudaError_t launch_block_jacobi(int kind, const SysDesc *d_descs, const uint64_t *d_prefix,
                                uint32_t nsys, uint64_t total_knots, int tri_layout,
                                cudaStream_t stream, const SysDesc *one, const JacobiClasses *cls) {
    if (total_knots == 0) return cudaSuccess;
    SysDesc o;
    if (one) o = *one;
    else memset(&o, 0, sizeof(o));
    bool quads[5] = {};  // classes of the kernel with four rows a lane
    if (kind == 0) {
        auto quad = [&](auto np) {
            constexpr int NP = decltype(np)::value, c = np_class(NP);
            const uint64_t knots = one ? (np_class(o.n) == c ? total_knots : 0) : cls->knots[c];
            if (knots < kQuadFrom) return;
            const uint32_t *sys = one ? nullptr : cls->sys + cls->first[c];
            const uint64_t *prefix = one ? nullptr : cls->prefix + cls->first[c];
            const uint64_t first = one ? 0 : cls->base[c];
            const uint32_t per = GjQuad<NP>::BLOCKS * (knots >= (uint64_t)GjQuad<NP>::BLOCKS * 4096 ? 2 : 1);
            const uint64_t warps = (knots + per - 1) / per;
            block_jacobi_quad_kernel<NP><<<(unsigned)((warps + kQuadWarps - 1) / kQuadWarps), kQuadWarps * 32, 0, stream>>>(
                d_descs, sys, prefix, one ? 1u : cls->count[c], first, first + knots, per, tri_layout, o);
            quads[c] = true;
        };
        quad(std::integral_constant<int, 24>());
        quad(std::integral_constant<int, 32>());
        quad(std::integral_constant<int, 16>());
        quad(std::integral_constant<int, 12>());
        quad(std::integral_constant<int, 8>());
    }
    // one row a lane for knots [first, first + knots) of the order of `sys`
    auto rest = [&](const uint32_t *sys, const uint64_t *prefix, uint32_t count, uint64_t first, uint64_t knots) {
        // knots a warp: side by side while the GPU has warps to spare, then several, as
        // many as a warp inverts at once for a single system
        const uint32_t most = d_descs ? 4u : (o.n <= 8 ? 4u : (o.n <= 16 ? 2u : 1u));
        const uint32_t per = knots < 8192 ? 1u : (knots < 32768 ? (most < 2 ? most : 2u) : most);
        const uint64_t warps = (knots + per - 1) / per;
        const dim3 grid((unsigned)((warps + kPrecWarps - 1) / kPrecWarps)), block(kPrecWarps * 32);
        if (kind == 1)
            block_jacobi_kernel<double, double, double><<<grid, block, 0, stream>>>(d_descs, sys, prefix, count, first,
                                                                                    first + knots, per, tri_layout, o);
        else if (kind == 2)
            block_jacobi_kernel<double, float, double><<<grid, block, 0, stream>>>(d_descs, sys, prefix, count, first,
                                                                                   first + knots, per, tri_layout, o);
        else
            block_jacobi_kernel<float, float, float><<<grid, block, 0, stream>>>(d_descs, sys, prefix, count, first,
                                                                                 first + knots, per, tri_layout, o);
    };
    bool any = false;
    for (bool q : quads) any |= q;
    if (!any) {
        rest(nullptr, d_prefix, nsys, 0, total_knots);
    } else if (!one) {
        // runs of neighbouring classes that are left: their knots only (with one launch
        // over all knots, most of whose warps found nothing to do, 1000 systems of n=6
        // and 10 of n=24, 100 knots each, took 74 us; now 32)
        for (int c = 0; c < 5;) {
            int e = c;
            uint32_t count = 0;
            uint64_t knots = 0;
            for (; e < 5 && !quads[e]; ++e) {
                count += cls->count[e];
                knots += cls->knots[e];
            }
            if (knots) rest(cls->sys + cls->first[c], cls->prefix + cls->first[c], count, cls->base[c], knots);
            c = e + 1;
        }
    }
    return cudaGetLastError();
}

}  // namespace gbdpcg
