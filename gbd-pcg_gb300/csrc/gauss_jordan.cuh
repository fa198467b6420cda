// Inverse of small symmetric blocks, positive definite in earnest, one row per lane
// (shared by the block-Jacobi builder and the fused Schur formation):
// Gauss-Jordan elimination without pivoting.
//
// A group of GL = 8, 16 or 32 lanes holds one block, so that a warp inverts four
// blocks of n <= 8, two of n <= 16 or one of n <= 32 at once.  Lane r holds row r
// in registers, padded with the identity to NP x NP.  Step k: lane k stores its
// row in shared memory, and every lane subtracts m = a_rk / a_kk times that row
// (16-byte broadcast loads) from its own.  Registers are renamed by a shift of
// two columns every two steps, so all indices are compile-time constants while
// the loop stays rolled, and FP32 rows are updated two columns an instruction
// (fma.rn.f32x2).
//
// The pivot row needs no selects: with m = 1 - 1/a_kk in its lane the common
// update is a_kj / a_kk.  For pivots in [u, 2) (u = 2^-24 in FP32, 2^-53 in
// FP64) that m is exact and the one rounding of the update is the quotient's.  So the
// rows are scaled by powers of two (exactly) to a diagonal in [1/4, 1), and a
// block whose first diagonal element is negative is inverted as its negative:
// every pivot of a positive or negative definite block is then at most 1, and the
// result is bit for bit that of the elimination that divides the pivot row.
// Other blocks (indefinite, singular, nearly singular) leave that range at some
// pivot; the elimination notes it, and the caller inverts the block again by
// gj_invert_any, which divides the pivot row and neither scales nor negates: a zero
// pivot then leaves its column unscaled.
//
// What bounds it is the issue of instructions: about 42 a column of an n = 24
// block (12 f32x2 FMAs, 12 shared-memory accesses) where scaling the pivot row in
// a pass of its own, with a select an element, took about 87; and two (n <= 16) or
// four (n <= 8) blocks a warp where it held one.  Measured: precond.cu, kkt.cu.
#pragma once
#include <stdint.h>

namespace gbdpcg {

template <typename CT>
struct PrecVec;  // 16-byte shared-memory loads
template <>
struct PrecVec<float> {
    static constexpr int W = 4;
    __device__ static void get(const float *p, float *v) {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
};
template <>
struct PrecVec<double> {
    static constexpr int W = 2;
    __device__ static void get(const double *p, double *v) {
        const double2 t = *reinterpret_cast<const double2 *>(p);
        v[0] = t.x; v[1] = t.y;
    }
};

// Two floats in one 64-bit register.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo2(unsigned long long v) {
    float x;
    asm("{\n\t.reg .b32 t;\n\tmov.b64 {%0, t}, %1;\n\t}" : "=f"(x) : "l"(v));
    return x;
}
__device__ __forceinline__ float hi2(unsigned long long v) {
    float x;
    asm("{\n\t.reg .b32 t;\n\tmov.b64 {t, %0}, %1;\n\t}" : "=f"(x) : "l"(v));
    return x;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The power of two s with s^2 |d| in [1/4, 1); 1 for zero, subnormal and
// non-finite d.
__device__ __forceinline__ float pow2_scale(float d) {
    const int e = (int)((__float_as_uint(d) >> 23) & 0xffu);
    if (e == 0 || e == 255) return 1.f;
    return __uint_as_float((uint32_t)(127 - ((e - 127 + 2) >> 1)) << 23);
}
__device__ __forceinline__ double pow2_scale(double d) {
    const int e = (int)(((uint32_t)__double2hiint(d) >> 20) & 0x7ffu);
    if (e == 0 || e == 2047) return 1.0;
    return __hiloint2double((int)((uint32_t)(1023 - ((e - 1023 + 2) >> 1)) << 20), 0);
}

// x s t for powers of two s and t.  FP64 multiplications issue at two lanes a
// clock per SM, so a normal x with a normal product has its exponent changed on
// the integer pipe.
__device__ __forceinline__ float mul_pow2(float x, float s, float t) { return x * (s * t); }
__device__ __forceinline__ double mul_pow2(double x, double s, double t) {
    const uint32_t h = (uint32_t)__double2hiint(x), e = (h >> 20) & 0x7ffu;
    const int k = (int)((uint32_t)__double2hiint(s) >> 20) + (int)((uint32_t)__double2hiint(t) >> 20) - 2046;
    const int to = (int)e + k;
    if (e - 1u < 2046u && to > 0 && to < 2047) return __hiloint2double((int)(h + ((uint32_t)k << 20)), __double2loint(x));
    if (((h << 1) | (uint32_t)__double2loint(x)) == 0u) return x;
    return x * s * t;
}

// How far a pivot lies outside [u, 2): the largest over a block's pivots stays
// within kPivotRange where all of them are inside (integer operations: NaN,
// infinities, zero and negative pivots are outside too).
__device__ __forceinline__ uint32_t pivot_off(float piv) { return __float_as_uint(piv) - 0x33800000u; }
__device__ __forceinline__ uint32_t pivot_off(double piv) { return (uint32_t)__double2hiint(piv) - 0x3ca00000u; }
template <typename CT>
constexpr uint32_t kPivotRange = sizeof(CT) == 4 ? 0x40000000u - 0x33800000u - 1u : 0x40000000u - 0x3ca00000u - 1u;

// Negative where d is (integer work: an FP64 comparison would wait for that pipe).
__device__ __forceinline__ int sign_word(float d) { return __float_as_int(d); }
__device__ __forceinline__ int sign_word(double d) { return __double2hiint(d); }

// lanes a block of NP rows takes
__host__ __device__ constexpr int gj_lanes(int NP) { return NP <= 8 ? 8 : (NP <= 16 ? 16 : 32); }
// shared memory of a warp, in elements: three rows of 32
constexpr int kGjElems = 96;

// In: a = row r of the block (identity rows and columns beyond n; anything for
// r >= NP), diag = its diagonal element, real = r < n.  Out: a = row r of
// (D A D)^-1 for the power-of-two diagonal D, D_r (returned), and D in s[2 GL ..]:
// (A^-1)_rc = a[c] D_r D_c; FP32, negative first diagonal element: a and the D_r
// returned are both negated.  `ok`: every pivot of the block was in range.  s: this
// group's 3 GL elements (16-byte aligned) of the warp's scratch; r: lane in the
// group.  Called by whole warps.
template <typename CT, int NP, int GL>
__device__ __forceinline__ CT gj_inverse(CT (&a)[NP], CT diag, bool real, CT *s, uint32_t r, bool &ok) {
    static_assert(NP % 2 == 0 && NP <= GL, "pairs of columns; a lane per row");
    constexpr int W = PrecVec<CT>::W;
    const bool row = r < (uint32_t)NP;
    uint32_t off = 0;
    const bool negative = __shfl_sync(0xffffffffu, sign_word(diag), 0, GL) < 0;
    CT scale = row ? pow2_scale(diag) : CT(0);
    if (row) s[2 * GL + r] = scale;
    // FP32 negates by the scale; FP64, whose scaling is integer work, the elements
    if constexpr (sizeof(CT) == 4) {
        if (real && negative) scale = -scale;
    } else if (real && negative) {
#pragma unroll
        for (int c = 0; c < NP; ++c) a[c] = -a[c];
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < NP; c += W) {
        CT t[W];
        PrecVec<CT>::get(s + 2 * GL + c, t);
#pragma unroll
        for (int u = 0; u < W; ++u) a[c + u] = row ? mul_pow2(a[c + u], scale, t[u]) : CT(0);
    }
    if constexpr (sizeof(CT) == 4) {
        constexpr int P = NP / 2;  // pairs of columns
        unsigned long long A[P], T[P];
#pragma unroll
        for (int p = 0; p < P; ++p) A[p] = pack2(a[2 * p], a[2 * p + 1]);
        auto pivot_row = [&](bool pivot, float *buf) {  // lane k's row to all lanes
            if (pivot) {
#pragma unroll
                for (int p = 0; p + 1 < P; p += 2) *reinterpret_cast<ulonglong2 *>(buf + 2 * p) = make_ulonglong2(A[p], A[p + 1]);
                if constexpr (P % 2) *reinterpret_cast<unsigned long long *>(buf + 2 * (P - 1)) = A[P - 1];
            }
            __syncwarp();
#pragma unroll
            for (int p = 0; p + 1 < P; p += 2) {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(buf + 2 * p);
                T[p] = t.x;
                T[p + 1] = t.y;
            }
            if constexpr (P % 2) T[P - 1] = *reinterpret_cast<const unsigned long long *>(buf + 2 * (P - 1));
        };
#pragma unroll 1
        for (uint32_t k = 0; k < (uint32_t)NP; k += 2) {
            // column k, the first of pair 0, in place
            bool pivot = r == k;
            pivot_row(pivot, s);
            float piv = lo2(T[0]);
            off = max(off, pivot_off(piv));
            float inv = 1.f / piv, m = pivot ? 1.f - inv : lo2(A[0]) * inv;
            unsigned long long nm = pack2(-m, -m);
#pragma unroll
            for (int p = 0; p < P; ++p) A[p] = fma2(nm, T[p], A[p]);
            A[0] = pack2(pivot ? inv : -m, hi2(A[0]));
            // column k + 1, the second of pair 0; the pairs move down by one and
            // pair 0 to the end (buffers alternate: one warp barrier a step)
            pivot = r == k + 1;
            pivot_row(pivot, s + GL);
            piv = hi2(T[0]);
            off = max(off, pivot_off(piv));
            inv = 1.f / piv;
            m = pivot ? 1.f - inv : hi2(A[0]) * inv;
            nm = pack2(-m, -m);
            const unsigned long long first = fma2(nm, T[0], A[0]);
#pragma unroll
            for (int p = 1; p < P; ++p) A[p - 1] = fma2(nm, T[p], A[p]);
            A[P - 1] = pack2(lo2(first), pivot ? inv : -m);
        }
#pragma unroll
        for (int p = 0; p < P; ++p) {
            a[2 * p] = lo2(A[p]);
            a[2 * p + 1] = hi2(A[p]);
        }
    } else {
#pragma unroll 1
        for (uint32_t k = 0; k < (uint32_t)NP; ++k) {
            const bool pivot = r == k;
            CT *buf = s + (k & 1) * GL;
            if (pivot) {
#pragma unroll
                for (int c = 0; c < NP; c += 2) *reinterpret_cast<double2 *>(buf + c) = make_double2(a[c], a[c + 1]);
            }
            __syncwarp();
            const CT piv = buf[0];
            off = max(off, pivot_off(piv));
            const CT inv = CT(1) / piv;
            // pivot ? 1 - inv : a[0] inv, in one FP64 instruction (x + -0 = x)
            const CT m = fma(pivot ? CT(-1) : a[0], inv, pivot ? CT(1) : CT(-0.0));
#pragma unroll
            for (int c = 0; c < NP; c += W) {
                CT t[W];
                PrecVec<CT>::get(buf + c, t);
#pragma unroll
                for (int u = 0; u < W; ++u)
                    if (c + u > 0) a[c + u - 1] = a[c + u] - m * t[u];
            }
            a[NP - 1] = pivot ? inv : -m;
        }
        if (real && negative) {
#pragma unroll
            for (int c = 0; c < NP; ++c) a[c] = -a[c];
        }
    }
    __syncwarp();
    ok = off <= kPivotRange<CT>;
    return scale;
}

// Inverts the block in X (element (r, c) at X[c ld + r], n <= 32) of any kind, with
// the pivot row divided; its inverse, symmetrised, to P (with zero blocks on both
// sides of it for `sides`).  The rows stay in shared memory, lane r working on row r,
// so that a kernel whose blocks seldom need it keeps its registers.  s: n elements.
// Called by whole warps.
template <typename CT, typename TO>
__device__ __forceinline__ void gj_invert_any(CT *X, uint32_t ld, TO *P, bool sides, uint32_t n, CT *s, uint32_t r) {
    const bool row = r < n;
    const uint32_t nn = n * n;
    for (uint32_t k = 0; k < n; ++k) {
        __syncwarp();
        CT piv = X[k * ld + k];
        if (piv == CT(0)) piv = CT(1);
        const CT inv = CT(1) / piv, m = row ? X[k * ld + r] : CT(0);
        if (row) s[r] = r == k ? inv : X[r * ld + k] * inv;
        __syncwarp();
        for (uint32_t c = 0; row && c < n; ++c) {
            CT *x = X + c * ld + r;
            *x = r == k ? s[c] : (c == k ? -(m * inv) : *x - m * s[c]);
        }
    }
    __syncwarp();
    for (uint32_t c = 0; row && c < n; ++c) {
        P[c * n + r] = TO(CT(0.5) * (X[c * ld + r] + X[r * ld + c]));
        if (sides) {
            (P - nn)[c * n + r] = TO(0);
            (P + nn)[c * n + r] = TO(0);
        }
    }
    __syncwarp();
}

// ---- four rows a lane (FP32)
//
// The same elimination with lane r of a group of NP / 4 lanes holding rows 4r ..
// 4r + 3: a warp inverts 16, 10, 8, 5 or 4 blocks of NP = 8, 12, 16, 24, 32 at
// once.  With one row a lane, what bounds it is the pivot row's way into every
// lane's registers (NP words a step and lane, 128 bytes a clock for the SM, from
// shared memory or by shuffles alike); four rows use each word four times, and
// the division and the warp barrier of a step serve all blocks of the warp.
template <int NP>
struct GjQuad {
    static constexpr int LANES = NP / 4, BLOCKS = 32 / LANES;
    // words from one block's row buffer to the next: a multiple of 4 (16-byte
    // accesses) that puts the blocks of a quarter warp on different banks
    static constexpr int KS = NP % 8 == 4 ? NP : NP + 4;
    static constexpr int SCRATCH = BLOCKS * KS;  // one row of every block
};

// In: A[t][p] = columns 2p, 2p + 1 of row 4r + t, diag its diagonal elements,
// real[t]: not an identity row, negative: the block's first diagonal element is.
// Out: A = rows of (s D A D)^-1, scale[t] = s D of its rows, D and s as in
// gj_inverse; returns whether every pivot was in range.  buf: this block's row
// buffer, the second one GjQuad::SCRATCH words on and D's a further SCRATCH on;
// r >= LANES: a lane without rows (its registers are arbitrary but finite, it
// stores nothing and reads a valid buffer).
template <int NP>
__device__ __forceinline__ bool gj_inverse_quad(unsigned long long (&A)[4][NP / 2], const float (&diag)[4],
                                                const bool (&real)[4], bool negative, float (&scale)[4], float *buf,
                                                uint32_t r) {
    using G = GjQuad<NP>;
    constexpr int P = NP / 2;
    const bool live = r < (uint32_t)G::LANES;
#pragma unroll
    for (int t = 0; t < 4; ++t) scale[t] = pow2_scale(diag[t]);
    if (live) *reinterpret_cast<float4 *>(buf + 2 * G::SCRATCH + 4 * r) = make_float4(scale[0], scale[1], scale[2], scale[3]);
#pragma unroll
    for (int t = 0; t < 4; ++t)
        if (real[t] && negative) scale[t] = -scale[t];
    uint32_t off = 0;
    __syncwarp();
#pragma unroll
    for (int p = 0; p < P; p += 2) {
        const ulonglong2 d = *reinterpret_cast<const ulonglong2 *>(buf + 2 * G::SCRATCH + 2 * p);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const unsigned long long sc = pack2(scale[t], scale[t]);
            A[t][p] = mul2(A[t][p], mul2(sc, d.x));
            A[t][p + 1] = mul2(A[t][p + 1], mul2(sc, d.y));
        }
    }
#pragma unroll 1
    for (uint32_t kq = 0; kq < (uint32_t)G::LANES; ++kq) {
        const bool owner = r == kq;
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // column 4 kq + q: half q & 1 of pair 0
            float *row = buf + (q & 1) * G::SCRATCH;
            if (owner) {
#pragma unroll
                for (int p = 0; p < P; p += 2)
                    *reinterpret_cast<ulonglong2 *>(row + 2 * p) = make_ulonglong2(A[q][p], A[q][p + 1]);
            }
            __syncwarp();
            const unsigned long long t0 = *reinterpret_cast<const unsigned long long *>(row);
            const float piv = (q & 1) ? hi2(t0) : lo2(t0);
            off = max(off, pivot_off(piv));
            const float inv = 1.f / piv;
            unsigned long long nm[4], end[4];
            float last[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float own = (q & 1) ? hi2(A[t][0]) : lo2(A[t][0]);
                const bool pivot = owner && t == q;
                const float m = pivot ? 1.f - inv : own * inv;
                nm[t] = pack2(-m, -m);
                last[t] = pivot ? inv : -m;
                end[t] = fma2(nm[t], t0, A[t][0]);
                if (!(q & 1)) A[t][0] = pack2(last[t], hi2(end[t]));  // in place
            }
#pragma unroll
            for (int p = 0; p < P; p += 2) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(row + 2 * p);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (q & 1) {  // the pairs move down by one
                        if (p > 0) A[t][p - 1] = fma2(nm[t], w.x, A[t][p]);
                        A[t][p] = fma2(nm[t], w.y, A[t][p + 1]);
                    } else {
                        if (p > 0) A[t][p] = fma2(nm[t], w.x, A[t][p]);
                        A[t][p + 1] = fma2(nm[t], w.y, A[t][p + 1]);
                    }
                }
            }
            if (q & 1) {
#pragma unroll
                for (int t = 0; t < 4; ++t) A[t][P - 1] = pack2(lo2(end[t]), last[t]);
            }
        }
    }
    __syncwarp();
    return off <= kPivotRange<float>;
}

}  // namespace gbdpcg
