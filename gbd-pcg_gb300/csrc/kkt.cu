// The steps on either side of the PCG in a trajectory-optimisation solver
// (the callers of solvePCG in MPCGPU / GATO, outside the reference repo):
// forming the Schur complement S and its right-hand side gamma from the
// problem data, and recovering the primal step from the multipliers lambda.
//
// Problem (one system): states x_0..x_N (n each), controls u_0..u_{N-1}
// (m each), z = (x, u); cost 1/2 z^T Theta z + g^T z with Theta =
// blockdiag(Q_0..Q_N, R_0..R_{N-1}), Q_k = diag(Qd_k), R_k = diag(Rd_k),
// g = (q_0..q_N, r_0..r_{N-1}); constraints C z = c with one block row
// [A_k  B_k  -I] per knot acting on (x_k, u_k, x_{k+1}), k = 0..N-1.  The KKT
// system [Theta C^T; C 0] [z; lambda] = [-g; c] reduces to
//     S lambda = gamma,  S = C Theta^-1 C^T,  gamma = -(c + C Theta^-1 g),
//     z = -Theta^-1 (g + C^T lambda):
//   S_kk      = A_k Q_k^-1 A_k^T + B_k R_k^-1 B_k^T + Q_{k+1}^-1
//   S_{k,k+1} = -Q_{k+1}^-1 A_{k+1}^T,  S_{k+1,k} = S_{k,k+1}^T
//   gamma_k   = -(c_k + A_k Q_k^-1 q_k + B_k R_k^-1 r_k - Q_{k+1}^-1 q_{k+1})
//   x_k = -Q_k^-1 (q_k + A_k^T lambda_k - lambda_{k-1})   (terms present for k < N, k > 0)
//   u_k = -R_k^-1 (r_k + B_k^T lambda_k)
// Inputs A_k (n x n) and B_k (n x m) are column-major blocks, knot-major:
// element (r, c) of A_k at k n^2 + c n + r, of B_k at k n m + c n + r.  S is
// written in the cbtd layout (padding blocks of knots 0 and N-1 zero), gamma
// and lambda are n N, x is n (N+1), u is m N.
//
// Both kernels read each input once and write each output once; a warp takes one to
// four knots.  The formation stages [A_k | B_k] in shared memory and forms its Gram
// product as a register tile per lane; S_kk is symmetrised through shared memory
// (0.5 (S + S^T), exactly symmetric), and the formation can invert S_kk in the same
// warp (the block-Jacobi Phi^-1).  In the back-substitution a lane reads a column of
// [A_k | B_k].  What bounds each stands at the kernels.
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <type_traits>

#include "../../include/gbdpcg.h"
#include "gauss_jordan.cuh"

namespace gbdpcg {
void set_last_error(const std::string &msg);
}

namespace {

constexpr int kKktMaxN = 32;  // n, m <= 32
// warps per CTA (4 float, 2 double: at most 40 KB of dynamic shared memory either
// way in the formation, at n = m = 32)
template <typename T>
constexpr int kkt_warps() { return sizeof(T) == 8 ? 2 : 4; }

// Shared-memory layout of one warp for the formation: Mt[l][r] = M[r][l] with
// M = [A_k | B_k] (n x (n + m)), i.e. row l of Mt is column l of A_k (l < n)
// or of B_k, contiguous in global memory; rows are NP + 4 elements (a 16-byte
// multiple), rows n..NP-1 zero.  X, the Gram product, takes Mt's place.  d, d w
// (L = n + m each) and Qi_{k+1} follow, then (with the fused inverse) the
// symmetrised S_kk of every knot the warp inverts at once, if several, Y[c][r] with
// rows of NP + 4, and the scratch of the inverse.
template <int NP>
__host__ __device__ constexpr uint32_t schur_ldt() { return NP + 4; }
// knots a warp inverts at once
template <int NP>
__host__ __device__ constexpr uint32_t schur_knots() { return 32 / gbdpcg::gj_lanes(NP); }

template <int NP>
__host__ __device__ constexpr uint32_t schur_mt_elems(uint32_t L) {
    const uint32_t mt = L * schur_ldt<NP>(), x = (NP * (NP + 1) + 3) & ~3u;
    return mt > x ? mt : x;
}
template <int NP, bool PINV>
__host__ __device__ constexpr uint32_t schur_warp_elems(uint32_t L) {
    return schur_mt_elems<NP>(L) + 2 * ((L + 3) & ~3u) + 32 +
           (PINV ? (schur_knots<NP>() > 1 ? schur_knots<NP>() * NP * schur_ldt<NP>() : 0) + gbdpcg::kGjElems : 0);
}

// Asynchronous copy of VW consecutive elements global -> shared (cp.async, no
// registers, nothing waits until cp_async_wait_all).
template <typename T, int VW>
__device__ __forceinline__ void cp_async_vec(T *smem, const T *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem),
                 "n"((int)(VW * sizeof(T)))
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// VW consecutive elements as one access (VW sizeof(T) bytes, 16 at most).
template <typename T, int VW>
__device__ __forceinline__ void store_vec(T *p, const T (&v)[VW]) {
    if constexpr (sizeof(T) * VW == 16 && sizeof(T) == 4)
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (sizeof(T) * VW == 16)
        *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    else if constexpr (sizeof(T) * VW == 8 && VW == 2)
        *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
    else
        p[0] = v[0];
}
template <typename T, int VW>
__device__ __forceinline__ void load_vec(const T *p, T (&v)[VW]) {
    if constexpr (sizeof(T) * VW == 16 && sizeof(T) == 4) {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (sizeof(T) * VW == 16) {
        const double2 t = *reinterpret_cast<const double2 *>(p);
        v[0] = t.x; v[1] = t.y;
    } else if constexpr (sizeof(T) * VW == 8 && VW == 2) {
        const float2 t = *reinterpret_cast<const float2 *>(p);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = p[0];
    }
}

// The Gram product M diag(d) M^T of the NP-row columns in Mt as a TR x TC tile
// per lane, rows from r0, columns from c0: acc[t][u] = sum_l fma(M[r0+t][l] d_l,
// M[c0+u][l], .) in ascending l; FP32 two rows an instruction (fma.rn.f32x2).
template <typename T, int TR, int TC>
__device__ __forceinline__ void gram_tile(const T *Mt, uint32_t ldt, const T *dv, uint32_t L, uint32_t r0, uint32_t c0,
                                          T (&acc)[TR][TC]) {
    if constexpr (sizeof(T) == 4) {
        unsigned long long s[TR / 2][TC];
#pragma unroll
        for (int t = 0; t < TR / 2; ++t)
#pragma unroll
            for (int u = 0; u < TC; ++u) s[t][u] = 0ull;
        const T *a = Mt + r0, *b = Mt + c0;
#pragma unroll 2
        for (uint32_t l = 0; l < L; ++l, a += ldt, b += ldt) {
            const float d = dv[l];
            const unsigned long long dd = gbdpcg::pack2(d, d);
            unsigned long long ad[TR / 2];
#pragma unroll
            for (int t = 0; t < TR / 2; ++t)
                ad[t] = gbdpcg::mul2(*reinterpret_cast<const unsigned long long *>(a + 2 * t), dd);
#pragma unroll
            for (int u = 0; u < TC; ++u) {
                const unsigned long long bb = gbdpcg::pack2(b[u], b[u]);
#pragma unroll
                for (int t = 0; t < TR / 2; ++t) s[t][u] = gbdpcg::fma2(ad[t], bb, s[t][u]);
            }
        }
#pragma unroll
        for (int t = 0; t < TR / 2; ++t)
#pragma unroll
            for (int u = 0; u < TC; ++u) {
                acc[2 * t][u] = gbdpcg::lo2(s[t][u]);
                acc[2 * t + 1][u] = gbdpcg::hi2(s[t][u]);
            }
    } else {
#pragma unroll
        for (int t = 0; t < TR; ++t)
#pragma unroll
            for (int u = 0; u < TC; ++u) acc[t][u] = T(0);
#pragma unroll 2
        for (uint32_t l = 0; l < L; ++l) {
            const T d = dv[l];
            T b[TC];
#pragma unroll
            for (int u = 0; u < TC; ++u) b[u] = Mt[l * ldt + c0 + u];
#pragma unroll
            for (int t = 0; t < TR; ++t) {
                const T ad = Mt[l * ldt + r0 + t] * d;
#pragma unroll
                for (int u = 0; u < TC; ++u) acc[t][u] += ad * b[u];
            }
        }
    }
}

// Schur formation: a warp forms kw knots in turn (1; with the fused inverse up to
// as many as it then inverts at once).  The Gram product S_kk = M diag(d) M^T is a
// 2D register tile per lane: lanes form a 4 x 8 grid, lane (rg, cg) owns rows
// rg TR .. rg TR + TR - 1 and columns cg TC .. cg TC + TC - 1 of the NP x NP
// product (TR = NP / 4, TC = NP / 8).  It is rounded as in gram_tile, then + Qi_{k+1}
// on the diagonal, and symmetrised as 0.5 (S + S^T) through shared memory.  With
// PINV the warp then inverts the symmetrised S_kk (the block-Jacobi builder's own
// routine and rounding) and writes the compact block-Jacobi Phi^-1, so the
// preconditioner is built with S and never re-read.
//
// VW: elements of one global access (16 bytes where n is a multiple of their
// number and the arrays are aligned, else 8, else one element).  The blocks are
// contiguous, so a warp walks them in pieces of VW with one division an access.
//
// What bounds it: instruction issue and the shared-memory pipe (n=24, m=12: 5930
// instructions a knot with one element an access, one row an FMA and a select an
// element of the inverse; now 4035, the pipe 84% busy).  Measured, us, before
// and now, N=65536 FP32: n=24 m=12 212 -> 183, with Phi^-1 382 -> 322; n=14 m=7
// 114 -> 102, 198 -> 140; n=6 m=3 with Phi^-1 96 -> 56.  FP64 is bound by the FP64
// pipe (n=14 m=7 N=30000 with Phi^-1 1365 -> 862), so it takes 16-byte accesses only
// with Phi^-1 (n=24 m=12 N=4096 without 274 us, 243 with 8 bytes; with Phi^-1 422
// and 475).
//
// CTAs an SM that the registers allow: as many as hide the latency of a knot's
// stages.  FP32 n=31 m=15 with five and its S_kk stored twice 327 us, with Phi^-1
// 631; now 310 and 561; n=32 m=32 with Phi^-1 688 -> 580; n=3 m=1 40 -> 34; FP64
// n=24 m=12 N=4096 with six 274 us, now 241.
template <typename T, int NP, bool PINV>
constexpr int schur_ctas() {
    if (sizeof(T) == 8) return 8;
    if (PINV) return NP <= 24 ? 7 : 6;
    return NP <= 8 ? 12 : (NP <= 24 ? 7 : 8);
}
template <typename T, int NP, int W, bool PINV, int VW>
__global__ void __launch_bounds__(W * 32, schur_ctas<T, NP, PINV>())
    form_schur_kernel(const T *__restrict__ A, const T *__restrict__ B, const T *__restrict__ Qd,
                      const T *__restrict__ Rd, const T *__restrict__ q, const T *__restrict__ r,
                      const T *__restrict__ c, uint32_t n, uint32_t m, uint32_t N, uint32_t kw, T *__restrict__ S,
                      T *__restrict__ gamma, T *__restrict__ Pinv) {
    constexpr int TR = NP / 4, TC = NP / 8, GL = gbdpcg::gj_lanes(NP);
    constexpr uint32_t ldt = schur_ldt<NP>(), xs = NP + 1, KW = PINV ? schur_knots<NP>() : 1;
    extern __shared__ __align__(16) unsigned char schur_smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t k0 = (blockIdx.x * W + warp) * kw;
    if (k0 >= N) return;  // warp-uniform; no CTA barrier below
    const uint32_t L = n + m, L4 = (L + 3) & ~3u, nn = n * n;
    T *Mt = reinterpret_cast<T *>(schur_smem) + (size_t)warp * schur_warp_elems<NP, PINV>(L);
    T *X = Mt, *dv = Mt + schur_mt_elems<NP>(L), *dw = dv + L4, *qn = dw + L4, *Y = qn + 32, *s = Y + (PINV && KW > 1 ? KW * NP * ldt : 0);
    // pieces of VW elements: n / VW in a column; x / cv = (x magic) >> 16 for x < 2048
    const uint32_t cv = n / VW, magic = (65536u + cv - 1) / cv;
    const uint32_t kend = min(k0 + kw, N);
    for (uint32_t k = k0; k < kend; ++k) {
        const T *Ak = A + (size_t)k * nn, *Bk = B + (size_t)k * n * m;
        // every column in flight at once (cp.async)
        for (uint32_t e = lane; e < L * cv; e += 32) {
            const uint32_t l = (e * magic) >> 16, p = (e - l * cv) * VW;
            cp_async_vec<T, VW>(Mt + l * ldt + p, l < n ? Ak + e * VW : Bk + (e - n * cv) * VW);
        }
        if (n < (uint32_t)NP)  // rows n..NP-1
            for (uint32_t l = lane; l < L; l += 32)
                for (uint32_t p = n; p < (uint32_t)NP; ++p) Mt[l * ldt + p] = T(0);
        if (lane < n) {
            const T d = T(1) / Qd[(size_t)k * n + lane];
            dv[lane] = d;
            dw[lane] = d * q[(size_t)k * n + lane];
            qn[lane] = T(1) / Qd[(size_t)(k + 1) * n + lane];
        }
        if (lane < m) {
            const T d = T(1) / Rd[(size_t)k * m + lane];
            dv[n + lane] = d;
            dw[n + lane] = d * r[(size_t)k * m + lane];
        }
        cp_async_wait_all();
        __syncwarp();
        T *Sk = S + (size_t)k * 3 * nn;
        // block 0 of row k: S_{k,k-1}, element (i, j) = -Qi_k[j] A_k[i][j]; block 2
        // of row k-1: S_{k-1,k}, element (i, j) = -Qi_k[i] A_k[j][i] (this warp holds
        // A_k, so each A_k is read once); the last row's block 2 is padding
        T *Sup = (k > 0) ? S + (size_t)(k - 1) * 3 * nn + 2 * (size_t)nn : nullptr;
        for (uint32_t e = lane; e < n * cv; e += 32) {
            const uint32_t col = (e * magic) >> 16, p = (e - col * cv) * VW;
            T v[VW], w[VW], d[VW];
            if (k > 0) {
                load_vec<T, VW>(Mt + col * ldt + p, v);
                load_vec<T, VW>(dv + p, d);
#pragma unroll
                for (int u = 0; u < VW; ++u) {
                    v[u] = -dv[col] * v[u];
                    w[u] = -d[u] * Mt[(p + u) * ldt + col];
                }
                store_vec<T, VW>(Sup + e * VW, w);
            } else {
#pragma unroll
                for (int u = 0; u < VW; ++u) v[u] = T(0);
            }
            store_vec<T, VW>(Sk + e * VW, v);
            if (k + 1 == N) {
#pragma unroll
                for (int u = 0; u < VW; ++u) v[u] = T(0);
                store_vec<T, VW>(Sk + 2 * (size_t)nn + e * VW, v);
            }
        }
        // gamma_k = -(c_k + M diag(d) w - Qi_{k+1} q_{k+1})
        if (lane < n) {
            T g = T(0);
#pragma unroll 4
            for (uint32_t l = 0; l < L; ++l) g += Mt[l * ldt + lane] * dw[l];
            gamma[(size_t)k * n + lane] = -(c[(size_t)k * n + lane] + g - qn[lane] * q[(size_t)(k + 1) * n + lane]);
        }
        const uint32_t r0 = (lane >> 3) * TR, c0 = (lane & 7) * TC;
        T acc[TR][TC];
        gram_tile<T, TR, TC>(Mt, ldt, dv, L, r0, c0, acc);
        __syncwarp();  // every lane is done with Mt: it now holds the product, row stride NP + 1
#pragma unroll
        for (int t = 0; t < TR; ++t)
#pragma unroll
            for (int u = 0; u < TC; ++u) {
                const uint32_t i = r0 + t, j = c0 + u;
                if (i < n && j < n) X[i * xs + j] = (i == j) ? acc[t][u] + qn[i] : acc[t][u];
            }
        __syncwarp();
        // block 1: S_kk symmetrised, kept for the inverse
        T *Yk = Y + (k - k0) * NP * ldt;
        for (uint32_t e = lane; e < n * cv; e += 32) {
            const uint32_t col = (e * magic) >> 16, p = (e - col * cv) * VW;
            T v[VW];
#pragma unroll
            for (int u = 0; u < VW; ++u) v[u] = T(0.5) * (X[(p + u) * xs + col] + X[col * xs + p + u]);
            store_vec<T, VW>(Sk + nn + e * VW, v);
            if constexpr (PINV && KW > 1) store_vec<T, VW>(Yk + col * ldt + p, v);
        }
        __syncwarp();  // X is free for the next knot's columns, Y complete
    }
    if constexpr (PINV) {
        // group g of GL lanes: knot k0 + g; lane rr: row rr of the symmetrised S_kk
        // (the values just written), identity beyond n
        const uint32_t g = lane / GL, rr = lane % GL;
        const bool mine = k0 + g < kend && rr < n;
        T *Yg = KW > 1 ? Y + g * NP * ldt : X;
        T a[NP];
#pragma unroll
        for (int cc = 0; cc < NP; ++cc) {
            a[cc] = (uint32_t)cc == rr ? T(1) : T(0);
            if (mine && (uint32_t)cc < n) a[cc] = KW > 1 ? Yg[cc * ldt + rr] : T(0.5) * (Yg[rr * xs + cc] + Yg[cc * xs + rr]);
        }
        const T diag = mine ? Yg[rr * (KW > 1 ? ldt : xs) + rr] : T(1);
        T *sg = s + g * 3 * GL;
        bool ok;
        const T h = T(0.5) * gbdpcg::gj_inverse<T, NP, GL>(a, diag, mine, sg, rr, ok);  // ends with a warp sync: Y is free
        if (!__all_sync(0xffffffffu, ok)) {
            if constexpr (KW > 1) {
                for (uint32_t k = k0; k < kend; ++k)
                    gbdpcg::gj_invert_any(Y + (k - k0) * NP * ldt, ldt, Pinv + (size_t)k * nn, false, n, s, lane);
            } else {
                for (uint32_t cc = 0; lane < n && cc < lane; ++cc)
                    X[lane * xs + cc] = X[cc * xs + lane] = T(0.5) * (X[lane * xs + cc] + X[cc * xs + lane]);
                gbdpcg::gj_invert_any(X, xs, Pinv + (size_t)k0 * nn, false, n, s, lane);
            }
            return;
        }
        const T *D = sg + 2 * GL;
        T *Xg = Yg;
        if (rr < (uint32_t)NP) {
#pragma unroll
            for (int cc = 0; cc < NP; ++cc) Xg[rr * xs + cc] = a[cc];
        }
        __syncwarp();
        if (mine) {  // symmetrised, compact n^2 per knot, column-major
            T *Pk = Pinv + (size_t)(k0 + g) * nn;
#pragma unroll
            for (int cc = 0; cc < NP; ++cc)
                if ((uint32_t)cc < n) Pk[cc * n + rr] = gbdpcg::mul_pow2(a[cc] + Xg[cc * xs + rr], h, D[cc]);
        }
    }
}

// s + sum_j col[j] w[j], j ascending, VW elements an access (n a multiple of VW,
// both addresses aligned to it), U accesses an iteration (0: as the compiler has it).
template <typename T, int VW, int U>
__device__ __forceinline__ T col_dot(const T *col, const T *w, uint32_t n, T s) {
    auto add = [&](uint32_t j) {
        T a[VW], b[VW];
        load_vec<T, VW>(col + j, a);
        load_vec<T, VW>(w + j, b);
#pragma unroll
        for (int u = 0; u < VW; ++u) s += a[u] * b[u];
    };
    if constexpr (U == 0) {
        for (uint32_t j = 0; j < n; j += VW) add(j);
    } else {
#pragma unroll U
        for (uint32_t j = 0; j < n; j += VW) add(j);
    }
    return s;
}

// Back-substitution: a lane per column of [A_k | B_k] (element l of x_k for l < n,
// of u_k beyond), GL lanes a knot, so that both blocks go in one pass and a warp
// takes two knots of n + m <= 16 or four of n + m <= 8.  From 25 columns on (TWO)
// the columns of A_k go first, then those of B_k: together their lines outgrow the
// L1 of an SM's 64 warps (n=24 m=12: 55 us against 50; n=24 m=8 46 / 44, n=16 m=8
// 31.3 / 32.0).  A lane reads its own
// contiguous column with accesses of 16 or 8 bytes where n and the addresses allow,
// U an iteration: one for 16-byte accesses in one pass and for FP64 in one pass, four
// for FP64 in two, as the compiler has it for the rest (n=13 m=6 N=60000: 21.7 us so,
// 23.6 with four).
//
// What bounds it: HBM and, for short columns, the L1 requests (a column is 24 to
// 128 bytes).  Measured, us, before (one pass for A_k, one for B_k, one element an
// access unless n is a multiple of 4) and now, one problem again and again (n=14: its
// 70 MB lie in the L2) / eight problems in turn (n=6: in the L2 still): n=14
// m=7 N=60000 27.6 -> 21.7 / 31.6 -> 25.2, n=6 m=3 21.3 -> 10.2 / 27.0 -> 12.5, n=12
// m=6 19.2 -> 14.9 / 27.4 -> 18.8, n=13 m=6 25.2 -> 21.7 / 30.3 -> 25.0, n=22 m=11
// 56.1 -> 42.6 / 55.8 -> 42.3; FP64 n=14 m=7 N=30000 81.8 -> 60.4 / 82.4 -> 62.0.
// n=24 m=12 (47.5) and FP64 of 25 columns or more, bound by its pipe, are
// as they were.
template <typename T, int GL, int VW, bool TWO, int kKktWarps>
__global__ void __launch_bounds__(kKktWarps * 32)
    kkt_backsub_kernel(const T *__restrict__ A, const T *__restrict__ B, const T *__restrict__ Qd,
                       const T *__restrict__ Rd, const T *__restrict__ q, const T *__restrict__ r,
                       const T *__restrict__ lambda, uint32_t n, uint32_t m, uint32_t N, T *__restrict__ x,
                       T *__restrict__ u) {
    constexpr int U = sizeof(T) == 8 ? (TWO ? 4 : 1) : (VW == 4 && !TWO ? 1 : 0);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t k = (blockIdx.x * kKktWarps + (threadIdx.x >> 5)) * (32 / GL) + lane / GL;
    if (k > N) return;  // knots 0..N (x) and 0..N-1 (u)
    const T *lk = lambda + (size_t)k * n;
    if constexpr (TWO) {
        const uint32_t l = lane;
        if (l < n) {
            T s = q[(size_t)k * n + l];
            if (k < N) s = col_dot<T, VW, U>(A + ((size_t)k * n + l) * n, lk, n, s);
            if (k > 0) s -= lambda[(size_t)(k - 1) * n + l];
            x[(size_t)k * n + l] = -s / Qd[(size_t)k * n + l];
        }
        if (k < N && l < m) {
            const T s = col_dot<T, VW, U>(B + ((size_t)k * m + l) * n, lk, n, r[(size_t)k * m + l]);
            u[(size_t)k * m + l] = -s / Rd[(size_t)k * m + l];
        }
        return;
    } else for (uint32_t l = lane % GL; l < (k < N ? n + m : n); l += GL) {
        const bool is_x = l < n;
        const size_t e = is_x ? (size_t)k * n + l : (size_t)k * m + (l - n);
        T s = is_x ? q[e] : r[e];
        const T d = is_x ? Qd[e] : Rd[e];
        if (k < N)  // + (A_k^T lambda_k)_i = sum_j A_k[j][i] lambda_k[j], B_k^T lambda_k alike
            s = col_dot<T, VW, U>(is_x ? A + ((size_t)k * n + l) * n : B + ((size_t)k * m + (l - n)) * n, lk, n, s);
        if (is_x) {
            if (k > 0) s -= lambda[(size_t)(k - 1) * n + l];
            x[e] = -s / d;
        } else {
            u[e] = -s / d;
        }
    }
}

int check(const void *const *ptrs, int np, uint32_t n, uint32_t m, uint32_t N) {
    for (int i = 0; i < np; ++i)
        if (!ptrs[i]) {
            gbdpcg::set_last_error("NULL pointer");
            return GBDPCG_ERR_INVALID_ARGUMENT;
        }
    if (n == 0 || m == 0 || N == 0) {
        gbdpcg::set_last_error("n, m and N must be positive");
        return GBDPCG_ERR_INVALID_ARGUMENT;
    }
    if (n > (uint32_t)kKktMaxN || m > (uint32_t)kKktMaxN) {
        gbdpcg::set_last_error("n and m must be <= 32");
        return GBDPCG_ERR_UNSUPPORTED;
    }
    return GBDPCG_SUCCESS;
}

int launched(const char *what) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        gbdpcg::set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
        return GBDPCG_ERR_CUDA;
    }
    return GBDPCG_SUCCESS;
}

template <typename T>
int form_schur(const T *A, const T *B, const T *Qd, const T *Rd, const T *q, const T *r, const T *c, uint32_t n,
               uint32_t m, uint32_t N, T *S, T *gamma, T *Pinv, cudaStream_t st) {
    const void *p[] = {A, B, Qd, Rd, q, r, c, S, gamma};
    int rc = check(p, 9, n, m, N);
    if (rc) return rc;
    constexpr int W = kkt_warps<T>();
    // elements of an access: what n and the blocks' addresses allow (FP64 without
    // Phi^-1: one, see the kernel)
    const uintptr_t at = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(S);
    constexpr uint32_t V16 = 16 / sizeof(T);
    const bool v16 = (sizeof(T) == 4 || Pinv) && n % V16 == 0 && (at & 15u) == 0, v8 = sizeof(T) == 4 && n % 2 == 0 && (at & 7u) == 0;
    auto go = [&](auto np) -> int {
        constexpr int NP = decltype(np)::value;
        auto launch = [&](auto kern, size_t smem, uint32_t knots) -> int {
            // (within the 48 KB that any kernel may have: no launch attribute, which
            // threads would set under one another)
            static_assert(W * sizeof(T) * schur_warp_elems<NP, true>(kKktMaxN + (NP < kKktMaxN ? NP : kKktMaxN)) <= 48 * 1024,
                          "shared memory of the formation");
            // few knots: one a warp, side by side (n=14 N=500: 10.5 us against 11.8
            // with two in turn); as many as a warp inverts at once from the knots
            // on that fill the GPU's warps
            if (N <= 4096) knots = 1;
            kern<<<(N + W * knots - 1) / (W * knots), W * 32, smem, st>>>(A, B, Qd, Rd, q, r, c, n, m, N, knots, S, gamma,
                                                                          Pinv);
            return launched("form_schur");
        };
        auto width = [&](auto vw) -> int {
            constexpr int VW = decltype(vw)::value;
            const size_t w = (size_t)W * sizeof(T);
            return Pinv ? launch(form_schur_kernel<T, NP, W, true, VW>, w * schur_warp_elems<NP, true>(n + m), schur_knots<NP>())
                        : launch(form_schur_kernel<T, NP, W, false, VW>, w * schur_warp_elems<NP, false>(n + m), 1);
        };
        if (v16) return width(std::integral_constant<int, (int)V16>());
        if constexpr (sizeof(T) == 4)
            if (v8) return width(std::integral_constant<int, 2>());
        return width(std::integral_constant<int, 1>());
    };
    if (n <= 8) return go(std::integral_constant<int, 8>());
    if (n <= 16) return go(std::integral_constant<int, 16>());
    if (n <= 24) return go(std::integral_constant<int, 24>());
    return go(std::integral_constant<int, 32>());
}

template <typename T>
int kkt_backsub(const T *A, const T *B, const T *Qd, const T *Rd, const T *q, const T *r, const T *lambda,
                uint32_t n, uint32_t m, uint32_t N, T *x, T *u, cudaStream_t st) {
    const void *p[] = {A, B, Qd, Rd, q, r, lambda, x, u};
    int rc = check(p, 9, n, m, N);
    if (rc) return rc;
    constexpr int W = 4;
    const uintptr_t at =
        reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(lambda);
    constexpr uint32_t V16 = 16 / sizeof(T);
    auto go = [&](auto gl, auto two, auto vw) {
        constexpr int GL = decltype(gl)::value, VW = decltype(vw)::value, K = W * (32 / GL);
        kkt_backsub_kernel<T, GL, VW, decltype(two)::value, W>
            <<<N / K + 1, W * 32, 0, st>>>(A, B, Qd, Rd, q, r, lambda, n, m, N, x, u);
    };
    auto width = [&](auto gl, auto two) {
        if (n % V16 == 0 && (at & 15u) == 0) return go(gl, two, std::integral_constant<int, (int)V16>());
        if constexpr (sizeof(T) == 4)
            if (n % 2 == 0 && (at & 7u) == 0) return go(gl, two, std::integral_constant<int, 2>());
        go(gl, two, std::integral_constant<int, 1>());
    };
    const std::false_type one;
    if (n + m <= 8) width(std::integral_constant<int, 8>(), one);
    else if (n + m <= 16) width(std::integral_constant<int, 16>(), one);
    else if (n + m <= 24) width(std::integral_constant<int, 32>(), one);
    else width(std::integral_constant<int, 32>(), std::true_type());
    return launched("kkt_backsub");
}

}  // namespace

extern "C" {

int gbdpcg_form_schur_f32(const float *d_A, const float *d_B, const float *d_Qd, const float *d_Rd,
                          const float *d_q, const float *d_r, const float *d_c, uint32_t n, uint32_t m, uint32_t N,
                          float *d_S, float *d_gamma, gbdpcg_stream_t stream) {
    return form_schur<float>(d_A, d_B, d_Qd, d_Rd, d_q, d_r, d_c, n, m, N, d_S, d_gamma, nullptr,
                             (cudaStream_t)stream);
}
int gbdpcg_form_schur_f64(const double *d_A, const double *d_B, const double *d_Qd, const double *d_Rd,
                          const double *d_q, const double *d_r, const double *d_c, uint32_t n, uint32_t m, uint32_t N,
                          double *d_S, double *d_gamma, gbdpcg_stream_t stream) {
    return form_schur<double>(d_A, d_B, d_Qd, d_Rd, d_q, d_r, d_c, n, m, N, d_S, d_gamma, nullptr,
                              (cudaStream_t)stream);
}
int gbdpcg_form_schur_pinv_f32(const float *d_A, const float *d_B, const float *d_Qd, const float *d_Rd,
                               const float *d_q, const float *d_r, const float *d_c, uint32_t n, uint32_t m,
                               uint32_t N, float *d_S, float *d_gamma, float *d_Pinv, gbdpcg_stream_t stream) {
    if (!d_Pinv) {
        gbdpcg::set_last_error("NULL pointer");
        return GBDPCG_ERR_INVALID_ARGUMENT;
    }
    return form_schur<float>(d_A, d_B, d_Qd, d_Rd, d_q, d_r, d_c, n, m, N, d_S, d_gamma, d_Pinv,
                             (cudaStream_t)stream);
}
int gbdpcg_form_schur_pinv_f64(const double *d_A, const double *d_B, const double *d_Qd, const double *d_Rd,
                               const double *d_q, const double *d_r, const double *d_c, uint32_t n, uint32_t m,
                               uint32_t N, double *d_S, double *d_gamma, double *d_Pinv, gbdpcg_stream_t stream) {
    if (!d_Pinv) {
        gbdpcg::set_last_error("NULL pointer");
        return GBDPCG_ERR_INVALID_ARGUMENT;
    }
    return form_schur<double>(d_A, d_B, d_Qd, d_Rd, d_q, d_r, d_c, n, m, N, d_S, d_gamma, d_Pinv,
                              (cudaStream_t)stream);
}
int gbdpcg_kkt_backsub_f32(const float *d_A, const float *d_B, const float *d_Qd, const float *d_Rd,
                           const float *d_q, const float *d_r, const float *d_lambda, uint32_t n, uint32_t m,
                           uint32_t N, float *d_x, float *d_u, gbdpcg_stream_t stream) {
    return kkt_backsub<float>(d_A, d_B, d_Qd, d_Rd, d_q, d_r, d_lambda, n, m, N, d_x, d_u, (cudaStream_t)stream);
}
int gbdpcg_kkt_backsub_f64(const double *d_A, const double *d_B, const double *d_Qd, const double *d_Rd,
                           const double *d_q, const double *d_r, const double *d_lambda, uint32_t n, uint32_t m,
                           uint32_t N, double *d_x, double *d_u, gbdpcg_stream_t stream) {
    return kkt_backsub<double>(d_A, d_B, d_Qd, d_Rd, d_q, d_r, d_lambda, n, m, N, d_x, d_u, (cudaStream_t)stream);
}

}  // extern "C"
