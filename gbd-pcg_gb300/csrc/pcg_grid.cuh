// PCG of one long system over the whole GPU: one CTA per SM, knots split over
// the CTAs, in a cooperative launch (every CTA resident, as the reference's
// kernel needs, include/pcg.cuh:43-46).  For a lone system that a cluster's 16
// SMs hold badly or not at all: its rows then have up to 152 SMs' caches, load
// units and FP64 pipes instead of 16.
//
// Arithmetic and exit tests are pcg_cluster_kernel's standard form
// (include/pcg.cuh:119-208).  The rows of S are held in registers where a CTA's
// fit (one a thread; n=14 FP32: 54 knots an SM), else they are read in every
// product as in pcg_stream_kernel, and so is Phi^-1, with read-only loads that
// the SM's L1 keeps.
//
// The reference's four grid barriers an iteration become two exchanges through
// mailboxes in global memory.  A mailbox word is 8 bytes: 32 bits of payload and
// the number of the exchange, written and read as one access, so a word that
// carries the right number is complete and no fence or barrier counter is
// needed.  Per exchange every CTA posts its sum of each reduced value once; one
// warp per value polls the words of all CTAs (5 a lane for 152), adds them in
// rank order and a butterfly, and evaluates the quotient and the exit tests,
// while another warp polls each neighbour's boundary values; a CTA barrier
// hands the results to every thread.  All CTAs add the same words in the same
// order, so they take the same decisions.  Two sets of mailboxes alternate: a
// CTA posts exchange e + 2 only after it has read every CTA's word of e + 1,
// which that CTA posted after it had read all of e.
//
// Every wait gives up after about a second (the CTAs start together: beside another
// solve that held one SM for 2.5 s, the launch waited and no wait ran out).  A CTA
// that gives up uses none of the words it has and posts none any more: it ends as
// TIMEOUT, and so does, a wait later, every CTA that needs its next word.  CTA 0,
// whose status is the solve's, needs a word of every CTA to go on, so it reports
// another end only if all that was left to do was to stop.
//
// Every CTA posts to mailboxes of each receiver's own (152 words a value): with
// one word a CTA that all poll, 152 SMs queue at the same few lines (3.5 us an
// exchange instead of 2.3).
//
// What bounds it: two exchanges an iteration (stores to L2, a poll from it, the
// CTA-wide stages: about 2.3 us each), then the products (n=14 N=8192: 1.3 us
// with S in registers, 2.7 from the L1).  One system of n=14 N=8192 FP32, 39
// passes, device time: 2150 us with streamed rows on 16 SMs, 240 us here, 299 with S
// from the L1; N=20000 5916 against 445.  The rule with both sides measured is
// grid_pays in capi.cu.
#pragma once
#include "pcg_cluster.cuh"

namespace gbdpcg {

// CTA size bound.  Rows of S in registers (REG): what 64K registers hold at the
// 3 NP words of a row and about 40 (FP64: 70) more.  Streamed rows: 64 registers
// a thread, 128 where a row's chunk of a block and of its window take more
// (FP64, wide blocks).
template <typename T, int NP, bool REG>
constexpr int grid_threads() {
    if (!REG) return sizeof(T) == 8 || NP > 16 ? 512 : 1024;
    if (sizeof(T) == 8) return NP <= 8 ? 512 : (NP <= 16 ? 384 : 256);
    return NP <= 6 ? 1024 : (NP <= 8 ? 896 : (NP <= 14 ? 768 : (NP <= 16 ? 640 : (NP <= 24 ? 512 : 384))));
}

template <typename T, typename A, int NP, bool PTRI>
struct SmemPlanGrid {
    __host__ __device__ static size_t vec(uint32_t kmax) { return round_up((size_t)(kmax + 2) * NP * sizeof(T), 32); }
    __host__ __device__ static size_t halo() { return round_up((size_t)2 * NP * sizeof(T), 32); }
    // partials of the warps (float: one a warp; double: one a lane)
    __host__ __device__ static size_t part(uint32_t nwarps) {
        return round_up((size_t)2 * 32 * (kOneWarpSums<A> ? nwarps : 1) * sizeof(A), 32);
    }
    __host__ __device__ static size_t bytes(uint32_t kmax, uint32_t, uint32_t nwarps) {
        return 2 * vec(kmax) + 2 * halo() + part(nwarps) + 128;
    }
};

__device__ __forceinline__ void mail_post(uint64_t *p, uint32_t seq, uint32_t payload) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((uint64_t)seq << 32 | payload) : "memory");
}
__device__ __forceinline__ uint64_t mail_peek(const uint64_t *p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// 32-bit words of a value
template <typename V>
__device__ __forceinline__ uint32_t word_of(V v, int w) {
    if constexpr (sizeof(V) == 8) return (uint32_t)(w ? __double2hiint(v) : __double2loint(v));
    else return __float_as_uint(v);
}
template <typename V>
__device__ __forceinline__ V from_words(uint32_t lo, uint32_t hi) {
    if constexpr (sizeof(V) == 8) return __hiloint2double((int)hi, (int)lo);
    else return __uint_as_float(lo);
}

// A bounded spin: counts the failed polls and gives up after `limit` ns.
struct SpinLimit {
    uint64_t t0 = 0;
    uint32_t spins = 0;
    __device__ __forceinline__ bool expired(volatile uint32_t *timed_out, uint64_t limit) {
        if (*timed_out) return true;
        if (spins == 0) t0 = global_ns();
        if ((++spins & 63u) == 0 && global_ns() - t0 > limit) *timed_out = 1u;
        return *timed_out != 0;
    }
};

// What an exchange leaves in shared memory.
template <typename T, typename A>
struct GridOut {
    A sum[2];
    T ratio;
    uint32_t code[2];
    uint32_t timed_out;
};

// One exchange: the sums over all CTAs of NQ values (in v, identical in every
// thread of every CTA), and, with `halos`, the neighbours' boundary values
// posted for this exchange, from the left into hl and from the right into hr.
// fin(q, sum, out): run by the warp that added value q (quotient, exit tests).
// Returns whether it is complete.
template <typename T, typename A, int NP, bool PROBE, int NQ, typename F>
__device__ __forceinline__ bool grid_exchange(A (&v)[NQ], A *part, GridOut<T, A> *out, const GridParams &gp, uint32_t &seq,
                                              uint32_t C, uint32_t rank, uint32_t n, bool halos, T *hl, T *hr, F &&fin) {
    constexpr int NW = sizeof(A) / 4, TW = sizeof(T) / 4;
    constexpr uint32_t kHaloWords = 2 * NP;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint64_t limit = PROBE ? gp.probe_limit_ns : 1000000000ull;
    ++seq;
    const uint32_t buf = seq & 1u;
    // [receiver][word][sender]: every CTA polls lines of its own
    uint64_t *sums = gp.sums + (size_t)buf * kGridWords * C * C;
    if constexpr (kOneWarpSums<A>) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) part[((uint32_t)q * nwarps + warp) * 32 + lane] = v[q];
    } else {
        A t[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) t[q] = v[q];
        warp_sum_n<A, NQ>(t);
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) part[q * 32 + warp] = t[q];
        }
    }
    __syncthreads();
    for (uint32_t job = warp; job < (uint32_t)NQ + (halos ? 2u : 0u); job += nwarps) {
        if (job < (uint32_t)NQ) {
            // this CTA's sum of value `job`
            A t[1];
            if constexpr (kOneWarpSums<A>) {
                const A *x = part + (size_t)job * nwarps * 32 + lane;
                A c1 = A(0);
                t[0] = x[0];
                uint32_t w = 1;
                for (; w + 1 < nwarps; w += 2) {
                    t[0] += x[w * 32];
                    c1 += x[w * 32 + 32];
                }
                if (w < nwarps) t[0] += x[w * 32];
                t[0] += c1;
            } else {
                t[0] = lane < nwarps ? part[job * 32 + lane] : A(0);
            }
            warp_sum_n<A, 1>(t);
#pragma unroll
            for (uint32_t u = 0; u < kGridMaxCtas / 32; ++u) {
                const uint32_t to = u * 32 + lane;
                if (to < C && !(PROBE && seq == gp.probe_seq && rank == gp.probe_from && to == gp.probe_to)) {
#pragma unroll
                    for (int k = 0; k < NW; ++k)
                        mail_post(sums + ((size_t)to * kGridWords + job * 2 + k) * C + rank, seq, word_of(t[0], k));
                }
            }
            // every CTA's word, all loads of a lane in flight
            const uint64_t *in = sums + ((size_t)rank * kGridWords + job * 2) * C;
            uint64_t w[kGridMaxCtas / 32][NW];
            SpinLimit spin;
            for (;;) {
                bool ok = true;
#pragma unroll
                for (uint32_t u = 0; u < kGridMaxCtas / 32; ++u) {
                    const uint32_t r = u * 32 + lane;
                    if (u * 32 < C) {
#pragma unroll
                        for (int k = 0; k < NW; ++k) w[u][k] = r < C ? mail_peek(in + (size_t)k * C + r) : (uint64_t)seq << 32;
                    }
                }
#pragma unroll
                for (uint32_t u = 0; u < kGridMaxCtas / 32; ++u) {
                    if (u * 32 < C) {
#pragma unroll
                        for (int k = 0; k < NW; ++k) ok = ok && (uint32_t)(w[u][k] >> 32) == seq;
                    }
                }
                if (__all_sync(0xffffffffu, ok)) break;
                const bool late = spin.expired(&out->timed_out, limit);
                if (__any_sync(0xffffffffu, late)) break;
            }
            A s[1] = {A(0)};
#pragma unroll
            for (uint32_t u = 0; u < kGridMaxCtas / 32; ++u)
                if (u * 32 < C) s[0] += from_words<A>((uint32_t)w[u][0], (uint32_t)w[u][NW - 1]);
            warp_sum_n<A, 1>(s);
            if (lane == 0) out->sum[job] = s[0];
            fin((int)job, s[0], out, lane);
        } else {
            const uint32_t side = job - NQ;  // 0: from the left neighbour, 1: from the right
            if (side == 0 ? rank > 0 : rank + 1 < C) {
                const uint64_t *in = gp.halos + (((size_t)buf * C + rank) * 2 + side) * kHaloWords;
                uint32_t *dst = reinterpret_cast<uint32_t *>(side == 0 ? hl : hr);
                SpinLimit spin;
                for (uint32_t e = lane; e < n * TW; e += 32) {
                    uint64_t w = mail_peek(in + e);
                    while ((uint32_t)(w >> 32) != seq) {
                        if (spin.expired(&out->timed_out, limit)) break;
                        w = mail_peek(in + e);
                    }
                    dst[e] = (uint32_t)w;
                }
            }
        }
        __syncwarp();
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = out->sum[q];
    return out->timed_out == 0u;
}

// Posts row i's boundary value for the next exchange into neighbour `to`'s
// mailbox (side 0: `to` receives it from its left, 1: from its right).
template <typename T, int NP>
__device__ __forceinline__ void grid_post_halo(const GridParams &gp, uint32_t seq, uint32_t C, uint32_t to, uint32_t side,
                                               uint32_t i, T v) {
    constexpr int TW = sizeof(T) / 4;
    uint64_t *m = gp.halos + (((size_t)((seq + 1) & 1u) * C + to) * 2 + side) * (2 * NP) + i * TW;
#pragma unroll
    for (int w = 0; w < TW; ++w) mail_post(m + w, seq + 1, word_of(v, w));
}

// One row times its window from global memory: NB blocks of n columns at M (the
// row's element of the first block's column 0), one FMA chain per present block
// [b0, b1) in ascending column, summed in block order.
template <typename T, int NP, int NB>
__device__ __forceinline__ T grid_row(const T *__restrict__ M, int b0, int b1, const T *x, uint32_t n) {
    T acc[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        acc[b] = T(0);
        if (b < b0 || b >= b1) continue;
        const T *col = M + (size_t)b * n * n, *xb = x + b * NP;
        if (n == (uint32_t)NP) {  // a full block: a chunk's loads all in flight
            constexpr int CH = sizeof(T) == 8 ? 8 : 16, LAST = NP % CH == 0 ? CH : NP % CH;
#pragma unroll
            for (int j0 = 0; j0 < NP; j0 += CH) {
                if (j0 + CH <= NP) {
                    T m[CH], xv[CH];
#pragma unroll
                    for (int j = 0; j < CH; ++j) m[j] = __ldg(col + (size_t)(j0 + j) * NP);
                    lds_row<T, CH>(xv, xb + j0);
#pragma unroll
                    for (int j = 0; j < CH; ++j) acc[b] = fma_rn(m[j], xv[j], acc[b]);
                } else {
                    T m[LAST], xv[LAST];
#pragma unroll
                    for (int j = 0; j < LAST; ++j) m[j] = __ldg(col + (size_t)(j0 + j) * NP);
                    lds_row<T, LAST>(xv, xb + j0);
#pragma unroll
                    for (int j = 0; j < LAST; ++j) acc[b] = fma_rn(m[j], xv[j], acc[b]);
                }
            }
        } else {
#pragma unroll 4
            for (uint32_t j = 0; j < n; ++j) acc[b] = fma_rn(__ldg(col + (size_t)j * n), xb[j], acc[b]);
        }
    }
    T s = acc[0];
#pragma unroll
    for (int b = 1; b < NB; ++b) s += acc[b];
    return s;
}

// G: rows per thread (thread t owns rows t, t + blockDim.x, ... of its CTA).
// REG: the rows of S are held in registers for the whole solve (G = 1); else
// they are read in every product, like Phi^-1 always.
// PROBE: the wait limit is the launch's, and one sum of one exchange is not posted
// (gbdpcg_probe_grid_timeout).
template <typename T, typename A, int NP, bool PTRI, int G, bool REG, bool PROBE = false>
__global__ void __launch_bounds__(grid_threads<T, NP, REG>(), 1) pcg_grid_kernel(const GridParams gp) {
    static_assert(!REG || G == 1, "one row a thread in registers");
    using Plan = SmemPlanGrid<T, A, NP, PTRI>;
    constexpr int NBP = PTRI ? 3 : 1;
    const SysDesc &d = gp.one;
    const uint32_t C = gridDim.x, rank = blockIdx.x, tid = threadIdx.x, nthr = blockDim.x;
    const uint32_t n = d.n, N = d.N, K = gp.kmax;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *sp = smem_raw;
    T *vp = reinterpret_cast<T *>(sp); sp += Plan::vec(K);
    T *vr = reinterpret_cast<T *>(sp); sp += Plan::vec(K);
    T *uh = reinterpret_cast<T *>(sp); sp += Plan::halo();
    T *zh = reinterpret_cast<T *>(sp); sp += Plan::halo();
    A *part = reinterpret_cast<A *>(sp); sp += Plan::part(nthr >> 5);
    GridOut<T, A> *out = reinterpret_cast<GridOut<T, A> *>(sp);
    static_assert(sizeof(GridOut<T, A>) <= 128, "the last bytes of the plan");
    const uint32_t zero_elems = (uint32_t)((2 * Plan::vec(K) + 2 * Plan::halo()) / sizeof(T));
    for (uint32_t e = tid; e < zero_elems; e += nthr) vp[e] = T(0);
    if (tid == 0) out->timed_out = 0u;

    const uint32_t kb = min(rank * K, N), ke = min(kb + K, N), nk = ke - kb;
    const bool relres = (d.flags & SYS_EXIT_RELRES) != 0;
    const T *__restrict__ S = static_cast<const T *>(d.S);
    const T *__restrict__ P = static_cast<const T *>(d.P);
    const T *__restrict__ gamma = static_cast<const T *>(d.gamma);
    const T *lam0 = (d.flags & SYS_LAMBDA0_ZERO) ? nullptr : static_cast<const T *>(d.lambda0);
    const uint32_t blkS = 3 * n * n, blkP = NBP * n * n;
    const bool has_left = kb > 0 && nk > 0, has_right = ke < N && nk > 0;
    if (tid == 0 && nk > 0) {  // the first products' rows into L2 at once
        prefetch_l2_range(S + (size_t)kb * blkS, (size_t)nk * blkS * sizeof(T));
        prefetch_l2_range(P + (size_t)kb * blkP, (size_t)nk * blkP * sizeof(T));
    }
    // this thread's rows: local knot, row in it
    uint32_t lk[G], ri[G];
    bool act[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t row = (uint32_t)g * nthr + tid;
        lk[g] = row / n;
        ri[g] = row - lk[g] * n;
        act[g] = lk[g] < nk;
    }
    auto first = [&](int g) { return act[g] && lk[g] == 0 && kb > 0; };
    auto last = [&](int g) { return act[g] && lk[g] + 1 == nk && ke < N; };
    auto b0 = [&](int g) { return kb + lk[g] == 0 ? 1 : 0; };
    auto b1 = [&](int g) { return kb + lk[g] + 1 == N ? 2 : 3; };
    T Sr[1][REG ? 3 * NP : 1];
    if constexpr (REG) {
        const T *Sk = S + (size_t)(kb + lk[0]) * blkS + ri[0];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const bool present = act[0] && b >= b0(0) && b < b1(0);
#pragma unroll
            for (int j = 0; j < NP; ++j)
                Sr[0][b * NP + j] = (present && (uint32_t)j < n) ? __ldg(Sk + (size_t)(b * n + j) * n) : T(0);
        }
    }
    auto matS = [&](int g) {
        if constexpr (REG) {
            T v[1] = {T(0)};
            if (act[0]) reg_matvec<T, NP, 3, 1>(Sr, vp + lk[0] * NP, v);
            return v[0];
        } else
        return act[g] ? grid_row<T, NP, 3>(S + (size_t)(kb + lk[g]) * blkS + ri[g], b0(g), b1(g), vp + lk[g] * NP, n) : T(0);
    };
    auto matP = [&](int g) {
        if (!act[g]) return T(0);
        if constexpr (PTRI)
            return grid_row<T, NP, 3>(P + (size_t)(kb + lk[g]) * blkP + ri[g], b0(g), b1(g), vr + lk[g] * NP, n);
        else return grid_row<T, NP, 1>(P + (size_t)(kb + lk[g]) * blkP + ri[g], 0, 1, vr + (lk[g] + 1) * NP, n);
    };
    // both neighbours get row values of the boundary knots
    uint32_t seq = 0;
    auto post = [&](int g, T v) {
        if (first(g)) grid_post_halo<T, NP>(gp, seq, C, rank - 1, 1, ri[g], v);
        if (last(g)) grid_post_halo<T, NP>(gp, seq, C, rank + 1, 0, ri[g], v);
    };
    // the copies of the neighbours' boundary knots: h(t) for t < 2 n
    auto halo_update = [&](T *win, const T *in, auto f) {
        for (uint32_t t = tid; t < 2 * n; t += nthr) {
            if (t < n && has_left) win[t] = f(win[t], in[t]);
            if (t >= n && has_right) {
                T *h = win + (nk + 1) * NP + (t - n);
                *h = f(*h, in[NP + t - n]);
            }
        }
    };
    __syncthreads();

    // ---- r = gamma - S lambda0   (include/pcg.cuh:119-126)
    T lam[G], r[G], p[G], z[G], y[G];
    A gg;
    bool alive;
    {
        if (lam0) {
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (act[g]) vp[(lk[g] + 1) * NP + ri[g]] = lam0[(size_t)(kb + lk[g]) * n + ri[g]];
            for (uint32_t t = tid; t < 2 * n; t += nthr) {
                if (t < n && has_left) vp[t] = lam0[(size_t)(kb - 1) * n + t];
                if (t >= n && has_right) vp[(nk + 1) * NP + (t - n)] = lam0[(size_t)ke * n + (t - n)];
            }
            __syncthreads();
        }
        A v1[1] = {A(0)};
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const size_t row = (size_t)(kb + lk[g]) * n + ri[g];
            const T gm = act[g] ? gamma[row] : T(0);
            lam[g] = (act[g] && lam0) ? lam0[row] : T(0);
            r[g] = (act[g] && lam0) ? gm - matS(g) : gm;
            acc_madd(v1[0], gm, gm);
            if (act[g]) vr[(lk[g] + 1) * NP + ri[g]] = r[g];
            if constexpr (PTRI) post(g, r[g]);
        }
        alive = grid_exchange<T, A, NP, PROBE, 1>(v1, part, out, gp, seq, C, rank, n, PTRI, vr, vr + (nk + 1) * NP,
                                                  [](int, A, GridOut<T, A> *, uint32_t) {});
        gg = v1[0];
    }
    // ---- z = Phi^-1 r; p = z; eta = r.z   (include/pcg.cuh:131-149)
    A eta = A(0);
    if (alive) {
        A v1[1] = {A(0)};
#pragma unroll
        for (int g = 0; g < G; ++g) {
            z[g] = matP(g);
            p[g] = z[g];
            if (act[g]) vp[(lk[g] + 1) * NP + ri[g]] = p[g];
            post(g, z[g]);
            acc_madd(v1[0], r[g], z[g]);
        }
        alive = grid_exchange<T, A, NP, PROBE, 1>(v1, part, out, gp, seq, C, rank, n, true, vp, vp + (nk + 1) * NP,
                                                  [](int, A, GridOut<T, A> *, uint32_t) {});
        eta = v1[0];
    }
    const A thr = A(d.tol * d.tol * (double)gg), tol = A(d.tol);

    // ---- main loop   (include/pcg.cuh:154-208)
    uint32_t iter = 0;
    int32_t status = alive ? ST_MAX_ITER : ST_TIMEOUT;
    A eta_new = A(0), rr = A(0);
    const uint32_t max_iter = alive ? d.max_iter : 0u;
    for (; iter < max_iter;) {
        uint32_t bad;
        {
            A v1[1] = {A(0)};
#pragma unroll
            for (int g = 0; g < G; ++g) {
                y[g] = matS(g);
                if constexpr (PTRI) post(g, y[g]);  // the neighbours' r halo
                acc_madd(v1[0], p[g], y[g]);
            }
            alive = grid_exchange<T, A, NP, PROBE, 1>(v1, part, out, gp, seq, C, rank, n, PTRI, uh, uh + NP,
                                                      [&](int, A s, GridOut<T, A> *o, uint32_t lane) {
                                                          const T a = (s == A(0)) ? T(0) : acc_ratio<T>(eta, s);
                                                          if (lane == 0) {
                                                              o->ratio = a;
                                                              o->code[0] = acc_finite(s) ? 0u : kNotFinite;
                                                          }
                                                      });
        }
        if (!alive) { status = ST_TIMEOUT; break; }
        const T alpha = out->ratio;
        bad = out->code[0];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            lam[g] = fma_rn(alpha, p[g], lam[g]);
            r[g] = fma_rn(-alpha, y[g], r[g]);
            if (act[g]) vr[(lk[g] + 1) * NP + ri[g]] = r[g];
        }
        if constexpr (PTRI) halo_update(vr, uh, [&](T h, T u) { return fma_rn(-alpha, u, h); });
        __syncthreads();
        {
            A v2[2] = {A(0), A(0)};
#pragma unroll
            for (int g = 0; g < G; ++g) {
                z[g] = matP(g);
                post(g, z[g]);
                acc_madd(v2[0], r[g], z[g]);
                if (relres) acc_madd(v2[1], r[g], r[g]);
            }
            alive = grid_exchange<T, A, NP, PROBE, 2>(v2, part, out, gp, seq, C, rank, n, true, zh, zh + NP,
                                                      [&](int q, A s, GridOut<T, A> *o, uint32_t lane) {
                                                          if (q == 0) {
                                                              const T b = acc_ratio<T>(s, eta);
                                                              if (lane == 0) {
                                                                  o->ratio = b;
                                                                  o->code[0] = (acc_finite(s) ? 0u : kNotFinite) |
                                                                               (acc_abs(s) < tol ? kExitTest : 0u);
                                                              }
                                                          } else if (lane == 0) {
                                                              o->code[1] = s <= thr ? kExitTest : 0u;
                                                          }
                                                      });
            eta_new = v2[0];
            rr = v2[1];
        }
        ++iter;
        const T beta = out->ratio;
        bad |= out->code[0] & kNotFinite;
        if (!alive) { status = ST_TIMEOUT; break; }
        if (bad) { status = ST_BREAKDOWN; break; }
        if (out->code[relres ? 1 : 0] & kExitTest) { status = ST_CONVERGED; break; }
        eta = eta_new;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            p[g] = fma_rn(beta, p[g], z[g]);
            if (act[g]) vp[(lk[g] + 1) * NP + ri[g]] = p[g];
        }
        halo_update(vp, zh, [&](T h, T zz) { return fma_rn(beta, h, zz); });
        __syncthreads();
    }

    // ---- outputs   (include/pcg.cuh:212-217)
    T *lam_out = static_cast<T *>(d.lambda);
#pragma unroll
    for (int g = 0; g < G; ++g)
        if (act[g]) lam_out[(size_t)(kb + lk[g]) * n + ri[g]] = lam[g];
    if (rank == 0 && tid == 0) {
        SysResult res;
        res.iters = iter;
        res.status = status;
        res.eta = (double)eta_new;
        res.rr = relres ? (double)rr : -1.0;
        res.gg = (double)gg;
        res.outer = 0;
        res.pad = 0;
        *gp.result = res;
    }
}

}  // namespace gbdpcg
