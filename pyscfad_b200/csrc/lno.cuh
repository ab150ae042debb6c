// LNO (T): the triples energy with a projector on the first occupied index,
//   E = (1/3) sum_{ijk, abc} Wt[ijk,abc] Q[ijk,abc],
//   Wt[i..] = sum_l mat[l,i] WW[l..],   Q = r3(WW + VV/2) / D,
// the energy of lnoccsdt_contract (pyscfadlib/pyscfadlib/vjp/cc/lno_ccsd_t.c:6-29
// with the job weights of lno_ccsd_t.c:73-94 and the 2/3 of
// pyscfad/lno/ccsd_t.py:111; mat = identity gives the canonical E(T)), and
// its adjoint (lnoccsdt_energy_vjp, lno_ccsd_t_vjp.c:74-122 and 400-566).
//
// WW and Q are symmetric under simultaneous permutations of the occupied and
// virtual indices, so one box of virtuals (a in A, b in B, c in C) with all
// occupied triples (i, j, k) holds everything of a chunk; what the projector
// breaks is restored by projecting each of the three occupied slots:
//   E    = g sum_box PW Q,  PW = sum over slots of the projected WW,
//   PQ   = sum over slots of the transposed projector on Q,
//   Zbar = f PW / D,  Dbar = -(g ybar / f) Zbar Q,  WWbar = f PQ + r3(Zbar),
//   VVbar = r3(Zbar) / 2,
//   mat_bar[l,i] = g ybar sum over slots of sum WW[..l..] Q[..i..]
// with f = 2 ybar / 3 and g = (distinct orderings of the blocks A, B, C) / 9.  Every
// raw amplitude of an ordering of the blocks is one box position permuted, and
// its adjoint is that position's WWbar (VVbar); with equal blocks the box holds
// each value once per permutation, hence g.
//
// Three kernels over FP64 arrays [i][j][k][e] of the box (e: 512 slots per
// triple of 8-wide sub-ranges, in the thread order of the orbit kernels; l0 l1 l2
// slots, row-major, where a sub-range is short):
//   k_lno_fwd   an occupied representative and a sub-range triple per CTA: six
//               orderings of two elements per thread, WW and Q of the six
//               occupied orders out as whole lines
//   k_lno_proj  one occupied slot, streaming over columns: three products on the
//               FP64 tensor cores; the slots add up over three launches, the last
//               one forms Zbar
//   k_lno_adj   as k_lno_fwd: r3, Wbar and V-term gradients (FP64 sums) written
//               back over the leading regions, orbital-energy gradients
// and k_lno_fwd_e, k_lno_adj_e with a thread per element for the chunks of short
// sub-ranges.
// Bytes per raw amplitude: 4 or 8 + 16/6, 128/6, 24/6 + 4 or 8: a third of what
// the four passes over arrays of all orderings took (104 and 120), which were
// bound by shared-memory gathers and memory latency.  Measured, nocc 14 nvir 96
// mixed, forward / projection / adjoint (+ V gradients): 42.9 / 44.0 / 49.4 + 29.4 ms
// to 11.6 / 20.6 / 18.0; nocc 9 nvir 45 FP64: 4.7 / 2.2 / 4.5 + 2.7 to 1.2 / 2.6 / 1.4 ms.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "f2.cuh"
#include "f2e.cuh"
#include "f2m.cuh"
#include "gemm_fp64.cuh"

namespace tb {

constexpr int kLnoMaxO = 64;    // largest nocc of the LNO path (projection tiles)
constexpr int kLnoThreads = kF2Threads;

struct LnoArgs {
    int o, v;
    int nsub;                   // sub-range triples of the box (all of them)
    int kn, ne;                 // log2 of the slots of one, slots of an occupied triple (even)
    F2mSub sub[kF2mMaxSub];     // pat: equal blocks; regions as in the canonical epilogue
    int n_ijk;
    const int *ijk;             // occupied representatives i >= j >= k
    const void *S;              // raw w of the chunk (blocked staging, FP64 or FP32)
    double *WW, *Q, *PW, *PQ;   // box arrays; PW becomes Zbar
    const double *mat, *mo_e, *t1, *t2, *ovov, *fvo;
    void *SW;                   // Wbar staging per ordering: FP64 [y][p][x][q][rzp], or
                                // 16-bit hi/lo planes (rows or 8 x 8 tiles, wbar_tiled) at 2 swoff
    const double *wscale;       // power-of-two scale of the fp16 split
    double *mat_bar, *mo_bar, *t1_bar, *t2_bar, *ovov_bar, *fvo_bar;
    double ybar, f, g;
    int want_grad;
    double *part;               // energy partials, one per block and slot
};

// ---------------------------------------------------------------------------
// orbit kernels: two elements (a, b, c), (a + 4, b, c) per thread, as in f2.cuh
// ---------------------------------------------------------------------------
// box index of ordering s at slot e: the occupied index paired with virtual slot c is ijk[t] with s[t] = c
template <int S>
__device__ __forceinline__ long long lno_box(int o, long long ne, int i0, int i1, int i2) {
    int ps[3] = {0, 0, 0}, inv[3] = {0, 0, 0};
    perm_of(S, ps);
    inv[ps[0]] = 0;
    inv[ps[1]] = 1;
    inv[ps[2]] = 2;
    const int ids[3] = {i0, i1, i2};
    return (((long long)ids[inv[0]] * o + ids[inv[1]]) * o + ids[inv[2]]) * ne;
}

template <typename F>
__device__ __forceinline__ void lno_for_s(F &&f) {
    f(std::integral_constant<int, 0>{});
    f(std::integral_constant<int, 1>{});
    f(std::integral_constant<int, 2>{});
    f(std::integral_constant<int, 3>{});
    f(std::integral_constant<int, 4>{});
    f(std::integral_constant<int, 5>{});
}

template <typename StageT>
__global__ void __launch_bounds__(kLnoThreads, 2) k_lno_fwd(const __grid_constant__ LnoArgs A) {
    extern __shared__ __align__(16) uint8_t lno_raw[];
    double2 *tab = reinterpret_cast<double2 *>(lno_raw), *tf = tab + 36 * 64;
    const int o = A.o;
    // sub-range triple fastest: the CTAs of one representative run together
    const int rep = blockIdx.x / A.nsub, sub = blockIdx.x - rep * A.nsub;
    const F2mSub &R = A.sub[sub];
    const int i0 = A.ijk[3 * rep], i1 = A.ijk[3 * rep + 1], i2 = A.ijk[3 * rep + 2];
    int ca, cb, cc;
    f2_element(threadIdx.x, ca, cb, cc);
    f2_load_tables(A, R, i0, i1, i2, tab, tf);
    double WW[2][6], VV[2][6];
    f2_amplitudes(reinterpret_cast<const StageT *>(A.S), R, o, i0, i1, i2, ca, cb, cc, true, true, tab, tf, WW, VV);
    const double *ev = A.mo_e + o;
    const double e_occ = A.mo_e[i0] + A.mo_e[i1] + A.mo_e[i2];
    const double e_bc = ev[R.st[1] + cb] + ev[R.st[2] + cc];
    const long long ne = A.ne;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        double X[6], Z[6];
#pragma unroll
        for (int s = 0; s < 6; s++) X[s] = WW[e][s] + 0.5 * VV[e][s];
        f2_r3(X, Z);
        const double rD = 1.0 / (e_occ - ev[R.st[0] + ca + 4 * e] - e_bc);
        const int slot = sub * 512 + e * 256 + threadIdx.x;
        lno_for_s([&](auto sc) {
            constexpr int s = decltype(sc)::value;
            const long long at = lno_box<s>(o, ne, i0, i1, i2) + slot;
            A.WW[at] = WW[e][s];
            A.Q[at] = Z[s] * rD;
        });
    }
}

// k_lno_fwd of a chunk with a short sub-range: a thread per element (f2e.cuh)
template <typename StageT>
__global__ void __launch_bounds__(kElemThreads, 2) k_lno_fwd_e(const __grid_constant__ LnoArgs A) {
    const int o = A.o;
    const Elem E = elem_of(A, blockIdx.x * kElemThreads + threadIdx.x);
    const F2mSub &R = A.sub[E.sub];
    const int ids[3] = {A.ijk[3 * E.rep], A.ijk[3 * E.rep + 1], A.ijk[3 * E.rep + 2]};
    double WW[6], VV[6], X[6], Z[6];
    elem_amplitudes<StageT>(A, R, ids, E.loc, WW, VV);
#pragma unroll
    for (int s = 0; s < 6; s++) X[s] = WW[s] + 0.5 * VV[s];
    f2_r3(X, Z);
    const double *ev = A.mo_e + o;
    const double rD = 1.0 / (A.mo_e[ids[0]] + A.mo_e[ids[1]] + A.mo_e[ids[2]] - ev[R.st[0] + E.loc[0]] -
                             ev[R.st[1] + E.loc[1]] - ev[R.st[2] + E.loc[2]]);
    if (!E.ok) return;
    const int slot = (E.sub << A.kn) + E.el;
    lno_for_s([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        const long long at = lno_box<s>(o, A.ne, ids[0], ids[1], ids[2]) + slot;
        A.WW[at] = WW[s];
        A.Q[at] = Z[s] * rD;
        if (A.ne > A.nsub << A.kn && slot == 0) A.WW[at + 1] = A.Q[at + 1] = 0.0;   // a single element: the unused slot
    });
}

// ---------------------------------------------------------------------------
// projection of one occupied slot (0, 1, 2), streaming over columns
// ---------------------------------------------------------------------------
// Rows: all o values of the slot, a row stride apart; columns: the other two
// occupied indices and e, COLS at a time (consecutive e).  Per tile
//   PW[i] = sum_l mat[l,i] WW[l],  PQ[l] = sum_i mat[l,i] Q[i],  Gram += WW Q^T
// and at the end energy = <mat, Gram> (= sum PW Q)
// on the FP64 tensor cores (per 8x8 output tile a thread holds D[g][2t],
// D[g][2t+1], A[g][t] and B[t][g] of each k-step, g = lane / 4, t = lane % 4).
// FIRST: PW and PQ are stored, else added to; slot 0 runs last and forms Zbar
// and f PQ.  Streams WW, Q and the running sums: HBM; wide tiles at small o and the
// running sums loaded before the tile's copies are waited for keep enough bytes
// in flight.  The running sums are the accumulators, and a warp's fragments serve
// all its rows and columns.  Up to four Gram tiles are shared by the eight warps
// by columns, in two chains each; the shares are added in shared memory, since
// every CTA adds its o x o sums to mat_bar and those atomics all meet on o^2
// addresses (added there share by share the kernel took twice as long; the grid
// is what is resident for the same reason).  Nocc 14 nvir 96: 20.7 to 17.3 ms of
// a call against a tile at a time, energies from PW and a Gram tile per warp.
template <int COLS>
struct LnoProj {
    static constexpr int LD = COLS + 4;   // conflict-free fragment loads
    static constexpr int MAXO = 2048 / COLS;                      // 16, 32, 64
    static constexpr int NG = (MAXO / 8) * (MAXO / 8);            // Gram tiles
    static constexpr int GW = NG < kLnoThreads / 32 ? 1 : NG / (kLnoThreads / 32);   // Gram tiles per warp
    // output tiles per warp: IT of 8 rows (every one, or every second), JT of 8 columns
    static constexpr int JT = COLS >= 64 ? COLS / 64 : 1, IT = COLS >= 64 ? MAXO / 8 : MAXO / 16;
    static constexpr int TW = IT * JT;
    static size_t smem(int o) {
        const int rows = (o + 7) / 8 * 8;
        return (size_t)(4 * rows * LD + o * o + kLnoMaxO + 2 * COLS) * sizeof(double);
    }
};

// FULL: three full sub-ranges, 512 slots a triple: a tile of columns is consecutive (the general form, with
// a division per thread and column, took 2 % more of a call at nocc 14 nvir 96, 6 % of this kernel at
// nocc 49 nvir 24).
template <int COLS, bool FULL>
__global__ void __launch_bounds__(kLnoThreads, 2) k_lno_proj(const __grid_constant__ LnoArgs A, int slot, int first) {
    using C = LnoProj<COLS>;
    constexpr int LD = C::LD;
    extern __shared__ __align__(16) uint8_t lno_raw[];
    const int o = A.o, o4 = (o + 3) & ~3, o8 = (o + 7) / 8, rows = 8 * o8;
    double *sw_b = reinterpret_cast<double *>(lno_raw), *sq_b = sw_b + 2 * rows * LD, *sM = sq_b + 2 * rows * LD;
    double *s_eo = sM + o * o, *s_ecol_b = s_eo + kLnoMaxO;
    __shared__ double red[kLnoThreads / 32];
    // columns: the other two occupied indices and e, `ncol` of them; the first `run` are consecutive, and
    // so on from o run on
    const int ne = A.ne, ncol = o * o * ne, ntile = (ncol + COLS - 1) / COLS;
    const int run = slot == 0 ? ncol : (slot == 1 ? o * ne : ne);
    const long long rstride = run;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int fg = lane >> 2, ft = lane & 3;
    const bool grad = A.want_grad != 0, last = slot == 0;
    const double gy = A.g * A.ybar;
    for (int k = threadIdx.x; k < o * o; k += blockDim.x) sM[k] = A.mat[k];
    for (int k = threadIdx.x; k < o; k += blockDim.x) s_eo[k] = A.mo_e[k];
    const int ngram = o8 * o8;
    // few Gram tiles: the warps share them by columns
    const int nks = ngram == 1 ? 8 : ngram <= 4 ? 2 : 1, ks = nks > 1 ? warp / ngram : 0;
    const int gram0 = nks > 1 ? (warp < ngram * nks ? warp % ngram : ngram) : warp;
    const int gc0 = ks * (COLS / nks), gc1 = gc0 + COLS / nks;
    double acc[C::GW][2], alt[C::GW][2];   // two chains
#pragma unroll
    for (int k = 0; k < C::GW; k++) acc[k][0] = acc[k][1] = alt[k][0] = alt[k][1] = 0.0;
    // this warp's output tile k = m JT + j: rows and columns
    auto row0 = [&](int m) -> int { return (COLS >= 64 ? m : (warp >> 2) + 2 * m) * 8; };
    auto col0 = [&](int j) -> int { return (COLS >= 64 ? warp + 8 * j : warp & 3) * 8; };
    // column c of row 0
    auto column = [&](int c) -> long long { return c + (long long)(c / run) * run * (o - 1); };
    auto issue = [&](int t, int b) {
        double *sw = sw_b + b * rows * LD, *sq = sq_b + b * rows * LD;
        auto copy = [&](int l, int j, long long at, int bytes) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(sw + l * LD + j)), "l"(A.WW + at), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(sq + l * LD + j)), "l"(A.Q + at), "r"(bytes) : "memory");
        };
        if constexpr (FULL) {
            const long long base = column(t * COLS);
            for (int e = threadIdx.x; e < rows * (COLS / 2); e += blockDim.x) {
                const int l = e / (COLS / 2), j = e % (COLS / 2) * 2;
                copy(l, j, base + (l < o ? l * rstride + j : 0), l < o ? 16 : 0);
            }
        } else {
            const int j = threadIdx.x % (COLS / 2) * 2;   // (this thread's columns in every turn)
            const bool in = t * COLS + j < ncol;
            const long long base = in ? column(t * COLS + j) : 0;
            for (int l = threadIdx.x / (COLS / 2); l < rows; l += kLnoThreads / (COLS / 2)) {
                const bool ok = in && l < o;
                copy(l, j, base + (ok ? l * rstride : 0), ok ? 16 : 0);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (grad && last && threadIdx.x < COLS) {
            // energies of the column: the other two occupied indices, a, b and c
            const int col = t * COLS + threadIdx.x, oth = col / ne, e = col - oth * ne, sub = e >> A.kn;
            double ec = -1e30;   // an unused slot: any non-zero value
            if (col < ncol && sub < A.nsub) {
                const F2mSub &R = A.sub[sub];
                const int pos = e & ((1 << A.kn) - 1);
                int a, b2, c;
                if (FULL) {   // the orbit kernels' order, else row-major
                    f2_element(pos & 255, a, b2, c);
                    a += 4 * (pos >> 8);
                } else {
                    c = pos % R.len[2];
                    b2 = pos / R.len[2] % R.len[1];
                    a = pos / (R.len[2] * R.len[1]);
                }
                const double *ev = A.mo_e + o;
                ec = A.mo_e[oth / o] + A.mo_e[oth % o] - ev[R.st[0] + a] - ev[R.st[1] + b2] - ev[R.st[2] + c];
            }
            s_ecol_b[b * COLS + threadIdx.x] = ec;
        }
    };
    int buf = 0;
    if ((int)blockIdx.x < ntile) issue(blockIdx.x, 0);
    for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
        if (t + (int)gridDim.x < ntile) issue(t + gridDim.x, buf ^ 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");   // keeps the wait count uniform
        const long long tile0 = FULL ? column(t * COLS) : 0;
        long long colat[C::JT];   // this thread's output columns (negative: beyond the last)
        if constexpr (!FULL) {
#pragma unroll
            for (int j = 0; j < C::JT; j++) {
                const int c = t * COLS + col0(j) + 2 * ft;
                colat[j] = c < ncol ? column(c) : -1;
            }
        }
        auto output = [&](int i, int j) -> long long { return (FULL ? tile0 + col0(j) + 2 * ft : colat[j]) + i * rstride; };
        double2 pw[C::TW], pq[C::TW];   // running sums of this thread's output positions
#pragma unroll
        for (int k = 0; k < C::TW; k++) {
            const int i = row0(k / C::JT) + fg;
            pw[k] = pq[k] = double2{0.0, 0.0};
            if (grad && !first && i < o && (FULL || colat[k % C::JT] >= 0)) {
                const long long at = output(i, k % C::JT);
                pw[k] = *reinterpret_cast<const double2 *>(A.PW + at);
                pq[k] = *reinterpret_cast<const double2 *>(A.PQ + at);
            }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const double *sw = sw_b + buf * rows * LD, *sq = sq_b + buf * rows * LD;
        const double *s_ecol = s_ecol_b + buf * COLS;
        if (grad) {
#pragma unroll 1
            for (int k0 = 0; k0 < o4; k0 += 4) {
                const int l = k0 + ft;
                double bw[C::JT], bq[C::JT];
#pragma unroll
                for (int j = 0; j < C::JT; j++) {
                    bw[j] = sw[l * LD + col0(j) + fg];
                    bq[j] = sq[l * LD + col0(j) + fg];
                }
#pragma unroll
                for (int m = 0; m < C::IT; m++) {
                    if (row0(m) >= o) continue;
                    const int i = row0(m) + fg;
                    const bool in = i < o && l < o;
                    const double aw = in ? sM[l * o + i] : 0.0, aq = in ? sM[i * o + l] : 0.0;
#pragma unroll
                    for (int j = 0; j < C::JT; j++) {
                        dmma_884(pw[m * C::JT + j].x, pw[m * C::JT + j].y, aw, bw[j]);
                        dmma_884(pq[m * C::JT + j].x, pq[m * C::JT + j].y, aq, bq[j]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < C::TW; k++) {
                const int i = row0(k / C::JT) + fg, cl = col0(k % C::JT) + 2 * ft;
                if (i < o && (FULL || colat[k % C::JT] >= 0)) {
                    const long long at = output(i, k % C::JT);
                    double2 w = pw[k], r = pq[k];
                    if (last) {
                        w.x = A.f * w.x / (s_eo[i] + s_ecol[cl]);
                        w.y = A.f * w.y / (s_eo[i] + s_ecol[cl + 1]);
                        r.x *= A.f;
                        r.y *= A.f;
                    }
                    *reinterpret_cast<double2 *>(A.PW + at) = w;
                    *reinterpret_cast<double2 *>(A.PQ + at) = r;
                }
            }
        }
        // Gram[l, i] += sum_c WW[l, c] Q[i, c]
#pragma unroll
        for (int k = 0; k < C::GW; k++) {
            const int gt = gram0 + k * (kLnoThreads / 32);
            if (gt < ngram) {
                const double *gw = sw + (gt / o8 * 8 + fg) * LD + ft, *gq = sq + (gt % o8 * 8 + fg) * LD + ft;
#pragma unroll 4
                for (int c = gc0; c < gc1; c += 8) {
                    dmma_884(acc[k][0], acc[k][1], gw[c], gq[c]);
                    dmma_884(alt[k][0], alt[k][1], gw[c + 4], gq[c + 4]);
                }
            }
        }
        __syncthreads();   // buffer buf is refilled two tiles from now
        buf ^= 1;
    }
    // The energy is <mat, Gram>.  Shares of a Gram tile are added in shared memory: the blocks
    // of all SMs meet on the o^2 addresses of mat_bar.
    double *share = reinterpret_cast<double *>(lno_raw);   // (the loop's last barrier is behind)
    if (nks > 1) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
    }
    double en = 0.0;
#pragma unroll
    for (int k = 0; k < C::GW; k++) {
        const int gt = gram0 + k * (kLnoThreads / 32);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            acc[k][h] += alt[k][h];
            const int l = gt / o8 * 8 + fg, i = gt % o8 * 8 + 2 * ft + h;
            if (gt < ngram && l < o && i < o) en += sM[l * o + i] * acc[k][h];
            if (nks > 1) share[(warp * 32 + lane) * 2 + h] = acc[k][h];
        }
    }
    for (int off = 16; off > 0; off >>= 1) en += __shfl_xor_sync(0xffffffffu, en, off);
    if (lane == 0) red[warp] = en;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kLnoThreads / 32; w++) s += red[w];
        A.part[slot * gridDim.x + blockIdx.x] = A.g * s;
    }
    if (!grad || ks > 0) return;
#pragma unroll
    for (int k = 0; k < C::GW; k++) {
        const int gt = gram0 + k * (kLnoThreads / 32);
        if (gt < ngram) {
            const int l = gt / o8 * 8 + fg;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int i = gt % o8 * 8 + 2 * ft + h;
                double gv = acc[k][h];
                for (int w = 1; w < nks; w++) gv += share[((warp + w * ngram) * 32 + lane) * 2 + h];
                if (l < o && i < o && gv != 0.0) red_add(&A.mat_bar[l * o + i], gy * gv);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// adjoint of the raw amplitudes, V-term and orbital-energy gradients
// ---------------------------------------------------------------------------
// SPLIT 0: FP64 Wbar; 1: fp16 hi/lo of wbar * wscale (exact power of two); 2: bf16
// hi/lo, unscaled -- the operand formats of the adjoint contractions.
template <int SPLIT>
__global__ void __launch_bounds__(kLnoThreads, 2) k_lno_adj(const __grid_constant__ LnoArgs A) {
    using WT = typename F2Smem<SPLIT>::W;
    extern __shared__ __align__(16) uint8_t lno_raw[];
    double2 *tab = reinterpret_cast<double2 *>(lno_raw), *tf = tab + 36 * 64;
    double *sV = reinterpret_cast<double *>(lno_raw + F2Smem<SPLIT>::TABLES);
    WT *sW = reinterpret_cast<WT *>(sV + 6 * 512);
    __shared__ int s_res[3][8];
    __shared__ double s_part[8][12];
    const int o = A.o, tid = threadIdx.x;
    const int rep = blockIdx.x / A.nsub, sub = blockIdx.x - rep * A.nsub;
    const F2mSub &R = A.sub[sub];
    const int i0 = A.ijk[3 * rep], i1 = A.ijk[3 * rep + 1], i2 = A.ijk[3 * rep + 2];
    const int opat = (i0 == i2) ? 3 : (i0 == i1 ? 1 : (i1 == i2 ? 2 : 0));
    const int vpat = R.pat;
    if (tid < 24) s_res[tid >> 3][tid & 7] = f2m_res(tid >> 3, tid & 7);
    int ca, cb, cc;
    f2_element(tid, ca, cb, cc);
    const int gidx = f2m_res(0, ca) ^ f2m_res(1, cb) ^ f2m_res(2, cc);
    const long long ne = A.ne;
    const float wsc = SPLIT == 1 ? (float)*A.wscale : 1.0f;
    // Dbar = -(g ybar / f) Zbar Q, each occupied order once
    const double dfac = -(A.g * A.ybar / A.f) / (opat == 0 ? 1.0 : (opat == 3 ? 6.0 : 2.0));
    double dd[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int slot = sub * 512 + e * 256 + tid;
        double Z[6], P[6], X[6];
        double ds = 0.0;
        lno_for_s([&](auto sc) {
            constexpr int s = decltype(sc)::value;
            const long long at = lno_box<s>(o, ne, i0, i1, i2) + slot;
            Z[s] = __ldg(&A.PW[at]);
            P[s] = __ldg(&A.PQ[at]);
            ds += Z[s] * __ldg(&A.Q[at]);
        });
        dd[e] = A.f != 0.0 ? dfac * ds : 0.0;
        f2_r3(Z, X);
        const int g = e == 0 ? gidx : gidx ^ 4;
#pragma unroll
        for (int s = 0; s < 6; s++) {
            const double wb = P[s] + X[s];
            sV[s * 512 + g] = 0.5 * X[s];
            if constexpr (SPLIT == 0) sW[s * 512 + g] = wb;
            else sW[s * 512 + g] = f2m_split<SPLIT>((float)wb, wsc);
        }
    }
    f2_load_tables(A, R, i0, i1, i2, tab, tf);
    f2_dd_partials(dd, s_part);
    __syncthreads();
    f2_dd_add(s_part, R, o, i0, i1, i2, A.mo_bar);
    f2_writeback<SPLIT>(A, R, i0, i1, i2, opat, vpat, tab, tf, s_res, sW, sV);
}

// k_lno_adj of a chunk with a short sub-range: a thread per element
template <int SPLIT>
__global__ void __launch_bounds__(kElemThreads, 2) k_lno_adj_e(const __grid_constant__ LnoArgs A) {
    using WT = typename F2Smem<SPLIT>::W;
    __shared__ double sV[6 * kElemThreads];
    __shared__ WT sW[6 * kElemThreads];
    const int o = A.o;
    const Elem E = elem_of(A, blockIdx.x * kElemThreads + threadIdx.x);
    const F2mSub &R = A.sub[E.sub];
    const int ids[3] = {A.ijk[3 * E.rep], A.ijk[3 * E.rep + 1], A.ijk[3 * E.rep + 2]};
    const int opat = (ids[0] == ids[2]) ? 3 : (ids[0] == ids[1] ? 1 : (ids[1] == ids[2] ? 2 : 0));
    const float wsc = SPLIT == 1 ? (float)*A.wscale : 1.0f;
    const double dfac = -(A.g * A.ybar / A.f) / (opat == 0 ? 1.0 : (opat == 3 ? 6.0 : 2.0));
    const int slot = (E.sub << A.kn) + E.el;
    double Z[6], P[6], X[6], ds = 0.0;
    lno_for_s([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        const long long at = lno_box<s>(o, A.ne, ids[0], ids[1], ids[2]) + slot;
        Z[s] = __ldg(&A.PW[at]);
        P[s] = __ldg(&A.PQ[at]);
        ds += Z[s] * __ldg(&A.Q[at]);
    });
    f2_r3(Z, X);
#pragma unroll
    for (int s = 0; s < 6; s++) {
        const double wb = P[s] + X[s];
        sV[s * kElemThreads + threadIdx.x] = 0.5 * X[s];
        if constexpr (SPLIT == 0) sW[s * kElemThreads + threadIdx.x] = wb;
        else sW[s * kElemThreads + threadIdx.x] = f2m_split<SPLIT>((float)wb, wsc);
    }
    elem_dd(A, R, E, ids, E.ok && A.f != 0.0 ? dfac * ds : 0.0);
    elem_writeback<SPLIT>(A, R, E, ids, opat, R.pat, sW, sV);
}

// ---------------------------------------------------------------------------
// orbit bookkeeping of 4-wide sub-ranges as host tables (triples_lno_tables; no
// kernel reads them): candidate region c = 6 pi + rho holds occupied triple
// (ijk[pi0], ijk[pi1], ijk[pi2]) over the virtual sub-ranges (U[rho0], U[rho1], U[rho2])
// ---------------------------------------------------------------------------
constexpr int kLnoSB = 4;
constexpr int kLnoRegion = kLnoSB * kLnoSB * kLnoSB;
__host__ __device__ constexpr int lno_pad(int slot) { return slot + 3 * (slot >> 4); }

struct alignas(16) LnoTables {
    unsigned char symsl[6][kLnoRegion];      // 16-byte multiples first
    unsigned char r3sl[2][6][kLnoRegion];
    unsigned char symc[36][6];
    unsigned char r3c[2][36][6];
};
inline void lno_build_tables(LnoTables &t) {
    static const int r3p[6][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}, {0, 2, 1}, {1, 0, 2}};
    for (int cc = 0; cc < 36; cc++)
        for (int s = 0; s < 6; s++) {
            int pp[3], pr[3], ps[3], m[3];
            perm_of(cc / 6, pp);
            perm_of(cc % 6, pr);
            perm_of(s, ps);
            t.symc[cc][s] = (unsigned char)(6 * perm_index(pp[ps[0]], pp[ps[1]]) + perm_index(pr[ps[0]], pr[ps[1]]));
            for (int k = 0; k < 3; k++) m[r3p[s][k]] = k;
            t.r3c[0][cc][s] = (unsigned char)(6 * (cc / 6) + perm_index(pr[m[0]], pr[m[1]]));
            for (int k = 0; k < 3; k++) m[k] = r3p[s][k];
            t.r3c[1][cc][s] = (unsigned char)(6 * (cc / 6) + perm_index(pr[m[0]], pr[m[1]]));
        }
    for (int s = 0; s < 6; s++)
        for (int sl = 0; sl < kLnoRegion; sl++) {
            const int l[3] = {sl / (kLnoSB * kLnoSB), (sl / kLnoSB) % kLnoSB, sl % kLnoSB};
            int ps[3], m[3];
            perm_of(s, ps);
            t.symsl[s][sl] = (unsigned char)lno_pad((l[ps[0]] * kLnoSB + l[ps[1]]) * kLnoSB + l[ps[2]]);
            for (int k = 0; k < 3; k++) m[r3p[s][k]] = k;
            t.r3sl[0][s][sl] = (unsigned char)lno_pad((l[m[0]] * kLnoSB + l[m[1]]) * kLnoSB + l[m[2]]);
            for (int k = 0; k < 3; k++) m[k] = r3p[s][k];
            t.r3sl[1][s][sl] = (unsigned char)lno_pad((l[m[0]] * kLnoSB + l[m[1]]) * kLnoSB + l[m[2]]);
        }
}

struct LnoPattern {
    unsigned char nslab;
    unsigned char cand[36];
    unsigned char prim[36];
};
inline void lno_build_patterns(LnoPattern pats[16]) {
    for (int pid = 0; pid < 16; pid++) {
        const int eo01 = (pid >> 3) & 1, eo12 = (pid >> 2) & 1, ev01 = (pid >> 1) & 1, ev12 = pid & 1;
        int occ[3] = {2, 1, 0}, vr[3] = {2, 1, 0};
        if (eo12) occ[1] = occ[2];
        if (eo01) occ[0] = occ[1];
        if (ev12) vr[1] = vr[2];
        if (ev01) vr[0] = vr[1];
        int key[36][6], first[36];
        for (int c = 0; c < 36; c++) {
            int pp[3], pr[3];
            perm_of(c / 6, pp);
            perm_of(c % 6, pr);
            for (int k = 0; k < 3; k++) {
                key[c][k] = occ[pp[k]];
                key[c][3 + k] = vr[pr[k]];
            }
            first[c] = c;
            for (int c2 = 0; c2 < c; c2++) {
                bool same = true;
                for (int k = 0; k < 6; k++) same = same && key[c2][k] == key[c][k];
                if (same) {
                    first[c] = c2;
                    break;
                }
            }
        }
        LnoPattern &P = pats[pid];
        int n = 0, prim[36];
        for (int c = 0; c < 36; c++)
            if (first[c] == c) {
                prim[c] = n;
                P.cand[n++] = (unsigned char)c;
            }
        for (int c = n; c < 36; c++) P.cand[c] = 0;
        for (int c = 0; c < 36; c++) P.prim[c] = (unsigned char)prim[first[c]];
        P.nslab = (unsigned char)n;
    }
}

}  // namespace tb
