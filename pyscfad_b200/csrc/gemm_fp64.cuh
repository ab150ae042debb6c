// FP64 GEMM tile with multi-index operand maps.  This is the "plain FP64
// GPU form" of the (T) contractions: the same chunked algorithm as the
// mixed-precision path, computed on the FP64 tensor cores
// (mma.sync.m8n8k4.f64: per 8x8 output tile a thread holds D[g][2t..2t+1],
// and A[g][t], B[t][g] of each k-step, g = lane / 4, t = lane % 4).
//
//   C(m,n) (+)= alpha * [ sum_k A(m,k) B(n,k) + alpha2 * sum_k A2(m,k) B2(n,k) ]
//   A(m,k) = A.p[apply(A.mn, m) + apply(A.k, k)], likewise B, A2, B2, C.
//
// BM x BN output tile, 256 threads, K tiles of 16 in a three-stage cp.async
// pipeline (8-byte copies, zero-filled past the edges: the operands' rows are
// only 8-byte aligned).  KFA / KFB: the operand is contiguous along k, so its
// tile is copied along k and kept as [row][k], else along the rows and kept as
// [k][row]; both leading dimensions are 4 (mod 16) doubles, so the fragment
// loads of a half-warp hit 16 distinct 8-byte banks.  The k part of every
// operand offset is tabulated in shared memory one barrier ahead of its use.
//
// What bounds it: the FP64 tensor pipe for the ovvv contractions (N = nvir),
// the stream of Wbar for the ooov ones (N = nocc).  The tile sizes are chosen
// on the host (gemm_tile in triples.cu) because M and N are nocc * 16, nvir
// and nocc: with one 128 x 128 tile the ooov kinds did 8 to 25 times the
// arithmetic they need.  Measured, nocc 12 nvir 100, E + VJP: W contraction 40.4
// to 19.6 ms, ovvv kinds 48.8 and 48.0 to 21.1 and 22.4 ms, ooov kinds 50.2 and
// 46.7 to 7.2 and 6.7 ms (the 128 x 128 x 8 register-staged tile before).
#pragma once
#include "common.cuh"

namespace tb {

struct GOp {
    const double *p;
    Map4 mn;
    Map4 k;
};

struct GemmArgs {
    int M, N, K, K2;
    GOp A, B, A2, B2;
    double *C;
    Map4 cm, cn;
    double alpha, alpha2;
    int atomic;   // 1: C += result as FP64 atomic adds (tiles or K slices that share outputs), 0: C = result
};

constexpr int kGBK = 16, kGStages = 3, kGThreads = 256;

// 8 warps as WM x WN; each warp owns (BM / WM) x (BN / WN) of the tile
template <int BM, int BN, bool KFA, bool KFB>
struct GemmCfg {
    static constexpr int WN = BN >= 128 ? 4 : (BN == 64 ? (BM == 64 ? 4 : 2) : 1);
    static constexpr int WM = 8 / WN;
    static constexpr int TM = BM / WM / 8, TN = BN / WN / 8;   // 8 x 8 MMA tiles per warp
    static_assert(TM >= 1 && TN >= 1 && TM * WM * 8 == BM && TN * WN * 8 == BN, "warps tile the block");
    static constexpr int LDA = KFA ? kGBK + 4 : BM + 4, LDB = KFB ? kGBK + 4 : BN + 4;
    static constexpr int ELA = KFA ? BM * LDA : kGBK * LDA, ELB = KFB ? BN * LDB : kGBK * LDB;
    static constexpr int RING = kGStages + 1;
    static constexpr size_t TAB = 3 * (BM + BN) + RING * 2 * kGBK;   // row, output and k offsets
    static constexpr size_t SMEM = sizeof(double) * (size_t)(kGStages * (ELA + ELB)) + sizeof(long long) * TAB;
};

__device__ __forceinline__ void dmma_884(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// 8-byte asynchronous copy global -> shared, zero-filled when !valid (nothing is read then)
__device__ __forceinline__ void gemm_cp8(double *dst, const double *src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 8 : 0)
                 : "memory");
}

// One operand's K tile: R rows x 16 k values.
template <int R, bool KF, int LD>
__device__ __forceinline__ void gemm_load_tile(const double *__restrict__ p, const long long *rows,
                                               const long long *koff, int tid, double *dst) {
#pragma unroll
    for (int i = 0; i < (R * kGBK + kGThreads - 1) / kGThreads; i++) {
        const int e = tid + kGThreads * i;
        if ((R * kGBK) % kGThreads != 0 && e >= R * kGBK) break;
        const int kl = KF ? e % kGBK : e / R, ml = KF ? e / kGBK : e % R;
        const long long ro = rows[ml], ko = koff[kl];
        const bool ok = (ro | ko) >= 0;
        gemm_cp8(dst + (KF ? ml * LD + kl : kl * LD + ml), ok ? p + ro + ko : p, ok);
    }
}

// Tile (m0, n0), K slice `slice` of `nslice` (slices need atomic; K2 > 0 only with one slice).
template <int BM, int BN, bool KFA, bool KFB>
__device__ __forceinline__ void gemm_fp64_tile(const GemmArgs &g, int m0, int n0, int slice, int nslice,
                                               double *smem) {
    using C = GemmCfg<BM, BN, KFA, KFB>;
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int fg = lane >> 2, ft = lane & 3;   // fragment row / k index
    const int wm0 = (warp / C::WN) * C::TM * 8, wn0 = (warp % C::WN) * C::TN * 8;
    double *sA = smem, *sB = smem + kGStages * C::ELA;
    long long *rowA = reinterpret_cast<long long *>(smem + kGStages * (C::ELA + C::ELB));
    long long *rowB = rowA + BM, *rowA2 = rowB + BN, *rowB2 = rowA2 + BM, *koff = rowB2 + BN;
    long long *outM = koff + C::RING * 2 * kGBK, *outN = outM + BM;
    for (int t = tid; t < BM; t += kGThreads) {
        const bool ok = m0 + t < g.M;
        rowA[t] = ok ? apply(g.A.mn, m0 + t) : -1;
        rowA2[t] = (ok && g.K2 > 0) ? apply(g.A2.mn, m0 + t) : -1;
    }
    for (int t = tid; t < BN; t += kGThreads) {
        const bool ok = n0 + t < g.N;
        rowB[t] = ok ? apply(g.B.mn, n0 + t) : -1;
        rowB2[t] = (ok && g.K2 > 0) ? apply(g.B2.mn, n0 + t) : -1;
    }

    // K tiles: the second product first (its sum is scaled by alpha2 before the first product is added)
    const int kt2 = (g.K2 + kGBK - 1) / kGBK, kt_all = kt2 + (g.K + kGBK - 1) / kGBK;
    const int per = (kt_all + nslice - 1) / nslice;
    const int ktb = slice * per, kte = min(kt_all, ktb + per);
    if (ktb >= kte && g.atomic) return;   // an empty slice adds nothing

    auto tab_koff = [&](int kt) {
        if (tid < 2 * kGBK && kt < kte) {
            const int which = tid / kGBK, kl = tid % kGBK;
            const bool second = kt < kt2;
            const int k = (second ? kt : kt - kt2) * kGBK + kl;
            long long off = -1;
            if (k < (second ? g.K2 : g.K))
                off = which == 0 ? apply(second ? g.A2.k : g.A.k, k) : apply(second ? g.B2.k : g.B.k, k);
            koff[((kt % C::RING) * 2 + which) * kGBK + kl] = off;
        }
    };
    auto issue = [&](int kt) {
        if (kt < kte) {
            const bool second = kt < kt2;
            const int s = kt % kGStages;
            const long long *ko = koff + (kt % C::RING) * 2 * kGBK;
            gemm_load_tile<BM, KFA, C::LDA>(second ? g.A2.p : g.A.p, second ? rowA2 : rowA, ko, tid, sA + s * C::ELA);
            gemm_load_tile<BN, KFB, C::LDB>(second ? g.B2.p : g.B.p, second ? rowB2 : rowB, ko + kGBK, tid,
                                            sB + s * C::ELB);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    double acc[C::TM][C::TN][2];
#pragma unroll
    for (int i = 0; i < C::TM; i++)
#pragma unroll
        for (int j = 0; j < C::TN; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
    for (int s = 0; s < kGStages; s++) tab_koff(ktb + s);
    __syncthreads();
#pragma unroll
    for (int s = 0; s < kGStages - 1; s++) issue(ktb + s);
    // output offsets, while the first tiles arrive (read after the K loop's barriers)
    for (int t = tid; t < BM; t += kGThreads) outM[t] = apply(g.cm, m0 + t);
    for (int t = tid; t < BN; t += kGThreads) outN[t] = apply(g.cn, n0 + t);
    for (int kt = ktb; kt < kte; kt++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kGStages - 2) : "memory");
        __syncthreads();   // tile kt is complete, the buffer of tile kt - 1 is free
        issue(kt + kGStages - 1);
        tab_koff(kt + kGStages);
        if (kt == kt2 && kt2 > 0) {
#pragma unroll
            for (int i = 0; i < C::TM; i++)
#pragma unroll
                for (int j = 0; j < C::TN; j++) {
                    acc[i][j][0] *= g.alpha2;
                    acc[i][j][1] *= g.alpha2;
                }
        }
        const double *As = sA + (kt % kGStages) * C::ELA, *Bs = sB + (kt % kGStages) * C::ELB;
#pragma unroll
        for (int ks = 0; ks < kGBK; ks += 4) {
            double a[C::TM], b[C::TN];
#pragma unroll
            for (int i = 0; i < C::TM; i++)
                a[i] = KFA ? As[(wm0 + 8 * i + fg) * C::LDA + ks + ft] : As[(ks + ft) * C::LDA + wm0 + 8 * i + fg];
#pragma unroll
            for (int j = 0; j < C::TN; j++)
                b[j] = KFB ? Bs[(wn0 + 8 * j + fg) * C::LDB + ks + ft] : Bs[(ks + ft) * C::LDB + wn0 + 8 * j + fg];
#pragma unroll
            for (int i = 0; i < C::TM; i++)
#pragma unroll
                for (int j = 0; j < C::TN; j++) dmma_884(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

#pragma unroll
    for (int i = 0; i < C::TM; i++) {
        const int ml = wm0 + 8 * i + fg;
        if (m0 + ml >= g.M) continue;
        double *row = g.C + outM[ml];
#pragma unroll
        for (int j = 0; j < C::TN; j++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int nl = wn0 + 8 * j + 2 * ft + c;
                if (n0 + nl >= g.N) continue;
                const double val = g.alpha * acc[i][j][c];
                if (g.atomic) red_add(row + outN[nl], val);
                else row[outN[nl]] = val;
            }
    }
}

}  // namespace tb
