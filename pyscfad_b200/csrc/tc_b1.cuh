// Tensor-core (tcgen05) form of the adjoint contractions, one launch per kind for
// every ordering tau of the chunks of a group.  Wbar_tau is staged by the epilogue as fp16/bf16
// hi/lo splits (scaled by a per-chunk power of two), as rows
// [h][y][p][x][q][r][z] or, for x blocks of 8 and 16, as 8 x 8 tiles of (x, rz)
// (wbar_tiled); either serves all four products through TMA boxes, 128B-swizzled
// rows or unswizzled core matrices.  The MMA thread forms a step's descriptors
// by one addition each: field by field, it held up the MN-major kinds (8 % at
// nocc 40 nvir 72).
//
//   kind 0  ovvv:  G_A1[y][p][x][f] += sum_{q,rz} Wbar[y][p][x][q][rz] B1[q][rz][f]
//                  rows (p,x) K-major, batch y, K = (q, rz)
//   kind 1  t2:    G_B1[q][rz][f]   += sum_{y,p,x} Wbar[y][p][x][q][rz] A1[y][p][x][f]
//                  rows rz MN-major, batch q, K = (y, p, x)
//   kind 2  ovoo:  G_A2[q][p][x][m] -= sum_{y,rz} Wbar[y][p][x][q][rz] B2[y][rz][m]
//                  rows (p,x) K-major, batch q, K = (y, rz)
//   kind 3  t2:    G_B2[y][rz][m]   += sum_{q,p,x} Wbar[y][p][x][q][rz] A2n[q][p][x][m]
//                  rows rz MN-major, batch y, K = (q, p, x)   (A2n = -ovoo)
//
// (the adjoint GEMMs of get_eris_amps_bar, ccsd_t_vjp.c:139-246, batched over
// all occupied indices).  The second operand is always MN-major.  Products:
// hi*hi + hi*lo + lo*hi into FP32 TMEM; the epilogue adds the descaled tile
// into the FP64 gradient buffer.
#pragma once
#include "common.cuh"
#include "tc_f1.cuh"
#include "tc_ptx.cuh"

namespace tb {

// One launch covers one kind for ALL orderings tau of a chunk (tiles numbered
// ordering by ordering), so small per-ordering tile counts do not leave SMs
// idle.  Orderings that share an X (or Z) block write the same gradient rows,
// hence the FP64 atomic adds in the epilogue.
struct TcB1Params {
    CUtensorMap tmA[6];     // per ordering: Wbar_tau (first operand)
    CUtensorMap tmB[6];     // per ordering: second operand
    Dims d;
    PermBlock pb[6];
    int nperm;
    int kind;
    int nbatch[6], ntile_m[6], ntile_n;
    int nw, ncol;           // columns of an N tile (multiple of 16, at most BN), of the gradient rows
    int nk_outer[6], nk_inner[6];
    int cum[7];             // prefix of tile counts over orderings
    double *G;
    const double *wscale;   // device: per-chunk Wbar scale
    const double *oscale;   // device: scale of the second operand
    double sign;
    int *err;
    int bf16;
    int kseg;               // K blocks per TMEM accumulation segment
};

constexpr int kB1Threads = 320;   // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
// K segments summed in FP32 before the run goes into the FP64 gradient: runs of
// K <= 512 * 64 keep the rounding of the sum well below the fp16 split error
constexpr int kB1RunSegments = 512;

// N tiles are nw = 16 n columns wide: nvir (kinds 0, 1) or nocc (2, 3) rounded up
// to 16, or BN and a narrower last tile (nvir 180: 128 + 64; two of 96 took a
// 64-column load more per K block: ovvv and t2 kinds 197 to 183 ms at nocc 20).
// K blocks issue only the 16-wide steps that hold values.
template <bool A_MN, int BN>
struct TcB1Cfg {
    static constexpr int A_BYTES = kTcBM * kTcBK * 2;
    static constexpr int B_BYTES = BN * kTcBK * 2;
    static constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;
    static constexpr int STAGES = (200 * 1024) / STAGE_BYTES;
    // A 128 x 8 block of zeros: second K half of an 8-wide x block.
    static constexpr int ZERO_BYTES = A_MN ? 2048 : 0;
    // Barriers in the first 1024 bytes.  With the 1 KB that a block has reserved this stays within a
    // shared memory of 196 KB: a few hundred bytes more take the next size, 228 KB, and leave
    // 28 KB of L1 instead of 60 (the adjoint contractions of batched jobs then ran 1.25x as long).
    static constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + ZERO_BYTES;
    static_assert(SMEM + 1024 <= 196 * 1024, "one shared memory size up");
    static constexpr int NACC = 4;   // TMEM accumulators: the epilogue sums them in pairs
    static constexpr int TMEM_COLS = NACC * BN < 32 ? 32 : NACC * BN;
    static_assert(NACC * BN <= 512, "TMEM holds 512 columns");
};

// The tiles of the jobs (chunks, one kind) of a launch.
template <bool A_MN, int BN, typename JOBS>
__global__ void __launch_bounds__(kB1Threads, 1) k_b1_tc(const __grid_constant__ JOBS J) {
    using C = TcB1Cfg<A_MN, BN>;
    constexpr bool ONE = JOBS::kOne;
    JobCursor jcur;
    const TcB1Params &Pfirst = J.job[0];
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    if ((smem_u32(smem_raw) & 1023u) != 0) {   // the swizzle's pattern counts from 1024 B boundaries
        if (threadIdx.x == 0) atomicOr(Pfirst.err, 128);
        return;
    }
    uint8_t *smem = smem_raw + 1024;
    uint8_t *zero = smem + C::STAGES * C::STAGE_BYTES;
    uint64_t *full = (uint64_t *)smem_raw;
    uint64_t *empty = full + C::STAGES;
    uint64_t *tfull = empty + C::STAGES;
    uint64_t *tempty = tfull + C::NACC;
    uint64_t *drain = tempty + C::NACC;
    uint32_t *tmem_slot = (uint32_t *)(drain + 1);
    int &s_abort = *(int *)(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t leader = lane == 0 ? 1u : 0u;   // issues for the producer and MMA warps
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < C::STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < C::NACC; a++) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], 8);
        }
        mbar_init(drain, 1);
        fence_mbar_init();
    }
    if (ONE && warp == 0 && lane == 0) {
        for (int t = 0; t < Pfirst.nperm; t++) {
            tma_prefetch_desc(&Pfirst.tmA[t]);
            tma_prefetch_desc(&Pfirst.tmB[t]);
        }
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    if (A_MN) {
        for (int e = threadIdx.x; e < C::ZERO_BYTES / 4; e += kB1Threads) reinterpret_cast<uint32_t *>(zero)[e] = 0u;
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    volatile int *abortp = &s_abort;
    const int total = J.start[J.n];
    // columns an MMA of N tile nt covers
    auto width = [&](const TcB1Params &P, int nt) -> int {
        const int left = P.ncol - nt * P.nw;
        return left < P.nw ? (left + 15) / 16 * 16 : P.nw;
    };
    // tile t of the chunk with parameters P -> ordering, batch, M tile, N tile
    auto decode = [&](const TcB1Params &P, int t, int &tau, int &b, int &mt, int &nt) {
        tau = 0;
        while (tau + 1 < P.nperm && t >= P.cum[tau + 1]) tau++;
        int rem = t - P.cum[tau];
        const int per_batch = P.ntile_m[tau] * P.ntile_n;
        b = rem / per_batch;
        rem %= per_batch;
        mt = rem / P.ntile_n;
        nt = rem % P.ntile_n;
        // the column tiles of a row block are neighbours; their order turns with every round of
        // the grid, or a CTA could meet the last, narrower one each time
        if (P.ntile_n > 1) nt = (nt + t / P.ntile_n / max((int)gridDim.x / P.ntile_n, 1)) % P.ntile_n;
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        int stage = 0;
        uint32_t phase = 0;
        uint32_t pend_phase[C::STAGES];
        bool pending[C::STAGES];
        for (int s = 0; s < C::STAGES; s++) pending[s] = false;
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
            int lt;
            const int jb = jcur.at(J, t, lt);
            const TcB1Params &P = J.job[ONE ? 0 : jb];
            int tau, b, mt, nt;
            decode(P, lt, tau, b, mt, nt);
            const PermBlock &pb = P.pb[tau];
            const int Ty = pb.Ty, lz = 31 - __clz(pb.Tz);
            const int nk_inner = P.nk_inner[tau], nk = P.nk_outer[tau] * nk_inner;
            const CUtensorMap *tmA = &P.tmA[tau], *tmB = &P.tmB[tau];
            const int nbox = (width(P, nt) + 63) / 64, n0 = nt * P.nw;
            // A_MN K blocks hold 4 p: half the rows where an x block is one tile wide
            const bool tiled = wbar_tiled(pb);
            const int nxb = pb.Tx >> 3, o = P.d.o;
            const int bx = A_MN ? pb.X0 : pb.Z0, y0 = pb.Y0;
            const uint32_t abytes = A_MN && tiled && nxb == 1 ? C::A_BYTES / 2 : C::A_BYTES;
            const uint32_t bytes = 2 * abytes + (uint32_t)(2 * nbox * 8192);
            // K = (ko, ki): kinds 0 and 3 run q in ko with batch y, kinds 1 and 2 y in ko with batch q
            const bool ko_q = P.kind == 0 || P.kind == 3;
            int ko = 0, ki = 0;
            for (int kb = 0; kb < nk; kb++) {
                if (!mbar_wait_warp(&empty[stage], phase ^ 1u, abortp)) {
                    ok = false;
                    break;
                }
                pending[stage] = false;
                mbar_expect_tx(leader, &full[stage], bytes);
                uint8_t *sA = smem + stage * C::STAGE_BYTES;
                uint8_t *sB = sA + 2 * C::A_BYTES;
                const int aq = ko_q ? ko : b, ay = ko_q ? b : ko;
                const int b3 = ko_q ? ko : y0 + ko;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint8_t *a = sA + h * C::A_BYTES;
                    uint8_t *bb = sB + h * C::B_BYTES;
                    if (tiled) {
                        const int hyq = (h * Ty + ay) * o + aq;
                        if (A_MN) tma_load_5d(leader, a, tmA, &full[stage], 0, mt * 16, ki * 4 * nxb, hyq, 0);
                        else tma_load_5d(leader, a, tmA, &full[stage], 0, ki * 8, mt * 16, hyq, 0);
                    } else if (A_MN) {
#pragma unroll
                        for (int j = 0; j < 2; j++)
                            tma_load_5d(leader, a + j * 8192, tmA, &full[stage], mt * 128 + j * 64, aq, 0, ki * 4, h * Ty + ay);
                    } else {
                        tma_load_5d(leader, a, tmA, &full[stage], ki * 64, aq, 0, mt * 8, h * Ty + ay);
                    }
                    const int b2 = A_MN ? ki * 4 : (ki * 64) >> lz;
                    tma_load_5d(leader, bb, tmB, &full[stage], n0, bx, b2, b3, h);
                    if (BN > 64 && nbox > 1) tma_load_5d(leader, bb + 8192, tmB, &full[stage], n0 + 64, bx, b2, b3, h);
                }
                if (++ki == nk_inner) {
                    ki = 0;
                    ko++;
                }
                pending[stage] = true;
                pend_phase[stage] = phase;
                if (++stage == C::STAGES) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
        if (!ok) {
            *abortp = 1;
            if (leader) atomicOr(Pfirst.err, 8);
            for (int s = 0; s < C::STAGES; s++)
                if (pending[s]) {
                    for (uint32_t i = 0; i < kSpinLimit && !mbar_try_wait(&full[s], pend_phase[s]); i++) {
                    }
                }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: one TMEM buffer per K segment ----------------
        int stage = 0;
        uint32_t phase = 0;
        int seg = 0;   // running segment counter (same sequence as the epilogue)
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
            int lt;
            const int jb = jcur.at(J, t, lt);
            const TcB1Params &P = J.job[ONE ? 0 : jb];
            int tau, b, mt, nt;
            decode(P, lt, tau, b, mt, nt);
            const uint32_t idesc = make_idesc_f16(kTcBM, width(P, nt), P.bf16 != 0, A_MN, true);
            const int nk = P.nk_outer[tau] * P.nk_inner[tau];
            // K values of the inner blocks of one outer index: o Tz, or 16 per p
            const int klen = A_MN ? 16 * P.d.o : P.d.o * P.pb[tau].Tz;
            int left = klen;   // K values from the current inner block on
            // First operand: 128B-swizzled rows, or core matrices.  An 8-wide x block is the first
            // half of each 16-wide K step and a block of zeros the second: there the K stride is
            // the distance to that block, which falls as the address rises.
            const bool tiled = wbar_tiled(P.pb[tau]), half_k = A_MN && tiled && P.pb[tau].Tx == 8;
            const uint64_t a_unit = half_k ? 1ull - (1ull << 16) : 1ull;   // descriptor per 16 bytes of address
            const uint64_t a_base = !tiled  ? make_sdesc_sw128(0, A_MN ? 8192 : 16, 1024)
                                    : !A_MN ? make_sdesc_none(0, 128, 1024)
                                            : make_sdesc_none(0, half_k ? smem_u32(zero) : 2048u, 128);
            const uint64_t a_step = (tiled ? (A_MN ? (half_k ? 128 : 256) : 16) : (A_MN ? 128 : 2)) * a_unit;
            for (int k0 = 0; k0 < nk && ok; k0 += P.kseg, seg++) {
                const int acc = seg % C::NACC;
                const uint32_t accph = (seg / C::NACC) & 1;
                if (!mbar_wait_warp(&tempty[acc], accph ^ 1u, abortp)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
                const int k1 = (k0 + P.kseg < nk) ? k0 + P.kseg : nk;
                for (int kb = k0; kb < k1; kb++) {
                    if (!mbar_wait_warp(&full[stage], phase, abortp)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sA = smem_u32(smem + stage * C::STAGE_BYTES), sB = sA + 2 * C::A_BYTES;
                    const uint64_t a_h = a_base + (sA >> 4) * a_unit, a_l = a_h + (C::A_BYTES >> 4) * a_unit;
                    const uint64_t b_h = make_sdesc_sw128(sB, 8192, 1024), b_l = b_h + (C::B_BYTES >> 4);
                    const int nks = left < kTcBK ? (left + 15) >> 4 : kTcBK / 16;
                    left = left <= kTcBK ? klen : left - kTcBK;
#pragma unroll
                    for (int ks = 0; ks < kTcBK / 16; ks++) {
                        if (ks >= nks) break;
                        const uint64_t dah = a_h + a_step * ks, dal = a_l + a_step * ks;
                        const uint64_t dbh = b_h + 128 * ks, dbl = b_l + 128 * ks;
                        umma_f16(leader, d_tmem, dah, dbh, idesc, (kb > k0 || ks > 0) ? 1u : 0u);
                        umma_f16(leader, d_tmem, dah, dbl, idesc, 1u);
                        umma_f16(leader, d_tmem, dal, dbh, idesc, 1u);
                    }
                    umma_commit(leader, &empty[stage]);
                    if (++stage == C::STAGES) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                umma_commit(leader, &tfull[acc]);
            }
        }
        if (!ok) {
            *abortp = 1;
            if (leader) atomicOr(Pfirst.err, 16);
        }
        umma_commit(leader, drain);
        for (uint32_t i = 0; i < kSpinLimit && !mbar_try_wait(drain, 0); i++) {
        }
    } else if (warp >= 2) {
        // ---------------- epilogue: G += sign * sum_seg D_seg / (wscale * oscale) ----------------
        constexpr int HC = BN / 2;            // most columns of an epilogue warp: groups of 8,
                                              // 2 c + half for c = 0, 1, ...
        const int quarter = warp & 3;         // TMEM lane quarter this warp may access
        const int half = (warp - 2) >> 2;     // which of the column groups
        const int row = quarter * 32 + lane;
        const double sc0 = ONE ? Pfirst.sign / ((*Pfirst.wscale) * (*Pfirst.oscale)) : 0.0;   // single chunk: read once
        int seg = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
            int lt;
            const int jb = jcur.at(J, t, lt);
            const TcB1Params &P = J.job[ONE ? 0 : jb];
            const int o = P.d.o, v = P.d.v, Kp = P.d.Kp;
            int tau, b, mt, nt;
            decode(P, lt, tau, b, mt, nt);
            const PermBlock &pb = P.pb[tau];
            const int Tz = pb.Tz;
            const int nk = P.nk_outer[tau] * P.nk_inner[tau];
            const double sc = ONE ? sc0 : P.sign / ((*P.wscale) * (*P.oscale));
            long long roff = -1;
            if (P.kind == 0 || P.kind == 2) {
                const int xw = pb.Tx == 8 ? 8 : 16;   // rows of a p in the tile
                const int p = mt * (kTcBM / xw) + row / xw, x = row % xw;
                if (p < o && x < pb.Tx) {
                    if (P.kind == 0)
                        roff = ((((long long)pb.Y0 + b) * o + p) * v + pb.X0 + x) * Kp;
                    else
                        roff = (((long long)b * o + p) * v + pb.X0 + x) * o;
                }
            } else {
                const int rz = mt * 128 + row;
                if (rz < o * Tz) {
                    const int r = rz / Tz, z = rz % Tz;
                    if (P.kind == 1)
                        roff = (((long long)b * o + r) * v + pb.Z0 + z) * Kp;
                    else
                        roff = ((((long long)pb.Y0 + b) * o + r) * v + pb.Z0 + z) * o;
                }
            }
            const int nwid = width(P, nt), c0 = nt * P.nw + half * 8;
            const int lim = min(P.ncol - nt * P.nw, nwid) - half * 8;   // this warp's columns: c0 + [0, lim)
            float acc[HC];
#pragma unroll
            for (int j = 0; j < HC; j++) acc[j] = 0.f;
            // G += sc * acc, then acc = 0: the FP64 sum of a run of at most
            // kB1RunSegments FP32-summed segments
            auto flush = [&]() {
                if (roff >= 0) {
                    double *g = P.G + roff + c0;
#pragma unroll
                    for (int j = 0; j < HC; j++) {
                        const int col = (j >> 3) * 16 + (j & 7);
                        if (col < lim) red_add(g + col, sc * (double)acc[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < HC; j++) acc[j] = 0.f;
            };
            // segments in pairs, added into the FP32 run sum; every kB1RunSegments
            // segments the run goes into G in FP64
            const int nseg = (nk + P.kseg - 1) / P.kseg;
            for (int s0 = 0; s0 < nseg; s0 += 2, seg += 2) {
                const bool two = s0 + 1 < nseg;
                const int accA = seg % C::NACC, accB = (seg + 1) % C::NACC;
                if (!mbar_wait(&tfull[accA], (uint32_t)((seg / C::NACC) & 1), abortp) ||
                    (two && !mbar_wait(&tfull[accB], (uint32_t)(((seg + 1) / C::NACC) & 1), abortp))) {
                    *abortp = 1;
                    atomicOr(Pfirst.err, 32);
                    ok = false;
                    break;
                }
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < HC / 8; c++) {
                    // (columns beyond the tile's width hold nothing and are never added to G)
                    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((2 * c + half) * 8);
                    uint32_t va[8], vb[8];
                    tmem_ld8(lane_base + (uint32_t)(accA * BN), va);
                    if (two) tmem_ld8(lane_base + (uint32_t)(accB * BN), vb);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float sum = two ? __uint_as_float(va[j]) + __uint_as_float(vb[j]) : __uint_as_float(va[j]);
                        acc[c * 8 + j] += sum;
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&tempty[accA]);
                    if (two) mbar_arrive(&tempty[accB]);
                }
                if (!two) seg -= 1;   // an odd tail used one accumulator
                if ((s0 + 2) % kB1RunSegments == 0 || s0 + 2 >= nseg) flush();
            }
            if (!ok) break;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

}  // namespace tb
