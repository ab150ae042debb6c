// Element kernels: the epilogue of chunks whose sub-ranges are short (a
// remainder block, or blocks of 4 and less): the LNO calls, and the canonical ones
// that by_element (triples.cu) names, the mixed modes' among them.
//
// A short item has 1 to 256 elements a, b, c where the orbit kernels (f2.cuh) give
// every item a CTA with the tables and slots of 512.  Here a thread takes one
// element of one item, items lie one behind the other (l0 l1 l2 consecutive
// threads, c fastest), and everything is gathered straight from memory: the
// entries of an item are a few lines that its lanes meet in L1.  Sums over one of
// the three coordinates are butterflies over the lane bits that hold it; a
// coordinate that reaches into the next warp leaves a partial sum per warp.  Each
// thread keeps its six results of W and V in its own shared-memory column, which
// lets the loop over the regions run rolled.
// What bounds it: latency and issue of the gathers (126 loads per element).
// Measured against the orbit kernels and 512-slot boxes for every item, LNO E + VJP in
// FP64: nocc 64 nvir 3 57.5 to 2.3 ms, nocc 49 nvir 17 (16 + 1) 122 to 81, nocc 49 nvir 31
// 612 to 352, nocc 9 nvir 45 10.8 to 10.1 ms; FP64 energy: nocc 64 nvir 3 6.7 to 0.46 ms,
// nocc 160 nvir 9 324 to 94, nocc 32 nvir 17 4.4 to 3.2; FP64 E + VJP nocc 257 nvir 3 608 to 141 ms.
#pragma once
#include "common.cuh"
#include "f2.cuh"

namespace tb {

constexpr int kElemThreads = 256;

// The element of this thread.
struct Elem {
    int rep, sub, loc[3];   // item, coordinates
    int el, warps;          // slot in the item (row-major a, b, c), warps that share the item
    unsigned m[3], all;     // lane bits of each coordinate, of the item
    bool ok;                // false: beyond the last item
};

template <typename ARGS>
__device__ __forceinline__ Elem elem_of(const ARGS &A, int g) {
    const F2mSub &R = A.sub[0];   // the sub-ranges of a chunk have the same lengths
    const int k2 = 31 - __clz(R.len[2]), k1 = 31 - __clz(R.len[1]), k0 = 31 - __clz(R.len[0]), kn = k0 + k1 + k2;
    Elem E;
    const int item = g >> kn;
    E.el = g & ((1 << kn) - 1);
    E.rep = item / A.nsub;
    E.sub = item - E.rep * A.nsub;
    E.ok = E.rep < A.n_ijk;
    if (!E.ok) E.rep = A.n_ijk - 1;
    E.loc[2] = E.el & (R.len[2] - 1);
    E.loc[1] = (E.el >> k2) & (R.len[1] - 1);
    E.loc[0] = E.el >> (k1 + k2);
    E.warps = kn > 5 ? 1 << (kn - 5) : 1;
    E.m[2] = (unsigned)(R.len[2] - 1) & 31u;
    E.m[1] = ((unsigned)(R.len[1] - 1) << k2) & 31u;
    E.m[0] = ((unsigned)(R.len[0] - 1) << (k1 + k2)) & 31u;
    E.all = E.m[0] | E.m[1] | E.m[2];
    return E;
}

// Sum over the lanes that differ in the bits of `mask` (the same for all lanes).
__device__ __forceinline__ double elem_sum(double v, unsigned mask) {
#pragma unroll
    for (unsigned b = 1; b < 32; b <<= 1)
        if (mask & b) v += __shfl_xor_sync(0xffffffffu, v, b);
    return v;
}

// WW and VV of the element, six orderings each
template <typename StageT, typename ARGS>
__device__ __forceinline__ void elem_amplitudes(const ARGS &A, const F2mSub &R, const int (&ids)[3], const int (&loc)[3],
                                                double (&WW)[6], double (&VV)[6]) {
    const int o = A.o, v = A.v;
    const StageT *S[6];
#pragma unroll
    for (int pi = 0; pi < 6; pi++) {
        int pp[3] = {0, 0, 0};
        perm_of(pi, pp);
        const int x = loc[pp[0]], y = loc[pp[1]], z = loc[pp[2]], ex = R.len[pp[0]], ez = R.len[pp[2]];
        const int swz = sizeof(StageT) == 4 && ex == 8 && ez == 8 ? f2m_row_swizzle(y) : 0;
        S[pi] = static_cast<const StageT *>(A.S) + R.pi[pi].s0 + y * ex * ez + ((x * ez + z) ^ swz);
    }
    double tz[3][3], fz[3][3];   // t1[r, z], fvo[z, r]
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int s = 0; s < 3; s++) {
            const int z = R.st[s] + loc[s];
            tz[r][s] = __ldg(&A.t1[(long long)ids[r] * v + z]);
            fz[r][s] = __ldg(&A.fvo[(long long)z * o + ids[r]]);
        }
#pragma unroll
    for (int s = 0; s < 6; s++) WW[s] = VV[s] = 0.0;
#pragma unroll
    for (int rho = 0; rho < 6; rho++) {
        int pr[3] = {0, 0, 0};
        perm_of(rho, pr);
        const int p = ids[pr[0]], q = ids[pr[1]];
        const long long idx = ((long long)p * o + q) * o + ids[pr[2]];
#pragma unroll
        for (int pi = 0; pi < 6; pi++) {
            const int s = f2m_sof(pi, rho);
            int pp[3] = {0, 0, 0};
            perm_of(pi, pp);
            const int x = R.st[pp[0]] + loc[pp[0]], y = R.st[pp[1]] + loc[pp[1]];
            WW[s] += (double)__ldg(S[pi] + idx * R.pi[pi].rs);
            VV[s] += __ldg(&A.ovov[(((long long)p * v + x) * o + q) * v + y]) * tz[pr[2]][pp[2]] +
                     __ldg(&A.t2[(((long long)q * o + p) * v + y) * v + x]) * fz[pr[2]][pp[2]];
        }
    }
}

// Orbital-energy gradient of dd = dE/dD
template <typename ARGS>
__device__ __forceinline__ void elem_dd(const ARGS &A, const F2mSub &R, const Elem &E, const int (&ids)[3], double dd) {
    const int lane = threadIdx.x & 31;
    const double tot = elem_sum(dd, E.all);
    if (E.ok && (lane & E.all) == 0) {
#pragma unroll
        for (int k = 0; k < 3; k++) red_add(&A.mo_bar[ids[k]], tot);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const unsigned others = E.all & ~E.m[k];
        const double acc = elem_sum(dd, others);
        if (E.ok && (lane & others) == 0) red_add(&A.mo_bar[A.o + R.st[k] + E.loc[k]], -acc);
    }
}

// Write-back of the element's results, column threadIdx.x of sW and sV [6][kElemThreads]:
// Wbar, and the V-term gradients v = ovov[p,x,q,y] t1[r,z] + t2[q,p,y,x] fvo[z,r], over the leading
// regions (pi, rho).  Regions that share r and z share the column sums.
template <int SPLIT, typename ARGS>
__device__ __forceinline__ void elem_writeback(const ARGS &A, const F2mSub &R, const Elem &E, const int (&ids)[3], int opat,
                                               int vpat, const typename F2Smem<SPLIT>::W *sW, const double *sV) {
    const int o = A.o, v = A.v, lane = threadIdx.x & 31;
    const unsigned lead = opat == 0 ? 63u : opat == 1 ? 19u : opat == 2 ? 13u : 1u;    // orderings of f2m_lead
    const unsigned vlead = vpat == 0 ? 63u : vpat == 1 ? 19u : vpat == 2 ? 13u : 1u;
#pragma unroll 1
    for (int rz = 0; rz < 9; rz++) {
        const int rs = rz / 3, zs = rz % 3;   // slots of r and z
        const int zl = sel3(E.loc[0], E.loc[1], E.loc[2], zs), z = sel3(R.st[0], R.st[1], R.st[2], zs) + zl;
        const unsigned mz = zs == 0 ? E.m[0] : zs == 1 ? E.m[1] : E.m[2], others = E.all & ~mz;
        const int r = sel3(ids[0], ids[1], ids[2], rs);
        const double tv = __ldg(&A.t1[(long long)r * v + z]), fv = __ldg(&A.fvo[(long long)z * o + r]);
        double ct = 0.0, cf = 0.0;
#pragma unroll
        for (int u = 0; u < 4; u++) {   // (unrolled: the loads of four regions in flight)
            // the two other slots in either order: u & 1 for rho, u >> 1 for pi
            const int ra = rs == 0 ? 1 : 0, rb = rs == 2 ? 1 : 2, za = zs == 0 ? 1 : 0, zb = zs == 2 ? 1 : 2;
            const int pr0 = u & 1 ? rb : ra, pr1 = u & 1 ? ra : rb, pp0 = u >> 1 ? zb : za, pp1 = u >> 1 ? za : zb;
            const int rho = perm_index(pr0, pr1), pi = perm_index(pp0, pp1);
            const bool vl = (vlead >> pi) & 1u;
            if (!__any_sync(0xffffffffu, vl)) continue;
            const bool in = E.ok && vl && ((lead >> rho) & 1u);
            // s with s o rho = pi: its slots are the virtual ones paired with occupied slots 0 and 1
            const int s0 = pr0 == 0 ? pp0 : (pr1 == 0 ? pp1 : zs), s1 = pr0 == 1 ? pp0 : (pr1 == 1 ? pp1 : zs);
            const int at = perm_index(s0, s1) * kElemThreads + threadIdx.x;
            const int p = sel3(ids[0], ids[1], ids[2], pr0), q = sel3(ids[0], ids[1], ids[2], pr1);
            const int xl = sel3(E.loc[0], E.loc[1], E.loc[2], pp0), yl = sel3(E.loc[0], E.loc[1], E.loc[2], pp1);
            const int x = sel3(R.st[0], R.st[1], R.st[2], pp0) + xl, y = sel3(R.st[0], R.st[1], R.st[2], pp1) + yl;
            const long long ov = (((long long)p * v + x) * o + q) * v + y, tt = (((long long)q * o + p) * v + y) * v + x;
            const double vb = in ? sV[at] : 0.0;
            if (in) {
                const F2mPi &D = R.pi[pi];
                const long long w = f2m_wbar(D, p, q, r) + (long long)xl * D.wx + (long long)yl * D.wy + zl;
                if constexpr (SPLIT == 0) {
                    static_cast<double *>(A.SW)[w] = sW[at];
                } else {
                    const uint32_t pk = sW[at];
                    static_cast<uint16_t *>(A.SW)[w] = (uint16_t)pk;
                    static_cast<uint16_t *>(A.SW)[w + D.half] = (uint16_t)(pk >> 16);
                }
                ct += vb * __ldg(&A.ovov[ov]);
                cf += vb * __ldg(&A.t2[tt]);
            }
            const double r1 = elem_sum(vb * tv, mz), r2 = elem_sum(vb * fv, mz);
            if (in && (lane & mz) == 0) {
                red_add(&A.ovov_bar[ov], r1);
                red_add(&A.t2_bar[tt], r2);
            }
        }
        ct = elem_sum(ct, others);
        cf = elem_sum(cf, others);
        if (E.ok && (lane & others) == 0) {
            red_add(&A.t1_bar[(long long)r * v + z], ct);
            red_add(&A.fvo_bar[(long long)z * o + r], cf);
        }
    }
}

// The items of the jobs (chunks) of a launch, FP64; a job starts with a new CTA.
template <typename JOBS>
__global__ void __launch_bounds__(kElemThreads, 2) k_f2e(const __grid_constant__ JOBS J) {
    __shared__ double sV[6 * kElemThreads], sW[6 * kElemThreads];
    JobCursor jcur;
    int blk;
    const int jb = jcur.at(J, (int)blockIdx.x, blk);
    const F2P &A = J.job[JOBS::kOne ? 0 : jb];
    const Elem E = elem_of(A, blk * kElemThreads + threadIdx.x);
    const F2mSub &R = A.sub[E.sub];
    const int ids[3] = {A.ijk[3 * E.rep], A.ijk[3 * E.rep + 1], A.ijk[3 * E.rep + 2]};
    const int opat = (ids[0] == ids[2]) ? 3 : (ids[0] == ids[1] ? 1 : (ids[1] == ids[2] ? 2 : 0));
    const int vpat = R.pat, lane = threadIdx.x & 31;
    double WW[6], VV[6], X[6], Z[6], RW[6];
    elem_amplitudes<double>(A, R, ids, E.loc, WW, VV);
    // orbit weights as in k_f2t
    const double cocc = opat == 0 ? 2.0 : (opat == 3 ? 6.0 / 18.0 : 1.0);
    const double cen = vpat == 0 ? cocc : (vpat == 3 ? cocc / 6.0 : cocc * 0.5);
#pragma unroll
    for (int s = 0; s < 6; s++) X[s] = WW[s] + 0.5 * VV[s];
    f2_r3(X, Z);
    f2_r3(WW, RW);
    const double *ev = A.mo_e + A.o;
    const double rD = 1.0 / (A.mo_e[ids[0]] + A.mo_e[ids[1]] + A.mo_e[ids[2]] - ev[R.st[0] + E.loc[0]] -
                             ev[R.st[1] + E.loc[1]] - ev[R.st[2] + E.loc[2]]);
    double esum = 0.0;
#pragma unroll
    for (int s = 0; s < 6; s++) esum += WW[s] * Z[s];
    // one partial per item, or per warp of it
    const double en = elem_sum(E.ok ? cen * esum * rD : 0.0, E.all);
    if (E.ok && (lane & E.all) == 0) A.e_part[(long long)(E.sub * E.warps + (E.el >> 5)) * A.n_ijk + E.rep] = en;
    if (!A.want_grad) return;
    const double g0 = cocc * A.ybar * rD;
    double wb[6], vb[6], w3 = 0.0, v3 = 0.0;
#pragma unroll
    for (int s = 0; s < 6; s++) {
        wb[s] = g0 * (Z[s] + RW[s]);
        vb[s] = g0 * 0.5 * RW[s];
        w3 += wb[s];
        v3 += vb[s];
    }
    // equal occupied indices: the orderings that name the same raw amplitudes add up
#pragma unroll
    for (int s = 0; s < 6; s++) {
        const int s1 = perm_compose(s, 2), s2 = perm_compose(s, 1), at = s * kElemThreads + threadIdx.x;
        sW[at] = opat == 0 ? wb[s] : opat == 1 ? wb[s] + wb[s1] : opat == 2 ? wb[s] + wb[s2] : w3;
        sV[at] = opat == 0 ? vb[s] : opat == 1 ? vb[s] + vb[s1] : opat == 2 ? vb[s] + vb[s2] : v3;
    }
    elem_dd(A, R, E, ids, E.ok ? -cen * A.ybar * esum * rD * rD : 0.0);
    elem_writeback<0>(A, R, E, ids, opat, vpat, sW, sV);
}

// ---------------------------------------------------------------------------
// The mixed modes.  With the adjoint, items within a warp (at most 32 elements).  FP32 where k_f2m is, and the same
// FP32 operations in the same order, so that a chunk gives the same values in either kernel: V terms
// summed over rho, rows along z, columns over y + 4, then bit 0 of y, bits 2, 1 and 0 of x, bit 1 of y.
// (What k_f2m adds for coordinates beyond a short range are zeros.)
// ---------------------------------------------------------------------------
struct ElemBits {         // lane bit of bit `b` of coordinate t, 0 where the range is shorter
    int k[3], at[3];
    __device__ __forceinline__ unsigned operator()(int t, int b) const {
        return b < sel3(k[0], k[1], k[2], t) ? 1u << (sel3(at[0], at[1], at[2], t) + b) : 0u;
    }
};

// Column sum of vb * table over the item's (x, y), x and y in coordinates tx, ty
__device__ __forceinline__ float elem_column(float vb, float table, const ElemBits &bit, int tx, int ty) {
    float v = __fmul_rn(vb, table);
    const unsigned y2 = bit(ty, 2);
    if (y2) {   // (bits are the same for all lanes)
        const float low = __shfl_xor_sync(0xffffffffu, v, y2), both = fmaf(vb, table, low);
        const float other = __shfl_xor_sync(0xffffffffu, both, y2);
        v = threadIdx.x & y2 ? both : other;
    }
    const unsigned order[5] = {bit(ty, 0), bit(tx, 2), bit(tx, 1), bit(tx, 0), bit(ty, 1)};
#pragma unroll
    for (int i = 0; i < 5; i++)
        if (order[i]) v += __shfl_xor_sync(0xffffffffu, v, order[i]);
    return v;
}

template <int H, typename JOBS>
__global__ void __launch_bounds__(kElemThreads, 2) k_f2em(const __grid_constant__ JOBS J) {
    __shared__ float sV[6 * kElemThreads];
    __shared__ uint32_t sW[6 * kElemThreads];
    JobCursor jcur;
    int blk;
    const int jb = jcur.at(J, (int)blockIdx.x, blk);
    const F2P &A = J.job[JOBS::kOne ? 0 : jb];
    const Elem E = elem_of(A, blk * kElemThreads + threadIdx.x);
    const F2mSub &R = A.sub[E.sub];
    const int o = A.o, v = A.v, lane = threadIdx.x & 31;
    const int ids[3] = {A.ijk[3 * E.rep], A.ijk[3 * E.rep + 1], A.ijk[3 * E.rep + 2]};
    const int opat = (ids[0] == ids[2]) ? 3 : (ids[0] == ids[1] ? 1 : (ids[1] == ids[2] ? 2 : 0));
    const int vpat = R.pat;
    const float *S[6];
#pragma unroll
    for (int pi = 0; pi < 6; pi++) {
        int pp[3] = {0, 0, 0};
        perm_of(pi, pp);
        const int ex = R.len[pp[0]], ez = R.len[pp[2]], y = E.loc[pp[1]];
        const int swz = ex == 8 && ez == 8 ? f2m_row_swizzle(y) : 0;
        S[pi] = static_cast<const float *>(A.S) + R.pi[pi].s0 + y * ex * ez + ((E.loc[pp[0]] * ez + E.loc[pp[2]]) ^ swz);
    }
    float tz[3][3], fz[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int s = 0; s < 3; s++) {
            const int z = R.st[s] + E.loc[s];
            tz[r][s] = (float)__ldg(&A.t1[(long long)ids[r] * v + z]);
            fz[r][s] = (float)__ldg(&A.fvo[(long long)z * o + ids[r]]);
        }
    double WW[6], X[6], Z[6], RW[6];
    float VV[6];
#pragma unroll
    for (int s = 0; s < 6; s++) {
        WW[s] = 0.0;
        VV[s] = 0.f;
    }
#pragma unroll
    for (int rho = 0; rho < 6; rho++) {
        int pr[3] = {0, 0, 0};
        perm_of(rho, pr);
        const int p = ids[pr[0]], q = ids[pr[1]];
        const long long idx = ((long long)p * o + q) * o + ids[pr[2]];
#pragma unroll
        for (int pi = 0; pi < 6; pi++) {
            const int s = f2m_sof(pi, rho);
            int pp[3] = {0, 0, 0};
            perm_of(pi, pp);
            const int x = R.st[pp[0]] + E.loc[pp[0]], y = R.st[pp[1]] + E.loc[pp[1]];
            WW[s] += (double)__ldg(S[pi] + idx * R.pi[pi].rs);
            const float ov = (float)__ldg(&A.ovov[(((long long)p * v + x) * o + q) * v + y]);
            const float tt = (float)__ldg(&A.t2[(((long long)q * o + p) * v + y) * v + x]);
            VV[s] = __fadd_rn(VV[s], fmaf(ov, tz[pr[2]][pp[2]], __fmul_rn(tt, fz[pr[2]][pp[2]])));
        }
    }
    const double cocc = opat == 0 ? 2.0 : (opat == 3 ? 6.0 / 18.0 : 1.0);
    const double cen = vpat == 0 ? cocc : (vpat == 3 ? cocc / 6.0 : cocc * 0.5);
#pragma unroll
    for (int s = 0; s < 6; s++) X[s] = WW[s] + 0.5 * (double)VV[s];
    f2_r3(X, Z);
    f2_r3(WW, RW);
    const double *ev = A.mo_e + o;
    const double rD = 1.0 / (A.mo_e[ids[0]] + A.mo_e[ids[1]] + A.mo_e[ids[2]] - ev[R.st[0] + E.loc[0]] -
                             ev[R.st[1] + E.loc[1]] - ev[R.st[2] + E.loc[2]]);
    double esum = 0.0;
#pragma unroll
    for (int s = 0; s < 6; s++) esum += WW[s] * Z[s];
    const double en = elem_sum(E.ok ? cen * esum * rD : 0.0, E.all);
    if (E.ok && (lane & E.all) == 0) A.e_part[(long long)(E.sub * E.warps + (E.el >> 5)) * A.n_ijk + E.rep] = en;
    if (!A.want_grad) return;
    const float wsc = (float)*A.wscale;
    const double g0 = cocc * A.ybar * rD;
    float wb[6], vb[6];
    double w3 = 0.0, v3 = 0.0;
#pragma unroll
    for (int s = 0; s < 6; s++) {
        wb[s] = (float)(g0 * (Z[s] + RW[s]));
        vb[s] = (float)(g0 * 0.5 * RW[s]);
        w3 += (double)wb[s];
        v3 += (double)vb[s];
    }
#pragma unroll
    for (int s = 0; s < 6; s++) {
        const int s1 = perm_compose(s, 2), s2 = perm_compose(s, 1), at = s * kElemThreads + threadIdx.x;
        const float w = opat == 0 ? wb[s] : opat == 1 ? wb[s] + wb[s1] : opat == 2 ? wb[s] + wb[s2] : (float)w3;
        sV[at] = opat == 0 ? vb[s] : opat == 1 ? vb[s] + vb[s1] : opat == 2 ? vb[s] + vb[s2] : (float)v3;
        sW[at] = f2m_split<H>(w, wsc);
    }
    elem_dd(A, R, E, ids, E.ok ? -cen * A.ybar * esum * rD * rD : 0.0);
    // write-back as in elem_writeback
    ElemBits bit;
#pragma unroll
    for (int t = 0; t < 3; t++) bit.k[t] = 31 - __clz(R.len[t]);
    bit.at[2] = 0;
    bit.at[1] = bit.k[2];
    bit.at[0] = bit.k[2] + bit.k[1];
    const unsigned lead = opat == 0 ? 63u : opat == 1 ? 19u : opat == 2 ? 13u : 1u;
    const unsigned vlead = vpat == 0 ? 63u : vpat == 1 ? 19u : vpat == 2 ? 13u : 1u;
#pragma unroll 1
    for (int rz = 0; rz < 9; rz++) {
        const int rs = rz / 3, zs = rz % 3;
        const int zl = sel3(E.loc[0], E.loc[1], E.loc[2], zs), z = sel3(R.st[0], R.st[1], R.st[2], zs) + zl;
        const unsigned mz = zs == 0 ? E.m[0] : zs == 1 ? E.m[1] : E.m[2], others = E.all & ~mz;
        const int r = sel3(ids[0], ids[1], ids[2], rs), lz = sel3(R.len[0], R.len[1], R.len[2], zs);
        const int zat = sel3(bit.at[0], bit.at[1], bit.at[2], zs);
        const float tv = (float)__ldg(&A.t1[(long long)r * v + z]), fv = (float)__ldg(&A.fvo[(long long)z * o + r]);
        double ct = 0.0, cf = 0.0;
#pragma unroll 1
        for (int u = 0; u < 4; u++) {
            const int ra = rs == 0 ? 1 : 0, rb = rs == 2 ? 1 : 2, za = zs == 0 ? 1 : 0, zb = zs == 2 ? 1 : 2;
            const int pr0 = u & 1 ? rb : ra, pr1 = u & 1 ? ra : rb, pp0 = u >> 1 ? zb : za, pp1 = u >> 1 ? za : zb;
            const int rho = perm_index(pr0, pr1), pi = perm_index(pp0, pp1);
            const bool vl = (vlead >> pi) & 1u;
            if (!__any_sync(0xffffffffu, vl)) continue;
            const bool in = E.ok && vl && ((lead >> rho) & 1u);
            const int s0 = pr0 == 0 ? pp0 : (pr1 == 0 ? pp1 : zs), s1 = pr0 == 1 ? pp0 : (pr1 == 1 ? pp1 : zs);
            const int at = perm_index(s0, s1) * kElemThreads + threadIdx.x;
            const int p = sel3(ids[0], ids[1], ids[2], pr0), q = sel3(ids[0], ids[1], ids[2], pr1);
            const int xl = sel3(E.loc[0], E.loc[1], E.loc[2], pp0), yl = sel3(E.loc[0], E.loc[1], E.loc[2], pp1);
            const int x = sel3(R.st[0], R.st[1], R.st[2], pp0) + xl, y = sel3(R.st[0], R.st[1], R.st[2], pp1) + yl;
            const long long ov = (((long long)p * v + x) * o + q) * v + y, tt = (((long long)q * o + p) * v + y) * v + x;
            const float vbe = in ? sV[at] : 0.f;
            float ox = 0.f, oy = 0.f;
            if (in) {
                const F2mPi &D = R.pi[pi];
                const long long w = f2m_wbar(D, p, q, r) + (long long)xl * D.wx + (long long)yl * D.wy + zl;
                const uint32_t pk = sW[at];
                static_cast<uint16_t *>(A.SW)[w] = (uint16_t)pk;
                static_cast<uint16_t *>(A.SW)[w + D.half] = (uint16_t)(pk >> 16);
                ox = (float)__ldg(&A.ovov[ov]);
                oy = (float)__ldg(&A.t2[tt]);
            }
            float r1 = 0.f, r2 = 0.f;
#pragma unroll 1
            for (int c = 0; c < lz; c++) {   // along z
                const int src = (int)(lane & ~mz) | (c << zat);
                const float vc = __shfl_sync(0xffffffffu, vbe, src);
                r1 = fmaf(vc, __shfl_sync(0xffffffffu, tv, src), r1);
                r2 = fmaf(vc, __shfl_sync(0xffffffffu, fv, src), r2);
            }
            if (in && (lane & mz) == 0) {
                red_add(&A.ovov_bar[ov], (double)r1);
                red_add(&A.t2_bar[tt], (double)r2);
            }
            ct += (double)elem_column(vbe, ox, bit, pp0, pp1);
            cf += (double)elem_column(vbe, oy, bit, pp0, pp1);
        }
        if (E.ok && (lane & others) == 0) {
            red_add(&A.t1_bar[(long long)r * v + z], ct);
            red_add(&A.fvo_bar[(long long)z * o + r], cf);
        }
    }
}

}  // namespace tb
