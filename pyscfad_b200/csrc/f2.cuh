// FP64 orbit kernels: the chunk epilogue of the FP64 mode (k_f2t) and what the
// LNO kernels (lno.cuh) share with it.  The work items, the region layout and
// the treatment of repeated indices are those of f2m.cuh; here everything is
// FP64, one CTA of 256 threads takes one item, and the raw amplitudes are
// gathered straight from the contiguous regions of the staging buffer (every
// sector of a region is read by the CTA, the permuted gathers meet it in L1):
// V-term tables and element results fill the shared memory of two CTAs per SM.
// What bounds it: latency of the gathers and tables at 16 warps per SM, then the
// FP64 column sums.  Measured at nocc 12 nvir 100, E + VJP: 33.8 to 18.5 ms (4-wide sub-ranges,
// 64 threads per CTA and staged regions before).
#pragma once
#include <type_traits>

#include "common.cuh"
#include "f2m.cuh"

namespace tb {

constexpr int kF2Threads = 256;

struct F2P {
    int o, v;
    int nsub, n_ijk;
    const int *ijk;
    const double *mo_e, *t1, *t2, *ovov, *fvo;
    const void *S;      // W per ordering tau, blocked staging (FP64 rows are not exchanged)
    void *SW;           // Wbar out, per tau at ch.pb[tau].swoff: [y][p][x][q][r][z]
    const double *wscale;   // power-of-two scale of the fp16 split (element kernel of the mixed modes)
    double ybar;
    int want_grad;
    double *e_part;     // energy partial of each item, at sub * n_ijk + rep
    double *mo_bar, *t1_bar, *fvo_bar, *ovov_bar, *t2_bar;
    F2mSub sub[kF2mMaxSub];
};

// Shared memory: V-term tables, element results V (FP64) and W (FP64, or the
// 16-bit halves of the LNO mixed modes).
template <int SPLIT>
struct F2Smem {
    using W = typename std::conditional<SPLIT == 0, double, uint32_t>::type;
    static constexpr size_t TABLES = (36 * 64 + 72) * sizeof(double2);
    static constexpr size_t BYTES = TABLES + 6 * 512 * (sizeof(double) + sizeof(W));
};

// Sum NV (power of two) per-lane values over aligned groups of G lanes
// (NV <= G <= 32, G a power of two); afterwards lane l holds the group total
// of value (l % NV).
template <int NV, int G, typename T>
__device__ __forceinline__ T group_reduce_scatter(T (&v)[NV], int lane) {
#pragma unroll
    for (int h = NV / 2; h >= 1; h /= 2) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const T send = up ? v[i] : v[i + h];
            const T keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    T r = v[0];
#pragma unroll
    for (int h = NV; h < G; h *= 2) r += __shfl_xor_sync(0xffffffffu, r, h);
    return r;
}

// element (a, b, c) of thread t; its second one is (a + 4, b, c).  A warp spans 2 x 4 x 4 of them
__device__ __forceinline__ void f2_element(int t, int &a, int &b, int &c) {
    a = ((t >> 4) & 1) | (((t >> 7) & 1) << 1);
    b = ((t >> 2) & 3) | (((t >> 6) & 1) << 2);
    c = (t & 3) | (((t >> 5) & 1) << 2);
}

// 64-entry table block of 16-byte entries: eight lanes of a gather hit eight banks
__device__ __forceinline__ int f2_tab(int x, int y) { return y * 8 + (x ^ ((y & 1) << 2) ^ (y & 2)); }

// FP64 V-term tables of an item: {ovov[p,x,q,y], t2[q,p,y,x]} per (rho, pi), {t1[r,z], fvo[z,r]}
template <typename ARGS>
__device__ __forceinline__ void f2_load_tables(const ARGS &A, const F2mSub &R, int i0, int i1, int i2, double2 *tab,
                                               double2 *tf) {
    const int o = A.o, v = A.v;
    double *ts = reinterpret_cast<double *>(tab);
#pragma unroll 3
    for (int e = threadIdx.x; e < 36 * 64; e += kF2Threads) {
        const int blk = e >> 6, hi = (e >> 3) & 7, lo = e & 7;
        int pr[3], pp[3];
        perm_of(blk / 6, pr);
        perm_of(blk % 6, pp);
        const int p = sel3(i0, i1, i2, pr[0]), q = sel3(i0, i1, i2, pr[1]);
        const int lx = sel3(R.len[0], R.len[1], R.len[2], pp[0]), ly = sel3(R.len[0], R.len[1], R.len[2], pp[1]);
        const int sx = sel3(R.st[0], R.st[1], R.st[2], pp[0]), sy = sel3(R.st[0], R.st[1], R.st[2], pp[1]);
        // the fast index of each factor in turn runs over the lanes
        ts[2 * (blk * 64 + f2_tab(hi, lo))] =
            hi < lx && lo < ly ? __ldg(&A.ovov[(((long long)p * v + sx + hi) * o + q) * v + sy + lo]) : 0.0;
        ts[2 * (blk * 64 + f2_tab(lo, hi)) + 1] =
            lo < lx && hi < ly ? __ldg(&A.t2[(((long long)q * o + p) * v + sy + hi) * v + sx + lo]) : 0.0;
    }
    for (int e = threadIdx.x; e < 72; e += kF2Threads) {
        const int r = sel3(i0, i1, i2, e / 24), s = (e >> 3) % 3, zl = e & 7;
        const int z = sel3(R.st[0], R.st[1], R.st[2], s) + zl;
        const bool in = zl < sel3(R.len[0], R.len[1], R.len[2], s);
        tf[e] = in ? make_double2(__ldg(&A.t1[(long long)r * v + z]), __ldg(&A.fvo[(long long)z * o + r]))
                   : make_double2(0.0, 0.0);
    }
}

__device__ __forceinline__ void f2_r3(const double (&x)[6], double (&z)[6]) {
#pragma unroll
    for (int s = 0; s < 6; s++)
        z[s] = 4.0 * x[s] + x[perm_compose(s, 4)] + x[perm_compose(s, 3)] -
               2.0 * (x[perm_compose(s, 5)] + x[perm_compose(s, 1)] + x[perm_compose(s, 2)]);
}

// WW and VV of the thread's two elements, six orderings each: orbit sums over
// the regions of the item (StageT staging: FP32 rows are exchanged, FP64 rows not)
template <typename StageT>
__device__ __forceinline__ void f2_amplitudes(const StageT *__restrict__ S, const F2mSub &R, int o, int i0, int i1, int i2,
                                              int ca, int cb, int cc, bool ok0, bool ok1, const double2 *tab,
                                              const double2 *tf, double (&WW)[2][6], double (&VV)[2][6]) {
    const int loc[3] = {ca, cb, cc};
    int w0[6], w1[6], t0[6];   // this thread's positions in the regions (elements a, a + 4) and tables
#pragma unroll
    for (int pi = 0; pi < 6; pi++) {
        int pp[3] = {0, 0, 0};
        perm_of(pi, pp);
        const int x = loc[pp[0]], y = loc[pp[1]], z = loc[pp[2]];
        const int ex = R.len[pp[0]], ez = R.len[pp[2]];
        const bool swz = sizeof(StageT) == 4 && ex == 8 && ez == 8;
        const int dx = pp[0] == 0 ? 4 : 0, dy = pp[1] == 0 ? 4 : 0, dz = pp[2] == 0 ? 4 : 0;
        const int s0 = (x * ez + z) ^ (swz ? f2m_row_swizzle(y) : 0);
        const int s1 = ((x + dx) * ez + z + dz) ^ (swz ? f2m_row_swizzle(y + dy) : 0);
        w0[pi] = ok0 ? y * ex * ez + s0 : 0;
        w1[pi] = ok1 ? (y + dy) * ex * ez + s1 : w0[pi];
        t0[pi] = f2_tab(x, y);
    }
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
        for (int s = 0; s < 6; s++) WW[e][s] = VV[e][s] = 0.0;
    __syncthreads();   // the tables are complete
#pragma unroll
    for (int rho = 0; rho < 6; rho++) {
        int pr[3] = {0, 0, 0};
        perm_of(rho, pr);
        const int ids[3] = {i0, i1, i2};
        const long long idx = ((long long)ids[pr[0]] * o + ids[pr[1]]) * o + ids[pr[2]];
        const double2 *tr = tf + pr[2] * 24;
        const double2 tz[3] = {tr[ca], tr[8 + cb], tr[16 + cc]}, tz4 = tr[(ca + 4) & 7];
#pragma unroll
        for (int pi = 0; pi < 6; pi++) {
            const int s = f2m_sof(pi, rho);
            int pp[3] = {0, 0, 0};
            perm_of(pi, pp);
            const StageT *base = S + R.pi[pi].s0 + idx * R.pi[pi].rs;
            WW[0][s] += (double)__ldg(base + w0[pi]);
            WW[1][s] += (double)__ldg(base + w1[pi]);
            const double2 *tp = tab + (rho * 6 + pi) * 64;
            // a + 4 in slot x or y of the table block
            const double2 ot0 = tp[t0[pi]];
            const double2 ot1 = pp[0] == 0 ? tp[t0[pi] ^ 4] : (pp[1] == 0 ? tp[t0[pi] ^ 32] : ot0);
            const double2 z0 = tz[pp[2]], z1 = pp[2] == 0 ? tz4 : tz[pp[2]];
            VV[0][s] += ot0.x * z0.x + ot0.y * z0.y;
            VV[1][s] += ot1.x * z1.x + ot1.y * z1.y;
        }
    }
}

// Orbital-energy gradient: dd = dE/dD of the thread's elements.  Per-warp sums
// over two of the slots each, then dE/de of i, j, k (+ the total) and of the
// virtuals (- the sums of their slot).
__device__ __forceinline__ void f2_dd_partials(const double (&dd)[2], double (*s_part)[12]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double dc = dd[0] + dd[1], db = dc;
    dc += __shfl_xor_sync(0xffffffffu, dc, 4);
    dc += __shfl_xor_sync(0xffffffffu, dc, 8);
    dc += __shfl_xor_sync(0xffffffffu, dc, 16);
    db += __shfl_xor_sync(0xffffffffu, db, 1);
    db += __shfl_xor_sync(0xffffffffu, db, 2);
    db += __shfl_xor_sync(0xffffffffu, db, 16);
    const bool up = lane & 1;
    double da = (up ? dd[1] : dd[0]) + __shfl_xor_sync(0xffffffffu, up ? dd[0] : dd[1], 1);
    da += __shfl_xor_sync(0xffffffffu, da, 2);
    da += __shfl_xor_sync(0xffffffffu, da, 4);
    da += __shfl_xor_sync(0xffffffffu, da, 8);
    if (lane < 4) s_part[warp][lane] = dc;
    if ((lane & 19) == 0) s_part[warp][4 + (lane >> 2)] = db;
    if ((lane & 14) == 0) s_part[warp][8 + (lane >> 4) + 2 * (lane & 1)] = da;
}

__device__ __forceinline__ void f2_dd_add(double (*s_part)[12], const F2mSub &R, int o, int i0, int i1, int i2,
                                          double *mo_bar) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x >= 24) return;
    // warps with bit 0, 1, 2 = bit 2 of c, bit 2 of b, bit 1 of a (lanes: c, b, a)
    double acc = 0.0;
    const int l = lane & 7;
    for (int u = 0; u < 4; u++)
        acc += lane < 8 ? s_part[(l >> 2) + 2 * u][l & 3]
               : lane < 16 ? s_part[2 * (l >> 2) + (u & 1) + 4 * (u >> 1)][4 + (l & 3)]
                           : s_part[4 * ((l >> 1) & 1) + u][8 + (l & 1) + 2 * (l >> 2)];
    double tot = acc;
    tot += __shfl_xor_sync(0x00ffffffu, tot, 1);
    tot += __shfl_xor_sync(0x00ffffffu, tot, 2);
    tot += __shfl_xor_sync(0x00ffffffu, tot, 4);
    const int slot = 2 - (lane >> 3);
    if (l < sel3(R.len[0], R.len[1], R.len[2], slot))
        red_add(&mo_bar[o + sel3(R.st[0], R.st[1], R.st[2], slot) + l], -acc);
    if (lane < 3) red_add(&mo_bar[sel3(i0, i1, i2, lane)], tot);
}

// Write-back of the element results sW, sV (planes of 512 in f2m_res order): the
// leading regions, one per warp at a time, runs (yy, xx) of lane and u.  Wbar
// leaves as whole runs; V-term gradients v = ovov[p,x,q,y] t1[r,z] + t2[q,p,y,x] fvo[z,r]
// as row sums per run and column sums over the region.  Results and tables are
// zero beyond a short range.
template <int SPLIT, typename ARGS>
__device__ __forceinline__ void f2_writeback(const ARGS &A, const F2mSub &R, int i0, int i1, int i2, int opat, int vpat,
                                             const double2 *tab, const double2 *tf, const int (*s_res)[8],
                                             const typename F2Smem<SPLIT>::W *sW, const double *sV) {
    const int o = A.o, v = A.v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l0 = R.len[0], l1 = R.len[1], l2 = R.len[2];
    const int nro = f2m_nlead(opat), ntask = f2m_nlead(vpat) * nro;
    const int xx = lane & 7, y4 = lane >> 3;
#pragma unroll 1
    for (int task = 7 - warp; task < ntask; task += 8) {
        const int pi = f2m_lead(vpat, task / nro), rho = f2m_lead(opat, task % nro);
        int pp[3], pr[3];
        perm_of(pi, pp);
        perm_of(rho, pr);
        const int p = sel3(i0, i1, i2, pr[0]), q = sel3(i0, i1, i2, pr[1]), r = sel3(i0, i1, i2, pr[2]);
        const int lx = sel3(l0, l1, l2, pp[0]), ly = sel3(l0, l1, l2, pp[1]), lz = sel3(l0, l1, l2, pp[2]);
        const int inv0 = pr[0] == 0 ? 0 : (pr[1] == 0 ? 1 : 2), inv1 = pr[0] == 1 ? 0 : (pr[1] == 1 ? 1 : 2);
        const int s = perm_index(sel3(pp[0], pp[1], pp[2], inv0), sel3(pp[0], pp[1], pp[2], inv1));
        const F2mPi &D = R.pi[pi];
        const long long wl = f2m_wbar(D, p, q, r) + (long long)xx * D.wx;
        const double2 *trow = tf + (pr[2] * 3 + pp[2]) * 8;
        const double2 *tp = tab + (rho * 6 + pi) * 64;
        const int x = sel3(R.st[0], R.st[1], R.st[2], pp[0]) + xx;
        const int y0 = sel3(R.st[0], R.st[1], R.st[2], pp[1]);
        const int gx = s * 512, gxx = s_res[pp[0]][xx];
        double col[16];
#pragma unroll
        for (int c = 0; c < 16; c++) col[c] = 0.0;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int yy = y4 + 4 * u;
            const int g0 = gxx ^ s_res[pp[1]][yy];
            const bool in = xx < lx && yy < ly;
            int gz[8];
#pragma unroll
            for (int z = 0; z < 8; z++) gz[z] = gx + (g0 ^ s_res[pp[2]][z]);
            if (in) {
                if constexpr (SPLIT == 0) {
                    double *dst = reinterpret_cast<double *>(A.SW) + wl + (long long)yy * D.wy;
                    if (lz == 8) {
#pragma unroll
                        for (int z = 0; z < 8; z += 2)
                            *reinterpret_cast<double2 *>(dst + z) = make_double2(sW[gz[z]], sW[gz[z + 1]]);
                    } else {
#pragma unroll
                        for (int z = 0; z < 4; z++)
                            if (z < lz) dst[z] = sW[gz[z]];
                    }
                } else {
                    uint16_t *dst = reinterpret_cast<uint16_t *>(A.SW) + wl + (long long)yy * D.wy;
                    uint32_t pk[8];
#pragma unroll
                    for (int z = 0; z < 8; z++) pk[z] = (uint32_t)sW[gz[z]];
                    if (lz == 8) {
                        uint4 hi, lo;
                        hi.x = __byte_perm(pk[0], pk[1], 0x5410); lo.x = __byte_perm(pk[0], pk[1], 0x7632);
                        hi.y = __byte_perm(pk[2], pk[3], 0x5410); lo.y = __byte_perm(pk[2], pk[3], 0x7632);
                        hi.z = __byte_perm(pk[4], pk[5], 0x5410); lo.z = __byte_perm(pk[4], pk[5], 0x7632);
                        hi.w = __byte_perm(pk[6], pk[7], 0x5410); lo.w = __byte_perm(pk[6], pk[7], 0x7632);
                        *reinterpret_cast<uint4 *>(dst) = hi;
                        *reinterpret_cast<uint4 *>(dst + D.half) = lo;
                    } else {
#pragma unroll
                        for (int z = 0; z < 4; z++)
                            if (z < lz) {
                                dst[z] = (uint16_t)pk[z];
                                dst[D.half + z] = (uint16_t)(pk[z] >> 16);
                            }
                    }
                }
            }
            // v = ovov[p,x,q,y] t1[r,z] + t2[q,p,y,x] fvo[z,r] (results and tables are zero beyond a short range)
            const double2 ot = tp[f2_tab(xx, yy)];
            double r1 = 0.0, r2 = 0.0;
#pragma unroll
            for (int z = 0; z < 8; z++) {
                const double vb = sV[gz[z]];
                const double2 tr = trow[z];
                r1 += vb * tr.x;
                r2 += vb * tr.y;
                col[z] += vb * ot.x;
                col[8 + z] += vb * ot.y;
            }
            if (in) {
                red_add(&A.ovov_bar[(((long long)p * v + x) * o + q) * v + y0 + yy], r1);
                red_add(&A.t2_bar[(((long long)q * o + p) * v + y0 + yy) * v + x], r2);
            }
        }
        // column sums t1_bar[r, z] (values 0-7), fvo_bar[z, r] (8-15) over the region's runs
        const double cv = group_reduce_scatter<16, 32>(col, lane);
        if (lane < 16 && (lane & 7) < lz) {
            const int z = sel3(R.st[0], R.st[1], R.st[2], pp[2]) + (lane & 7);
            if (lane < 8) red_add(&A.t1_bar[(long long)r * v + z], cv);
            else red_add(&A.fvo_bar[(long long)z * o + r], cv);
        }
    }
}

// One CTA per item of the jobs (chunks) of a launch.
template <typename JOBS>
__global__ void __launch_bounds__(kF2Threads, 2) k_f2t(const __grid_constant__ JOBS J) {
    extern __shared__ __align__(16) uint8_t f2_raw[];
    double2 *tab = reinterpret_cast<double2 *>(f2_raw), *tf = tab + 36 * 64;
    double *sV = reinterpret_cast<double *>(f2_raw + F2Smem<0>::TABLES), *sW = sV + 6 * 512;
    __shared__ int s_res[3][8];
    __shared__ double s_part[8][12], s_e[8];
    JobCursor jcur;
    int blk;
    const int jb = jcur.at(J, (int)blockIdx.x, blk);
    const F2P &A = J.job[JOBS::kOne ? 0 : jb];
    const int o = A.o, tid = threadIdx.x;
    // sub-range triple fastest: the CTAs of one representative run together
    const int rep = blk / A.nsub, sub = blk - rep * A.nsub;
    const F2mSub &R = A.sub[sub];
    const int i0 = A.ijk[3 * rep], i1 = A.ijk[3 * rep + 1], i2 = A.ijk[3 * rep + 2];
    const int opat = (i0 == i2) ? 3 : (i0 == i1 ? 1 : (i1 == i2 ? 2 : 0));
    const int vpat = R.pat;
    if (tid < 24) s_res[tid >> 3][tid & 7] = f2m_res(tid >> 3, tid & 7);
    int ca, cb, cc;
    f2_element(tid, ca, cb, cc);
    const bool ok0 = ca < R.len[0] && cb < R.len[1] && cc < R.len[2];
    const bool ok1 = ok0 && ca + 4 < R.len[0];
    f2_load_tables(A, R, i0, i1, i2, tab, tf);
    const double *ev = A.mo_e + o;
    const double e_occ = A.mo_e[i0] + A.mo_e[i1] + A.mo_e[i2];
    const double e_bc = ok0 ? ev[R.st[1] + cb] + ev[R.st[2] + cc] : 0.0;
    double WW[2][6], VV[2][6];
    f2_amplitudes(static_cast<const double *>(A.S), R, o, i0, i1, i2, ca, cb, cc, ok0, ok1, tab, tf, WW, VV);
    // orbit weights: n_ijk n_abc / 18 for three distinct virtuals; the energy
    // counts each orbit once per ordering of equal sub-ranges
    const double cocc = opat == 0 ? 2.0 : (opat == 3 ? 6.0 / 18.0 : 1.0);
    const double cen = vpat == 0 ? cocc : (vpat == 3 ? cocc / 6.0 : cocc * 0.5);
    const int gidx = f2m_res(0, ca) ^ f2m_res(1, cb) ^ f2m_res(2, cc);
    double e_loc = 0.0, dd[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const bool ok = e == 0 ? ok0 : ok1;
        double X[6], Z[6], RW[6];
#pragma unroll
        for (int s = 0; s < 6; s++) X[s] = WW[e][s] + 0.5 * VV[e][s];
        f2_r3(X, Z);
        f2_r3(WW[e], RW);
        const double rD = ok ? 1.0 / (e_occ - ev[R.st[0] + ca + 4 * e] - e_bc) : 0.0;
        double esum = 0.0;
#pragma unroll
        for (int s = 0; s < 6; s++) esum += WW[e][s] * Z[s];
        e_loc += ok ? cen * esum * rD : 0.0;
        dd[e] = ok ? -cen * A.ybar * esum * rD * rD : 0.0;
        if (A.want_grad) {
            const double g0 = cocc * A.ybar * rD;
            double wb[6], vb[6];
#pragma unroll
            for (int s = 0; s < 6; s++) {
                wb[s] = ok ? g0 * (Z[s] + RW[s]) : 0.0;
                vb[s] = ok ? g0 * 0.5 * RW[s] : 0.0;
            }
            const int g = e == 0 ? gidx : gidx ^ 4;
            // equal occupied indices: the orderings that name the same raw amplitudes add up
            double w3 = 0.0, v3 = 0.0;
            if (opat == 3) {
#pragma unroll
                for (int s = 0; s < 6; s++) {
                    w3 += wb[s];
                    v3 += vb[s];
                }
            }
#pragma unroll
            for (int s = 0; s < 6; s++) {
                const int s1 = perm_compose(s, 2), s2 = perm_compose(s, 1);
                sW[s * 512 + g] = opat == 0 ? wb[s] : opat == 1 ? wb[s] + wb[s1] : opat == 2 ? wb[s] + wb[s2] : w3;
                sV[s * 512 + g] = opat == 0 ? vb[s] : opat == 1 ? vb[s] + vb[s1] : opat == 2 ? vb[s] + vb[s2] : v3;
            }
        }
    }
    for (int off = 16; off > 0; off >>= 1) e_loc += __shfl_xor_sync(0xffffffffu, e_loc, off);
    if ((tid & 31) == 0) s_e[tid >> 5] = e_loc;
    f2_dd_partials(dd, s_part);
    __syncthreads();
    if (tid == 32) {
        double es = 0.0;
        for (int w = 0; w < kF2Threads / 32; w++) es += s_e[w];
        A.e_part[(long long)sub * A.n_ijk + rep] = es;
    }
    if (!A.want_grad) return;
    f2_dd_add(s_part, R, o, i0, i1, i2, A.mo_bar);
    f2_writeback<0>(A, R, i0, i1, i2, opat, vpat, tab, tf, s_res, sW, sV);
}

// Sum of the energy partials of one epilogue launch, in a fixed order.
__device__ __forceinline__ void energy_sum_body(const double *__restrict__ e_part, int n, double *e_acc) {
    __shared__ double s[256];
    double acc = 0.0;
    for (int b = threadIdx.x; b < n; b += blockDim.x) acc += e_part[b];
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) *e_acc += s[0];
}

}  // namespace tb
