// Chunk epilogue of the mixed-precision modes: energy and adjoint of the raw
// triples amplitudes, every work item of a chunk in one launch.
//
// A work item is one occupied representative i >= j >= k and one triple of
// virtual sub-ranges R0 >= R1 >= R2 (8 wide; shorter only where a remainder
// block is).  Its 36 regions are the pairs (sub-range ordering pi, occupied
// ordering rho), 8^3 raw amplitudes each.  Per element (a, b, c) of
// R0 x R1 x R2, with d = s(abc) the six orderings,
//   WW(s) = sum_tau w(tau(ijk), tau(s abc)),  VV(s) likewise from v,
//   X = WW + VV/2,  Z = r3(X),  E += c_E sum_s WW Z / D,
//   Wbar(s) = c (Z + r3 WW)/D,  Vbar(s) = c r3(WW)/(2D)
// (pyscfad/cc/ccsd_t_slow.py:46-124, pyscfadlib/pyscfadlib/vjp/cc/ccsd_t_vjp.c:64-117),
// and every raw position of region (pi, rho) receives the element's result of
// the ordering s with s o rho = pi.
//
// Repeated indices need no element rules:
// * equal occupied indices: the orderings rho and t o rho (t the swap of the
//   equal slots) name the same raw amplitudes.  Both copies are loaded, the
//   element adds the results of s and s o t before it stores them, and only
//   the smaller of the two regions is written back.
// * equal sub-ranges: all 8^3 elements are evaluated, each orbit once per
//   ordering of its equal-range values, so the adjoint weight is that of three
//   distinct virtuals for every element, the energy weight is divided by the
//   number of orderings of the sub-ranges, and again only the leading
//   regions are written back.
//
// Persistent, two CTAs of 8 warps per SM.  Items are handed out in order by a
// counter, so that neighbouring items run at the same time: they read the same
// tables, and where Wbar is stored in rows (x blocks below 8) the two 16-byte
// halves of a sector come from two of them and meet in L2.  Bulk copies stream the items in:
// the regions of one rho at a time (6 x 2 KB, a ring of four that runs ahead
// into the next item; the last warp to read a stage refills it), and the
// V-term tables of the next item (FP32 pairs
// {ovov[p,x,q,y], t2[q,p,y,x]} of 8 x 8 blocks, prepared once per call).  A
// thread owns two elements (a and a + 4).  The regions are contiguous in the
// staging buffer, with the values of a row exchanged so that the six permuted
// gathers of a warp touch each bank at most twice; element results and tables
// are laid out the same way, conflict free for the write-back.
// The write-back gives a region to a warp, two 8-long z runs per lane: Wbar
// leaves as 16-byte hi and lo runs, the V-term gradients as row sums (per
// run) and column sums (over the region's runs) added to the FP64 gradients.
//
// What bounds it: latency at 16 warps per SM (registers and shared memory allow
// no more); issue slots are 45 % busy, HBM is at a quarter of its rate.  What
// holds the warps up are barriers, instruction fetch and memory in equal parts,
// so the code an item runs through is kept short (the instruction cache does
// not hold it otherwise): rare paths and the copies are out of line, the second
// element takes a second turn of the same code, regions are described once per
// item in shared memory.  Everything that prepares later items (next item's
// tables, the load record of the one after) is done by one warp each during the
// write-back, whose regions go to the warps as they come free.  The gradients
// are reached by explicitly global reductions: through generic pointers each
// one first tests for shared memory.
// Measured (nocc 40 nvir 360, one virtual block; nocc 40 nvir 72; nocc 20 nvir
// 180; 48 batched problems, ms):
//   a one-CTA persistent kernel for the all-distinct items and
//   a CTA per item for the rest                               343  285  493  119
//   this kernel, Wbar in rows                                 266  198  396   91
//   Wbar in 8 x 8 tiles: whole lines per warp, where rows
//   were 16-byte halves of sectors from two items             213  165  324   89
//   short code, records, preparation in the write-back          -  132  265   60
//   global reductions                                         156  119  242   56
// (In rows, items in fixed strides instead of by the counter: 454 ms in the first.)
//
// The FP32 sums keep a fixed order: rows run over z; columns over
// half regions of 32 runs where nothing coincides and every sub-range is
// full ("plain" items), else over the whole region.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tc_f1.cuh"
#include "tc_ptx.cuh"

namespace tb {

constexpr int kF2mThreads = 256;
constexpr int kF2mStages = 4;      // ring of W stages (the six regions of one rho)
constexpr int kF2mMaxSub = 8;      // sub-range triples of a chunk: (16 / 8)^3

// One ordering pi of a sub-range triple: where its regions lie.
struct F2mPi {
    long long s0;         // staging: region of p = q = r = 0
    long long w0;         // Wbar (hi plane): first position of that region
    long long half;       // lo plane - hi plane
    int rs;               // staging stride of r (q: o rs, p: o o rs)
    int wx, wy, wp, wq;   // Wbar strides of x, y, p, q
    int tz, zs;           // rz = r tz + zs + z
    int tiled;            // rz strides by 64 per 8 values (8 x 8 tiles), else by 1
    int bytes;            // of a region
};

// Wbar offset of (p, q, r), first x, y and z of a region
__device__ __forceinline__ long long f2m_wbar(const F2mPi &D, int p, int q, int r) {
    const int rz = r * D.tz + D.zs;
    return D.w0 + (long long)p * D.wp + (long long)q * D.wq + (D.tiled ? (rz >> 3) * 64 + (rz & 7) : rz);
}

struct F2mSub {
    int st[3], len[3];
    int pat;              // 0: distinct, 1: R0 = R1, 2: R1 = R2, 3: all equal
    int full;             // three full 8-wide sub-ranges
    int bulk;             // bit pi: the regions of pi are multiples of 16 bytes (bulk copies)
    int bulk_bytes;       // their bytes per rho
    F2mPi pi[6];
};

struct F2M {
    int o, v, nb8;        // nb8: 8-wide blocks of the virtual range
    int nsub, n_ijk;
    int whole;            // column sums over whole regions for every item
    const int *ijk;
    const double *mo_e, *t1, *t2, *ovov, *fvo;
    const float2 *ot;     // V-term tables [p][q][x block][y block][64] (f2m_tab order), or null
    const float2 *tf;     // {t1[r,z], fvo[z,r]} as [r][z block][8]
    const float *S;
    uint16_t *SW;
    const double *wscale;
    double ybar;
    int want_grad;
    double *e_part;       // energy partial of each item, at sub * n_ijk + rep
    double *mo_bar, *t1_bar, *fvo_bar, *ovov_bar, *t2_bar;
    int *err;
    unsigned *ticket;     // items handed out beyond the first of each CTA; zero before the launch
    F2mSub sub[kF2mMaxSub];
};

// position of (x, y) in a 64-entry V-term table block: 16 consecutive entries
// (8 bytes each) are one pass over the banks
__host__ __device__ inline int f2m_tab(int x, int y) {
    return ((y >> 1) << 4) | (x ^ ((y & 1) << 3) ^ (((y >> 1) & 1) * 12));
}

// position of element coordinate l of slot 0, 1, 2 in a result plane (XOR of the three)
__host__ __device__ inline int f2m_res(int slot, int l) {
    return slot == 0 ? l
           : slot == 1 ? ((l & 1) * 8) ^ (((l >> 1) & 1) * 27) ^ (((l >> 2) & 1) * 36)
                       : ((l & 1) * 73) ^ (((l >> 1) & 1) * 138) ^ (((l >> 2) & 1) * 260);
}

// the ordering s with perm_compose(s, rho) == pi
__host__ __device__ constexpr int f2m_sof(int pi, int rho) {
    int r = 0;
    for (int s = 0; s < 6; s++)
        if (perm_compose(s, rho) == pi) r = s;
    return r;
}

// Leading orderings (of the pairs named by one swap): 1: slots 0, 1 equal, 2: slots 1, 2 equal
__device__ __forceinline__ int f2m_lead(int pat, int k) {
    return pat == 0 ? k : pat == 3 ? 0 : (k == 0 ? 0 : (pat == 1 ? (k == 1 ? 1 : 4) : (k == 1 ? 2 : 3)));
}
__device__ __forceinline__ int f2m_nlead(int pat) { return pat == 0 ? 6 : (pat == 3 ? 1 : 3); }

__device__ __forceinline__ int sel3(int a, int b, int c, int i) { return i == 0 ? a : (i == 1 ? b : c); }

// A region to write back, formed once per item by one thread each.
struct __align__(16) F2mTask {
    uint16_t *w;          // Wbar: hi plane, first position
    double *ob, *tb;      // ovov_bar, t2_bar: first x and y
    unsigned code;        // bits 0-2 pi, 3-5 rho, 6-11 slots of pi, 12-14 s with s o rho = pi,
                          // 15-16 slot of r, 17-28 lx, ly, lz
    unsigned rz;          // r, first z << 16
};

struct F2mSmem {
    static constexpr int REGION = 512;                                    // floats
    static constexpr int STAGE = 6 * REGION;
    static constexpr int TAB = 36 * 64;                                   // float2 per table buffer
    static constexpr int TF = 9 * 8;                                      // float2
    static constexpr size_t OFF_TAB = sizeof(float) * kF2mStages * STAGE;
    static constexpr size_t OFF_TF = OFF_TAB + sizeof(float2) * 2 * TAB;
    static constexpr size_t OFF_RES = OFF_TF + sizeof(float2) * 2 * TF;
    static constexpr size_t OFF_REC = OFF_RES + sizeof(uint2) * 6 * 512;
    static constexpr size_t BYTES = OFF_REC + sizeof(F2mTask) * 36 + 128;   // +128: base alignment
    static_assert(2 * (BYTES + 2048 + 1024) <= 228 * 1024, "two blocks per SM, with the static arrays");
    static_assert(OFF_TAB % 16 == 0 && OFF_TF % 16 == 0 && OFF_RES % 16 == 0, "bulk copy destinations");
};

// {ovov[p,x,q,y], t2[q,p,y,x]} and {t1[r,z], fvo[z,r]} in FP32 blocks, zero beyond nvir
__global__ void k_prep_vtables(const double *__restrict__ ovov, const double *__restrict__ t2,
                               const double *__restrict__ t1, const double *__restrict__ fvo, int o, int v, int nb8,
                               float2 *__restrict__ ot, float2 *__restrict__ tf) {
    const long long n = (long long)o * o * nb8 * nb8 * 64;
    const long long stride = (long long)gridDim.x * blockDim.x, first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (long long e = first; e < n; e += stride) {
        const int yl = e & 7, xl = (e >> 3) & 7;
        long long t = e >> 6;
        const int yb = t % nb8;
        t /= nb8;
        const int xb = t % nb8;
        t /= nb8;
        const int q = t % o, p = t / o, x = xb * 8 + xl, y = yb * 8 + yl;
        float2 val = make_float2(0.f, 0.f);
        if (x < v && y < v)
            val = make_float2((float)ovov[(((long long)p * v + x) * o + q) * v + y],
                              (float)t2[(((long long)q * o + p) * v + y) * v + x]);
        ot[(e & ~63LL) + f2m_tab(xl, yl)] = val;
    }
    for (long long e = first; e < (long long)o * nb8 * 8; e += stride) {
        const int z = e % (nb8 * 8), r = e / (nb8 * 8);
        tf[e] = z < v ? make_float2((float)t1[(long long)r * v + z], (float)fvo[(long long)z * o + r])
                      : make_float2(0.f, 0.f);
    }
}

// hi and lo 16-bit halves of a scaled value, hi in the low half
template <int H>   // 1: fp16, 2: bf16
__device__ __forceinline__ uint32_t f2m_split(float w, float scale) {
    const float x = w * scale;
    if (H == 1) {
        const __half h = __float2half_rn(x), l = __float2half_rn(x - __half2float(h));
        return (uint32_t)__half_as_ushort(h) | ((uint32_t)__half_as_ushort(l) << 16);
    }
    const __nv_bfloat16 h = __float2bfloat16_rn(x), l = __float2bfloat16_rn(x - __bfloat162float(h));
    return (uint32_t)__bfloat16_as_ushort(h) | ((uint32_t)__bfloat16_as_ushort(l) << 16);
}

// What the loads of an item's regions need.
struct F2mSrc {
    const float *src;     // staging: region of pi, p = q = r = 0
    int rs;               // staging stride of r
    int bytes;            // of a region; negative: no bulk copies
};
struct F2mItem {
    int job, sub, rep, i0, i1, i2;
    float wscale;
};
struct F2mLoad {
    F2mSrc pi[6];
    int idx[6];           // (p o + q) o + r of each rho
    int bulk_bytes, pad;
};

// Out of line: the instruction cache holds the code of an item only if its
// rare paths are short.
__device__ __noinline__ void f2m_wait_slow(uint64_t *bar, uint32_t parity, volatile int *abortp, int *err) {
    if (*abortp == 0 && !mbar_wait(bar, parity, abortp)) {
        *abortp = 1;
        // no stage reaches its count of readers any more, so none is refilled
        for (int s = 1; s <= kF2mStages; s++) atomicAdd((int *)abortp - s, 1 << 16);
        atomicOr(err, 64);
    }
}

// After a wait that gave up no further copy is issued, and those in flight land before the CTA ends: each of
// the threads 0 to kF2mStages + 1 waits (with the same limit) for the phase that its barrier is in.  A
// stage or table buffer has at most one load outstanding, because its next one is issued only after every
// warp has waited for it, or not at all.  (A barrier without one waits to the limit.)
__device__ __noinline__ void f2m_drain(uint64_t *bar) {
    const uint32_t phase = mbar_try_wait(bar, 0) ? 1u : 0u;
#pragma unroll 1
    for (uint32_t i = 0; i < kSpinLimit && !mbar_try_wait(bar, phase); i++)
        if ((i & 255u) == 255u) __nanosleep(32);
}

// W stage n of the CTA (one warp): the regions of (item, rho) of a load record;
// every warp has read the stage's previous content.
__device__ __noinline__ void f2m_issue(const F2mLoad *L, int rho, int n, float *sW, uint64_t *full) {
    const int lane = threadIdx.x & 31, st = n & (kF2mStages - 1);
    fence_proxy_async_smem();
    if (lane == 0) mbar_expect_tx(&full[st], (uint32_t)L->bulk_bytes);
    __syncwarp();
    if (lane < 6) {
        const F2mSrc D = L->pi[lane];
        float *dst = sW + st * F2mSmem::STAGE + lane * F2mSmem::REGION;
        const float *src = D.src + (long long)L->idx[rho] * D.rs;
        if (D.bytes > 0) {
            bulk_load(dst, src, (uint32_t)D.bytes, &full[st]);
        } else {
#pragma unroll 1
            for (int e = 0; e < -D.bytes / 4; e++) dst[e] = src[e];   // one or two values
        }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&full[st]);
}

__device__ __forceinline__ void f2m_bar(int id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kF2mThreads) : "memory");
}

// The items of the jobs (chunks) of a launch.
template <int H, typename JOBS>
__global__ void __launch_bounds__(kF2mThreads, 2) k_f2m(const __grid_constant__ JOBS J) {
    constexpr bool ONE = JOBS::kOne;
    const int nitems = J.start[J.n];
    using C = F2mSmem;
    extern __shared__ uint8_t f2m_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)f2m_raw + 127) & ~(uintptr_t)127);
    float *sW = reinterpret_cast<float *>(smem);
    float2 *sTab = reinterpret_cast<float2 *>(smem + C::OFF_TAB);
    float2 *sTF = reinterpret_cast<float2 *>(smem + C::OFF_TF);
    uint2 *sRes = reinterpret_cast<uint2 *>(smem + C::OFF_RES);
    F2mTask *s_rec = reinterpret_cast<F2mTask *>(smem + C::OFF_REC);
    __shared__ uint64_t full[kF2mStages], tfull[2];
    // warps that have read the stage, abort flag, next item of the CTA by parity of the current one
    // (one array: the flag follows the counts, and the static arrays stay within 2048 bytes)
    __shared__ unsigned s_read[kF2mStages + 3];
    __shared__ unsigned s_task[36];                // per (pi, rho): slots of pi, of rho, and s with s o rho = pi
    __shared__ __align__(16) double s_en[2][32];   // energies of the item: 8 per slot, then i, j, k
    __shared__ __align__(16) int s_res[3][8];      // byte offsets of f2m_res
    __shared__ double s_part[8][14];               // per-warp partials: c, b, a sums (4 each), energy
    int *const s_next = reinterpret_cast<int *>(&s_read[kF2mStages + 1]);
    __shared__ __align__(16) F2mLoad s_load[2];    // of the current and the next item
    __shared__ F2mItem s_item[2];
    __shared__ unsigned s_tasks[2];                // regions handed out for write-back

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned *ticket = J.job[0].ticket;
    if (tid == 0) {
        s_read[kF2mStages] = 0u;
        s_next[0] = (int)(gridDim.x + atomicAdd(ticket, 1u));
        for (int s = 0; s < kF2mStages; s++) {
            mbar_init(&full[s], 2);
            s_read[s] = 0u;
        }
        mbar_init(&tfull[0], 2 + 32);
        mbar_init(&tfull[1], 2 + 32);
        fence_mbar_init();
    }
    if (tid < 24) s_res[tid >> 3][tid & 7] = 8 * f2m_res(tid >> 3, tid & 7);
    if (tid < 36) {
        int pp[3], pr[3], s = 0;
        perm_of(tid / 6, pp);
        perm_of(tid % 6, pr);
        for (int c = 0; c < 6; c++)
            if (perm_compose(c, tid % 6) == tid / 6) s = c;
        s_task[tid] = (unsigned)(pp[0] | (pp[1] << 2) | (pp[2] << 4) | (pr[0] << 6) | (pr[1] << 8) | (pr[2] << 10) | (s << 12));
    }
    __syncthreads();
    volatile int *abortp = reinterpret_cast<volatile int *>(&s_read[kF2mStages]);
    // Job of global item w and the item in it (w only grows).
    using Item = F2mItem;
    JobCursor jcur;
    auto item_at = [&](int w) -> Item {
        Item I;
        int lw;
        I.job = jcur.at(J, w, lw);
        const F2M &P = J.job[ONE ? 0 : I.job];
        I.rep = lw / P.nsub;
        I.sub = lw - I.rep * P.nsub;
        I.i0 = P.ijk[3 * I.rep];
        I.i1 = P.ijk[3 * I.rep + 1];
        I.i2 = P.ijk[3 * I.rep + 2];
        I.wscale = P.want_grad ? (float)*P.wscale : 1.0f;
        return I;
    };
    // every wait is bounded; after a timeout the status bit is set, nothing more is loaded and the
    // remaining items run through without waiting (no address depends on the data)
    auto wait = [&](uint64_t *bar, uint32_t parity) {
        if (!mbar_try_wait(bar, parity)) f2m_wait_slow(bar, parity, abortp, J.job[0].err);
    };
    // ---- the loads, each issued by one warp ----
    // V-term tables and energies of an item into table buffer b (its previous item is done)
    auto issue_tables = [&](const Item &I, int b) {
        const F2M &P = J.job[ONE ? 0 : I.job];
        const F2mSub &R = P.sub[I.sub];
        const int o = P.o, v = P.v;
        if (lane < 27) {
            const int sl = lane >> 3, l = lane & 7;
            const bool virt = lane < 24;
            const bool in = !virt || l < sel3(R.len[0], R.len[1], R.len[2], sl);
            const int at = virt ? o + sel3(R.st[0], R.st[1], R.st[2], sl) + l : sel3(I.i0, I.i1, I.i2, lane - 24);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(&s_en[b][lane])),
                         "l"(P.mo_e + (in ? at : 0)), "r"(in ? 8 : 0)
                         : "memory");
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&tfull[b])) : "memory");
        float2 *tab = sTab + b * C::TAB, *tf = sTF + b * C::TF;
        fence_proxy_async_smem();
        if (P.ot != nullptr) {
            if (lane == 0) mbar_expect_tx(&tfull[b], (C::TAB + C::TF) * (uint32_t)sizeof(float2));
            __syncwarp();
            for (int e = lane; e < 45; e += 32) {
                if (e < 36) {
                    int pr[3], pp[3];
                    perm_of(e / 6, pr);
                    perm_of(e % 6, pp);
                    const int p = sel3(I.i0, I.i1, I.i2, pr[0]), q = sel3(I.i0, I.i1, I.i2, pr[1]);
                    const int xb = sel3(R.st[0], R.st[1], R.st[2], pp[0]) >> 3;
                    const int yb = sel3(R.st[0], R.st[1], R.st[2], pp[1]) >> 3;
                    bulk_load(tab + e * 64, P.ot + (((long long)(p * o + q) * P.nb8 + xb) * P.nb8 + yb) * 64,
                              64 * sizeof(float2), &tfull[b]);
                } else {
                    const int r = sel3(I.i0, I.i1, I.i2, (e - 36) / 3);
                    const int zb = sel3(R.st[0], R.st[1], R.st[2], (e - 36) % 3) >> 3;
                    bulk_load(tf + (e - 36) * 8, P.tf + ((long long)r * P.nb8 + zb) * 8, 8 * sizeof(float2), &tfull[b]);
                }
            }
        } else {
            // no prepared tables (the caller's scratch is too small for them): gather the entries
            if (lane == 0) mbar_arrive(&tfull[b]);
            for (int pi = 0; pi < 6; pi++) {
                int pp[3];
                perm_of(pi, pp);
                const int lx = sel3(R.len[0], R.len[1], R.len[2], pp[0]), ly = sel3(R.len[0], R.len[1], R.len[2], pp[1]);
                const int sx = sel3(R.st[0], R.st[1], R.st[2], pp[0]), sy = sel3(R.st[0], R.st[1], R.st[2], pp[1]);
                for (int e = lane; e < 6 * lx * ly; e += 32) {
                    const int rho = e / (lx * ly), xl = (e / ly) % lx, yl = e % ly;
                    int pr[3];
                    perm_of(rho, pr);
                    const int p = sel3(I.i0, I.i1, I.i2, pr[0]), q = sel3(I.i0, I.i1, I.i2, pr[1]);
                    tab[(rho * 6 + pi) * 64 + f2m_tab(xl, yl)] =
                        make_float2((float)P.ovov[(((long long)p * v + sx + xl) * o + q) * v + sy + yl],
                                    (float)P.t2[(((long long)q * o + p) * v + sy + yl) * v + sx + xl]);
                }
            }
            for (int e = lane; e < C::TF; e += 32) {
                const int r = sel3(I.i0, I.i1, I.i2, e / 24), s = (e >> 3) % 3, zl = e & 7;
                const int z = sel3(R.st[0], R.st[1], R.st[2], s) + zl;
                if (zl < sel3(R.len[0], R.len[1], R.len[2], s))
                    tf[e] = make_float2((float)P.t1[(long long)r * v + z], (float)P.fvo[(long long)z * o + r]);
            }
            __syncwarp();
        }
        if (lane == 0) mbar_arrive(&tfull[b]);
    };
    // the load record of an item (one warp; the readers are ordered behind it by the stage counts)
    auto load_record = [&](const Item &I, F2mLoad &L) {
        const F2M &P = J.job[ONE ? 0 : I.job];
        const F2mSub &R = P.sub[I.sub];
        if (lane < 6) {
            const F2mPi &D = R.pi[lane];
            L.pi[lane] = F2mSrc{P.S + D.s0, D.rs, (R.bulk >> lane) & 1 ? D.bytes : -D.bytes};
            int pr[3];
            perm_of(lane, pr);
            L.idx[lane] = (sel3(I.i0, I.i1, I.i2, pr[0]) * P.o + sel3(I.i0, I.i1, I.i2, pr[1])) * P.o +
                          sel3(I.i0, I.i1, I.i2, pr[2]);
        }
        if (lane == 0) L.bulk_bytes = R.bulk_bytes;
        __syncwarp();
    };
    // elements (a, b, c) and (a + 4, b, c); a warp spans 2 x 4 x 4 of them
    const int ca = ((tid >> 4) & 1) | (((tid >> 7) & 1) << 1);
    const int cb = ((tid >> 2) & 3) | (((tid >> 6) & 1) << 2);
    const int cc = (tid & 3) | (((tid >> 5) & 1) << 2);
    const int gidx = f2m_res(0, ca) ^ f2m_res(1, cb) ^ f2m_res(2, cc);
    // positions of element (a, b, c) in the regions and tables of each pi
    int woff[6], toff[6];
    auto offsets = [&](const F2mSub &R, bool tables) {
        const int loc[3] = {ca, cb, cc};
#pragma unroll
        for (int pi = 0; pi < 6; pi++) {
            int pp[3] = {0, 0, 0};
            perm_of(pi, pp);
            const int x = loc[pp[0]], y = loc[pp[1]], z = loc[pp[2]];
            const int ex = R.len[pp[0]], ez = R.len[pp[2]];
            if (R.full || (ex == 8 && ez == 8)) woff[pi] = pi * C::REGION + y * 64 + ((x * 8 + z) ^ f2m_row_swizzle(y));
            else woff[pi] = pi * C::REGION + (((y * ex + x) * ez + z) & 255);   // beyond a short range: any slot
            // a short sub-range may start inside its 8-wide table block
            const int ox = tables && !R.full ? R.st[pp[0]] & 7 : 0, oy = tables && !R.full ? R.st[pp[1]] & 7 : 0;
            toff[pi] = f2m_tab((x + ox) & 7, (y + oy) & 7);
        }
    };

    if ((int)blockIdx.x >= nitems) return;
    Item cur = item_at(blockIdx.x);
    if (tid == 0) s_item[0] = cur;
    bool full_offsets = false;
    if (warp == 0) {
        issue_tables(cur, 0);
        load_record(cur, s_load[0]);
#pragma unroll 1
        for (int n = 0; n < kF2mStages; n++) f2m_issue(&s_load[0], n, n, sW, full);
    }
    // item w of the CTA's parity b, formed by one warp ahead of the first use
    auto announce = [&](int w, int b) {
        const Item I = item_at(w);
        if (lane == 0) s_item[b] = I;
        load_record(I, s_load[b]);
    };
    if (warp == 2 && s_next[0] < nitems) announce(s_next[0], 1);
#pragma unroll 1
    for (int k = 0;; k++) {
        const F2M &P = J.job[ONE ? 0 : cur.job];
        const int wn = s_next[k & 1];
        const bool more = wn < nitems;
        unsigned tk = 0;
        if (tid == 0 && more) tk = atomicAdd(ticket, 1u);
        const F2mSub &R = P.sub[cur.sub];
        const bool plain = !P.whole && R.full && R.pat == 0 && cur.i0 != cur.i2;
        if (!R.full || !full_offsets) {
            offsets(R, P.ot != nullptr);
            full_offsets = R.full != 0;
        }
        const bool shifted = !R.full && P.ot != nullptr;
        const int s0 = shifted ? R.st[0] & 7 : 0, s1 = shifted ? R.st[1] & 7 : 0, s2 = shifted ? R.st[2] & 7 : 0;
        const int tb_ = k & 1;
        const float2 *tab = sTab + tb_ * C::TAB, *tf = sTF + tb_ * C::TF;
        wait(&tfull[tb_], (k >> 1) & 1);

        double WW[2][6];
        float VV[2][6];
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
            for (int s = 0; s < 6; s++) {
                WW[e][s] = 0.0;
                VV[e][s] = 0.f;
            }
#pragma unroll
        for (int rho = 0; rho < 6; rho++) {
            const int n = 6 * k + rho, st = n & (kF2mStages - 1);
            int pr[3] = {0, 0, 0};
            perm_of(rho, pr);
            // {t1, fvo} of the occupied index pr[2] at a, a + 4, b, c
            const float2 *tr = tf + pr[2] * 24;
            const float2 tz[3] = {tr[(ca + s0) & 7], tr[8 + ((cb + s1) & 7)], tr[16 + ((cc + s2) & 7)]};
            const float2 tz4 = tr[ca + 4];
            wait(&full[st], (n / kF2mStages) & 1);
            const float *Ws = sW + st * C::STAGE;
#pragma unroll
            for (int pi = 0; pi < 6; pi++) {
                const int s = f2m_sof(pi, rho);
                int pp[3] = {0, 0, 0};
                perm_of(pi, pp);
                // the second element: a + 4 in slot x (+32), y (+256) or z (exchanged bit 2)
                const float w0 = Ws[woff[pi]];
                const float w1 = pp[0] == 0 ? Ws[woff[pi] + 32] : (pp[1] == 0 ? Ws[woff[pi] + 256] : Ws[woff[pi] ^ 4]);
                WW[0][s] += (double)w0;
                WW[1][s] += (double)w1;
                const float2 *tp = tab + (rho * 6 + pi) * 64;
                const float2 ot0 = tp[toff[pi]];
                const float2 ot1 = pp[0] == 0 ? tp[toff[pi] ^ 4] : (pp[1] == 0 ? tp[toff[pi] ^ 32] : ot0);
                const float2 z0 = tz[pp[2]], z1 = pp[2] == 0 ? tz4 : tz[pp[2]];
                if (plain) {
                    VV[0][s] = fmaf(ot0.x, z0.x, fmaf(ot0.y, z0.y, VV[0][s]));
                    VV[1][s] = fmaf(ot1.x, z1.x, fmaf(ot1.y, z1.y, VV[1][s]));
                } else {
                    VV[0][s] = __fadd_rn(VV[0][s], fmaf(ot0.x, z0.x, __fmul_rn(ot0.y, z0.y)));
                    VV[1][s] = __fadd_rn(VV[1][s], fmaf(ot1.x, z1.x, __fmul_rn(ot1.y, z1.y)));
                }
            }
            // the last warp to read the stage refills it
            __syncwarp();
            unsigned seen = 0;
            if (lane == 0) {
                __threadfence_block();
                seen = atomicAdd(&s_read[st], 1u);
            }
            seen = __shfl_sync(0xffffffffu, seen, 0);
            if (seen == 7u) {
                __threadfence_block();
                if (lane == 0) s_read[st] = 0u;
                if (rho + kF2mStages < 6) f2m_issue(&s_load[k & 1], rho + kF2mStages, n + kF2mStages, sW, full);
                else if (more) f2m_issue(&s_load[(k & 1) ^ 1], rho + kF2mStages - 6, n + kF2mStages, sW, full);
            }
        }

        // what only the second half needs is read here, not held in registers through the first
        const F2mItem it = s_item[k & 1];
        const int o = P.o, v = P.v;
        const int i0 = it.i0, i1 = it.i1, i2 = it.i2;
        const int opat = (i0 == i2) ? 3 : (i0 == i1 ? 1 : (i1 == i2 ? 2 : 0));
        const int vpat = R.pat;
        const int l0 = R.len[0], l1 = R.len[1], l2 = R.len[2];
        const bool ok0 = ca < l0 && cb < l1 && cc < l2, ok1 = ca + 4 < l0 && cb < l1 && cc < l2;
        // orbit weights: n_ijk n_abc / 18 for three distinct virtuals; the energy
        // counts each orbit once per ordering of equal sub-ranges
        const double cocc = opat == 0 ? 2.0 : (opat == 3 ? 6.0 / 18.0 : 1.0);
        const double cen = vpat == 0 ? cocc : (vpat == 3 ? cocc / 6.0 : cocc * 0.5);
        if (tid == 0) s_next[(k & 1) ^ 1] = more ? (int)(gridDim.x + tk) : nitems;
        if (tid == 0) s_tasks[k & 1] = 0u;   // (last used two items ago)
        f2m_bar(1);   // every warp is done with the previous item's results, partials and tables
        const double *en = s_en[tb_];
        const double e_occ = en[24] + en[25] + en[26];
        const int nro = f2m_nlead(opat), ntask = P.want_grad ? f2m_nlead(vpat) * nro : 0;
        if (tid >= 192 && tid - 192 < ntask) {
            const int pi = f2m_lead(vpat, (tid - 192) / nro), rho = f2m_lead(opat, (tid - 192) % nro);
            const unsigned code = s_task[pi * 6 + rho];
            const int p0 = code & 3u, p1 = (code >> 2) & 3u, p2 = (code >> 4) & 3u;
            const int p = sel3(i0, i1, i2, (code >> 6) & 3u), q = sel3(i0, i1, i2, (code >> 8) & 3u);
            const int r = sel3(i0, i1, i2, (code >> 10) & 3u);
            const int x = sel3(R.st[0], R.st[1], R.st[2], p0), y = sel3(R.st[0], R.st[1], R.st[2], p1);
            F2mTask t;
            t.w = P.SW + f2m_wbar(R.pi[pi], p, q, r);
            t.ob = P.ovov_bar + (((long long)p * v + x) * o + q) * v + y;
            t.tb = P.t2_bar + (((long long)q * o + p) * v + y) * v + x;
            t.code = (unsigned)(pi | (rho << 3)) | ((code & 63u) << 6) | (((code >> 12) & 7u) << 12) |
                     (((code >> 10) & 3u) << 15) | ((unsigned)sel3(l0, l1, l2, p0) << 17) |
                     ((unsigned)sel3(l0, l1, l2, p1) << 21) | ((unsigned)sel3(l0, l1, l2, p2) << 25);
            t.rz = (unsigned)r | ((unsigned)sel3(R.st[0], R.st[1], R.st[2], p2) << 16);
            s_rec[tid - 192] = t;
        }
        double e_loc = 0.0, dd[2] = {0.0, 0.0};
        // (a loop of two turns: the element's registers move down, half the code)
#pragma unroll 1
        for (int e = 0; e < 2; e++) {
            const bool ok = e == 0 ? ok0 : ok1;
            double X[6], Z[6], RW[6];
#pragma unroll
            for (int s = 0; s < 6; s++) X[s] = WW[0][s] + 0.5 * (double)VV[0][s];
#pragma unroll
            for (int s = 0; s < 6; s++) {
                Z[s] = 4.0 * X[s] + X[perm_compose(s, 4)] + X[perm_compose(s, 3)] -
                       2.0 * (X[perm_compose(s, 5)] + X[perm_compose(s, 1)] + X[perm_compose(s, 2)]);
                RW[s] = 4.0 * WW[0][s] + WW[0][perm_compose(s, 4)] + WW[0][perm_compose(s, 3)] -
                        2.0 * (WW[0][perm_compose(s, 5)] + WW[0][perm_compose(s, 1)] + WW[0][perm_compose(s, 2)]);
            }
            const double Dn = e_occ - en[ca + 4 * e] - en[8 + cb] - en[16 + cc];
            const double rD = 1.0 / Dn;
            double esum = 0.0;
#pragma unroll
            for (int s = 0; s < 6; s++) esum += WW[0][s] * Z[s];
            e_loc += ok ? cen * esum * rD : 0.0;
            dd[0] = dd[1];
            dd[1] = ok ? cen * P.ybar * esum * rD * rD : 0.0;   // dE/d e_abc (minus dE/dD)
            if (P.want_grad) {
                const double g0 = cocc * P.ybar * rD;
                float wb[6], vb[6];
#pragma unroll
                for (int s = 0; s < 6; s++) {
                    wb[s] = ok ? (float)(g0 * (Z[s] + RW[s])) : 0.f;
                    vb[s] = ok ? (float)(g0 * 0.5 * RW[s]) : 0.f;
                }
                if (opat == 1 || opat == 2) {
                    float w2[6], v2[6];
#pragma unroll
                    for (int s = 0; s < 6; s++) {
                        w2[s] = wb[s] + (opat == 1 ? wb[perm_compose(s, 2)] : wb[perm_compose(s, 1)]);
                        v2[s] = vb[s] + (opat == 1 ? vb[perm_compose(s, 2)] : vb[perm_compose(s, 1)]);
                    }
#pragma unroll
                    for (int s = 0; s < 6; s++) {
                        wb[s] = w2[s];
                        vb[s] = v2[s];
                    }
                } else if (opat == 3) {
                    double ws = 0.0, vs = 0.0;
#pragma unroll
                    for (int s = 0; s < 6; s++) {
                        ws += (double)wb[s];
                        vs += (double)vb[s];
                    }
#pragma unroll
                    for (int s = 0; s < 6; s++) {
                        wb[s] = (float)ws;
                        vb[s] = (float)vs;
                    }
                }
                uint2 *g = sRes + (e == 0 ? gidx : gidx ^ 4);
#pragma unroll
                for (int s = 0; s < 6; s++)
                    g[s * 512] = make_uint2(f2m_split<H>(wb[s], it.wscale), __float_as_uint(vb[s]));
            }
#pragma unroll
            for (int s = 0; s < 6; s++) {
                WW[0][s] = WW[1][s];
                VV[0][s] = VV[1][s];
            }
        }
        // per-warp partials: dE/d e_c (lanes 0-3), e_b (0, 4, 8, 12), e_a and e_(a+4), energy
        {
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
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) e_loc += __shfl_xor_sync(0xffffffffu, e_loc, off);
            if (lane < 4) s_part[warp][lane] = dc;
            if ((lane & 19) == 0) s_part[warp][4 + (lane >> 2)] = db;
            if ((lane & 14) == 0) s_part[warp][8 + (lane >> 4) + 2 * (lane & 1)] = da;
            if (lane == 0) s_part[warp][12] = e_loc;
        }
        f2m_bar(2);   // results and partials visible
        // (these warps take fewer regions below)
        if (warp == 1 && more && s_read[kF2mStages] == 0u) issue_tables(s_item[(k & 1) ^ 1], tb_ ^ 1);
        if (warp == 2 && s_next[(k & 1) ^ 1] < nitems) announce(s_next[(k & 1) ^ 1], k & 1);
        if (warp == 0) {
            // warps with bit 0, 1, 2 = bit 2 of c, bit 2 of b, bit 1 of a
            double acc = 0.0;
            if (lane < 8) {
                for (int u = 0; u < 4; u++) acc += s_part[(lane >> 2) + 2 * u][lane & 3];
            } else if (lane < 16) {
                const int b = lane - 8;
                for (int u = 0; u < 4; u++) acc += s_part[2 * (b >> 2) + (u & 1) + 4 * (u >> 1)][4 + (b & 3)];
            } else if (lane < 24) {
                const int a = lane - 16;
                for (int u = 0; u < 4; u++) acc += s_part[4 * ((a >> 1) & 1) + u][8 + (a & 1) + 2 * (a >> 2)];
            } else {
                acc = s_part[lane - 24][12];
            }
            double tot = acc;   // over each group of 8 lanes: the slot's total, the energy
            tot += __shfl_xor_sync(0xffffffffu, tot, 1);
            tot += __shfl_xor_sync(0xffffffffu, tot, 2);
            tot += __shfl_xor_sync(0xffffffffu, tot, 4);
            if (lane == 24) P.e_part[(long long)it.sub * P.n_ijk + it.rep] = tot;
            if (P.want_grad) {
                const int slot = 2 - (lane >> 3), l = lane & 7;
                if (lane < 24 && l < sel3(l0, l1, l2, slot))
                    red_add(&P.mo_bar[o + sel3(R.st[0], R.st[1], R.st[2], slot) + l], acc);
                if (lane >= 16 && lane < 19) red_add(&P.mo_bar[sel3(i0, i1, i2, lane - 16)], -tot);
            }
        }

        if (P.want_grad) {
            // ---- write-back: a region per warp, runs (yy, xx) of lane and u ----
            const int xx = lane & 7, h3 = (lane >> 3) & 1, h4 = lane >> 4;
            const int ys0 = plain ? 2 * h3 + 4 * h4 : h3 + 2 * h4, ydu = plain ? 1 : 4;
#pragma unroll 1
            for (int task = warp, next; task < ntask; task = next) {
                next = 0;
                if (lane == 0) next = 8 + (int)atomicAdd(&s_tasks[k & 1], 1u);   // further ones in order of arrival
                next = __shfl_sync(0xffffffffu, next, 0);
                const F2mTask T = s_rec[task];
                const int pi = T.code & 7u, rho = (T.code >> 3) & 7u;
                const int pp[3] = {(int)((T.code >> 6) & 3u), (int)((T.code >> 8) & 3u), (int)((T.code >> 10) & 3u)};
                const int s = (T.code >> 12) & 7u, pr2 = (T.code >> 15) & 3u;
                const int lx = (T.code >> 17) & 15u, ly = (T.code >> 21) & 15u, lz = (T.code >> 25) & 15u;
                const uint8_t *plane = reinterpret_cast<const uint8_t *>(sRes + s * 512);
                const int gx = s_res[pp[0]][xx];
                const int4 za = *reinterpret_cast<const int4 *>(&s_res[pp[2]][0]);
                const int4 zb = *reinterpret_cast<const int4 *>(&s_res[pp[2]][4]);
                const int zo[8] = {za.x, za.y, za.z, za.w, zb.x, zb.y, zb.z, zb.w};
                const F2mPi &D = R.pi[pi];
                uint16_t *const wl = T.w + (long long)xx * D.wx;
                const float2 *trow = tf + (pr2 * 3 + pp[2]) * 8;
                float2 trz[8];
                if (R.full) {
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const float4 t = reinterpret_cast<const float4 *>(trow)[c];
                        trz[2 * c] = make_float2(t.x, t.y);
                        trz[2 * c + 1] = make_float2(t.z, t.w);
                    }
                } else {
                    // beyond a short range the results are zero but the table may hold anything
                    const int sz = sel3(s0, s1, s2, pp[2]);
#pragma unroll
                    for (int z = 0; z < 8; z++) trz[z] = z < lz ? trow[(z + sz) & 7] : make_float2(0.f, 0.f);
                }
                const int sx = sel3(s0, s1, s2, pp[0]), sy = sel3(s0, s1, s2, pp[1]);
                const float2 *tp = tab + (rho * 6 + pi) * 64;
                float col[16], rs1[2], rs2[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int yy = ys0 + u * ydu;
                    const int g0 = gx ^ s_res[pp[1]][yy];
                    uint32_t pk[8];
                    float vb[8];
#pragma unroll
                    for (int z = 0; z < 8; z++) {
                        const uint2 t = *reinterpret_cast<const uint2 *>(plane + (g0 ^ zo[z]));
                        pk[z] = t.x;
                        vb[z] = __uint_as_float(t.y);
                    }
                    uint4 hi, lo;
                    hi.x = __byte_perm(pk[0], pk[1], 0x5410); lo.x = __byte_perm(pk[0], pk[1], 0x7632);
                    hi.y = __byte_perm(pk[2], pk[3], 0x5410); lo.y = __byte_perm(pk[2], pk[3], 0x7632);
                    hi.z = __byte_perm(pk[4], pk[5], 0x5410); lo.z = __byte_perm(pk[4], pk[5], 0x7632);
                    hi.w = __byte_perm(pk[6], pk[7], 0x5410); lo.w = __byte_perm(pk[6], pk[7], 0x7632);
                    if (xx < lx && yy < ly) {
                        uint16_t *dst = wl + (long long)yy * D.wy;
                        if (lz == 8) {
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
                    // v = ovov[p,x,q,y] t1[r,z] + t2[q,p,y,x] fvo[z,r]
                    const float2 ot = tp[f2m_tab((xx + sx) & 7, (yy + sy) & 7)];
                    const bool in = xx < lx && yy < ly;   // beyond a short range the table is not defined
                    const float ox = in ? ot.x : 0.f, oy = in ? ot.y : 0.f;
                    float r1 = 0.f, r2 = 0.f;
#pragma unroll
                    for (int z = 0; z < 8; z++) {
                        r1 = fmaf(vb[z], trz[z].x, r1);
                        r2 = fmaf(vb[z], trz[z].y, r2);
                    }
                    rs1[u] = r1;
                    rs2[u] = r2;
                    if (u == 0) {
#pragma unroll
                        for (int z = 0; z < 8; z++) {
                            col[z] = __fmul_rn(vb[z], ox);
                            col[8 + z] = __fmul_rn(vb[z], oy);
                        }
                    } else if (plain) {
#pragma unroll
                        for (int z = 0; z < 8; z++) {
                            col[z] = __fadd_rn(col[z], __fmul_rn(vb[z], ox));
                            col[8 + z] = __fadd_rn(col[8 + z], __fmul_rn(vb[z], oy));
                        }
                    } else {
#pragma unroll
                        for (int z = 0; z < 8; z++) {
                            col[z] = fmaf(vb[z], ox, col[z]);
                            col[8 + z] = fmaf(vb[z], oy, col[8 + z]);
                        }
                    }
                }
                // row sums: lanes of one x take four consecutive y (one sector of ovov_bar)
                int yr0 = ys0, yr1 = ys0 + ydu;
                if (plain) {
                    const float a1 = __shfl_xor_sync(0xffffffffu, h4 ? rs1[0] : rs1[1], 16);
                    const float a2 = __shfl_xor_sync(0xffffffffu, h4 ? rs2[0] : rs2[1], 16);
                    // h4 = 0 keeps y = 2 h3 and takes 4 + 2 h3; h4 = 1 takes 2 h3 + 1 and keeps 5 + 2 h3
                    const float k1 = h4 ? rs1[1] : rs1[0], k2 = h4 ? rs2[1] : rs2[0];
                    rs1[0] = h4 ? a1 : k1;
                    rs1[1] = h4 ? k1 : a1;
                    rs2[0] = h4 ? a2 : k2;
                    rs2[1] = h4 ? k2 : a2;
                    yr0 = 2 * h3 + h4;
                    yr1 = yr0 + 4;
                }
                double *ob = T.ob + (long long)(xx * o) * v;
                double *tb2 = T.tb + xx;
                if (xx < lx && yr0 < ly) {
                    red_add(ob + yr0, rs1[0]);
                    red_add(tb2 + (long long)yr0 * v, rs2[0]);
                }
                if (xx < lx && yr1 < ly) {
                    red_add(ob + yr1, rs1[1]);
                    red_add(tb2 + (long long)yr1 * v, rs2[1]);
                }
                // column sums t1_bar[r, z] (values 0-7), fvo_bar[z, r] (8-15); every
                // level adds lane pairs in the order bit 3, 2, 1, 0, 4 of the run
                int ci;
                bool act = true;
                auto fold = [&](int n, int bit) {   // 2n values -> n over lanes that differ in `bit`
                    const bool up = (lane & bit) != 0;
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (i < n) {
                            const float send = up ? col[i] : col[i + n];
                            const float keep = up ? col[i + n] : col[i];
                            col[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
                        }
                };
                // plain: bits 4, 2, 1, 8 (a half region per result), else 8, 4, 2, 1, then 16
                const int sh = plain ? 1 : 0;
                fold(8, 8 >> sh);
                fold(4, 4 >> sh);
                fold(2, 2 >> sh);
                fold(1, plain ? 8 : 1);
                if (plain) {
                    ci = ((lane & 7) << 1) | h3;
                } else {
                    col[0] += __shfl_xor_sync(0xffffffffu, col[0], 16);
                    ci = lane & 15;
                    act = lane < 16;
                }
                if (act && (ci & 7) < lz) {
                    const int r = T.rz & 0xffffu, z = (int)(T.rz >> 16) + (ci & 7);
                    if (ci < 8) red_add(&P.t1_bar[(long long)r * v + z], col[0]);
                    else red_add(&P.fvo_bar[(long long)z * o + r], col[0]);
                }
            }
        }
        if (!more) break;
        cur = s_item[(k & 1) ^ 1];
    }
    __syncthreads();   // (every warp's waits are behind)
    if (*abortp && tid < kF2mStages + 2) f2m_drain(tid < kF2mStages ? &full[tid] : &tfull[tid - kF2mStages]);
}

}  // namespace tb
