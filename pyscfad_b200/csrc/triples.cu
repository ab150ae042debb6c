// (T) energy and adjoint on B200: planner, layout kernels, chunk epilogue,
// FP64 contraction drivers and the C ABI (include/pyscfad_b200.h).
//
// Reference path replaced: pyscfad/cc/ccsd_t.py:28-192 (forward through
// pyscf's ccsd_t.kernel, backward through ccsd_t_energy_vjp,
// pyscfadlib/pyscfadlib/vjp/cc/ccsd_t_vjp.c:332-497).
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "gemm_fp64.cuh"
#include "tc_f1.cuh"
#include "f2m.cuh"
#include "f2.cuh"
#include "f2e.cuh"
#include "tc_b1.cuh"
#include "lno.cuh"
#include "pyscfad_b200.h"
#include "triples_internal.h"

namespace tb {

// Thread-local error record; every other setting travels with the call
// (Plan, from triples_options), so concurrent calls do not interfere.
static thread_local int g_last_cuda_error = 0;

#define TB_CUDA(call)                                     \
    do {                                                  \
        cudaError_t _e = (call);                          \
        if (_e != cudaSuccess) {                          \
            g_last_cuda_error = (int)_e;                  \
            return TRIPLES_ERR_CUDA;                      \
        }                                                 \
    } while (0)

#define TB_LAUNCH_CHECK() TB_CUDA(cudaGetLastError())

// ---------------------------------------------------------------------------
// optional per-kernel-class timing with CUDA events (on the launch stream)
// ---------------------------------------------------------------------------
enum ProfCat { P_PREP = 0, P_F1, P_F2, P_B1A, P_B1B, P_B1C, P_B1D, P_FOLD, P_LNO, P_LNO_PROJ, P_LNO_ADJ, P_NCAT };
static const char *kProfNames[P_NCAT] = {"prep", "f1_contract", "f2_epilogue",
                                         "b1a_ovvv_grad", "b1b_t2_grad", "b1c_ovoo_grad",
                                         "b1d_t2_ooov_grad", "fold", "lno_tile_fwd", "lno_projection",
                                         "lno_tile_adj"};
struct ProfRec {
    int cat;
    cudaEvent_t a, b;
};
// Profiling records belong to the host thread that enabled them: each
// thread sees only the launches of its own calls.
static thread_local bool g_prof = false;
static thread_local std::vector<ProfRec> g_prof_recs;
static thread_local std::vector<cudaEvent_t> g_event_pool;
static thread_local size_t g_pool_used = 0;

static cudaEvent_t prof_event() {
    if (g_pool_used == g_event_pool.size()) {
        cudaEvent_t e = nullptr;
        cudaEventCreate(&e);
        g_event_pool.push_back(e);
    }
    return g_event_pool[g_pool_used++];
}

template <typename F>
static void prof_wrap(int cat, cudaStream_t st, F &&launch) {
    cudaEvent_t a = nullptr;
    if (g_prof) {
        a = prof_event();
        cudaEventRecord(a, st);
    }
    launch();
    if (g_prof) {
        cudaEvent_t b = prof_event();
        cudaEventRecord(b, st);
        g_prof_recs.push_back({cat, a, b});
    }
}

#define TB_KLAUNCH(cat, ...)                              \
    do {                                                  \
        prof_wrap((cat), st, [&]() { __VA_ARGS__; });     \
        TB_LAUNCH_CHECK();                                \
    } while (0)

// ---------------------------------------------------------------------------
// planning
// ---------------------------------------------------------------------------
static int choose_tv(int o, int tv_request) {
    int tv = tv_request > 0 ? tv_request : 16;
    if (tv > kMaxTv) tv = kMaxTv;
    while (tv > 1 && tv * o > kMaxCols) tv >>= 1;
    int p2 = 1;   // largest power of two <= tv
    while (p2 * 2 <= tv) p2 *= 2;
    return p2;
}

static inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

static void make_chunk(const Dims &d, int A, int B, int C, ChunkDesc &ch) {
    const int blks[3] = {A, B, C};
    auto bsize = [&](int b) { return block_size(d, b); };
    for (int t = 0; t < 3; t++) {
        ch.blk[t] = blks[t];
        ch.nabc[t] = bsize(blks[t]);
        ch.base[t] = block_start(d, blks[t]);
    }
    ch.nperm = 0;
    long long off = 0, swoff = 0;
    const long long o3 = (long long)d.o * d.o * d.o;
    for (int s = 0; s < 6; s++) {
        int ps[3];
        perm_of(s, ps);
        int bx = blks[ps[0]], by = blks[ps[1]], bz = blks[ps[2]];
        bool dup = false;
        for (int t = 0; t < ch.nperm; t++)
            if (ch.pb[t].bx == bx && ch.pb[t].by == by && ch.pb[t].bz == bz) dup = true;
        if (dup) continue;
        PermBlock &pb = ch.pb[ch.nperm++];
        pb.bx = bx; pb.by = by; pb.bz = bz;
        pb.X0 = block_start(d, bx); pb.Tx = bsize(bx);
        pb.Y0 = block_start(d, by); pb.Ty = bsize(by);
        pb.Z0 = block_start(d, bz); pb.Tz = bsize(bz);
        pb.soff = off;
        off += (o3 * pb.Tx * pb.Ty * pb.Tz + 15) / 16 * 16;   // 64 B aligned sub-buffers
        pb.rzp = (d.o * pb.Tz + 7) / 8 * 8;
        pb.swoff = swoff;
        swoff += ((long long)pb.Ty * d.o * pb.Tx * d.o * pb.rzp + 15) / 16 * 16;
    }
}

static long long chunk_wbar_elems(const ChunkDesc &ch, const Dims &d) {
    long long s = 0;
    for (int t = 0; t < ch.nperm; t++)
        s += ((long long)ch.pb[t].Ty * d.o * ch.pb[t].Tx * d.o * ch.pb[t].rzp + 15) / 16 * 16;
    return s;
}

static long long chunk_stage_elems(const ChunkDesc &ch, const Dims &d) {
    long long o3 = (long long)d.o * d.o * d.o, s = 0;
    for (int t = 0; t < ch.nperm; t++) s += (o3 * ch.pb[t].Tx * ch.pb[t].Ty * ch.pb[t].Tz + 15) / 16 * 16;
    return s;
}

// LNO box slots of an occupied triple: every virtual triple of the chunk's blocks once, an even number
static int box_slots(const ChunkDesc &ch) { return (ch.nabc[0] * ch.nabc[1] * ch.nabc[2] + 1) / 2 * 2; }

static int plan_once(int precision, int nocc, int nvir, int packed, int want_grad, Plan &P, int lno,
                     const triples_options *opt, bool vtables, int most_group) {
    if (nocc < 1 || nvir < 1 || nocc > kMaxCols || nvir > 32767) return TRIPLES_ERR_INVALID_ARGUMENT;
    if (precision < TRIPLES_PRECISION_FP64 || precision > TRIPLES_PRECISION_MIXED_BF16)
        return TRIPLES_ERR_INVALID_ARGUMENT;
    if (lno && nocc > kLnoMaxO) return TRIPLES_ERR_UNSUPPORTED;
    P = Plan{};
    if (opt) {
        if (opt->block_size < 0 || opt->accumulation_segment < 0 || opt->chunk_a0 < 0)
            return TRIPLES_ERR_INVALID_ARGUMENT;
        P.a0 = opt->chunk_a0;
        P.a1 = opt->chunk_a1;
        P.kseg = opt->accumulation_segment > 0 ? opt->accumulation_segment : 1;
        if (opt->tile_n != 0 && opt->tile_n != 128 && opt->tile_n != 256) return TRIPLES_ERR_INVALID_ARGUMENT;
        P.f1_bn = opt->tile_n;
    } else {
        P.kseg = 1;
    }
    // W-contraction N tile: up to 256 columns (16 r x 16 z); 128 (a third pipeline
    // stage) where nocc needs no more than 8 r values
    if (P.f1_bn == 0) P.f1_bn = nocc <= 8 ? 128 : 256;
    // r values per tile: nocc over the fewest tiles, evenly, rounded up to even
    {
        const int most = P.f1_bn / 16, nt = (nocc + most - 1) / most;
        P.f1_rt = ((nocc + nt - 1) / nt + 1) / 2 * 2;
    }
    P.lno = lno ? 1 : 0;
    P.prec = precision;
    P.want_grad = want_grad ? 1 : 0;
    P.packed = packed ? 1 : 0;
    Dims &d = P.d;
    d.o = nocc;
    d.v = nvir;
    d.n = nocc + nvir;
    d.Tv = choose_tv(nocc, opt ? opt->block_size : 0);
    if (lno) {
        // halve the block until four FP64 arrays of six times a chunk's box would fit the budget (from
        // nocc 50 on).  The box arrays take a sixth of that; the rule stays because it decides
        // the decomposition, and with it the order of the FP32 sums of the mixed modes.
        const double o3 = (double)nocc * nocc * nocc;
        while (d.Tv > 4 && kLnoArrays * 6.0 * o3 * d.Tv * d.Tv * d.Tv * sizeof(double) > kLnoBudgetBytes) d.Tv >>= 1;
    }
    d.Kp = nvir;
    P.Kp8 = (nvir + 7) / 8 * 8;
    P.Op8 = (nocc + 7) / 8 * 8;
    P.nb = num_blocks(d);
    P.n_ijk = nocc * (nocc + 1) * (nocc + 2) / 6;
    long long maxst = 0, maxwb = 0;
    int maxbox = 1;
    for (int A = 0; A < P.nb; A++)
        for (int B = 0; B <= A; B++)
            for (int C = 0; C <= B; C++) {
                ChunkDesc ch;
                make_chunk(d, A, B, C, ch);
                long long s = chunk_stage_elems(ch, d);
                if (s > maxst) maxst = s;
                long long w = chunk_wbar_elems(ch, d);
                if (w > maxwb) maxwb = w;
                maxbox = std::max(maxbox, box_slots(ch));
            }
    P.stage_elems = (size_t)maxst;
    P.wbar_elems = (size_t)maxwb;
    P.stage_slot = (P.stage_elems + 63) / 64 * 64;   // slots start 256-byte aligned
    P.wbar_slot = (P.wbar_elems + 63) / 64 * 64;
    const bool mixed = precision != TRIPLES_PRECISION_FP64;
    P.stage_bytes = mixed ? sizeof(float) : sizeof(double);

    const size_t o = nocc, v = nvir, Kp = d.Kp;
    const size_t el = sizeof(double);
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t at = off; off = align256(off + bytes); return at; };
    P.off_ctrl = take(kCtrlBytes);
    // FP64 operand layouts: only the FP64 contractions read them (the split
    // operands of the mixed modes are built straight from the inputs)
    if (!mixed) {
        P.off_A1 = take(v * o * v * Kp * el);
        P.off_B1 = take(o * o * v * Kp * el);
        P.off_A2 = take(o * o * v * o * el);
        P.off_B2 = take(v * o * v * o * el);
    } else {
        P.off_A1 = P.off_B1 = P.off_A2 = P.off_B2 = 0;
    }
    if (mixed) {
        P.off_A1h = take(2 * v * o * v * P.Kp8 * 2);
        P.off_B1h = take(2 * o * o * v * P.Kp8 * 2);
        P.off_A2h = take(2 * o * o * v * P.Op8 * 2);
        P.off_B2h = take(2 * v * o * v * P.Op8 * 2);
    }
    // Chunk slots: the chunks of a group run in one launch per kernel, as many
    // as kGroupBytes hold.
    P.group = 1;
    if (!lno && most_group > 1) {
        const size_t chunk = P.stage_slot * P.stage_bytes + (want_grad ? P.wbar_slot * (mixed ? 4 : 8) : 0);
        long long nchunk = 0;
        for (int A = P.a0; A < P.nb && (P.a1 <= 0 || A < P.a1); A++) nchunk += (long long)(A + 1) * (A + 2) / 2;
        const long long fit = (long long)(kGroupBytes / chunk);
        P.group = (int)std::max(1LL, std::min(std::min(fit, nchunk), (long long)most_group));
    }
    P.off_S = take(((P.group - 1) * P.stage_slot + P.stage_elems) * P.stage_bytes);
    if (want_grad) {
        P.off_SW = take(((P.group - 1) * P.wbar_slot + P.wbar_elems) * (mixed ? 4 : 8));
        P.off_GA1 = take(v * o * v * Kp * el);
        P.off_GB1 = take(o * o * v * Kp * el);
        P.off_GA2 = take(o * o * v * o * el);
        P.off_GB2 = take(v * o * v * o * el);
    }
    // FP32 V-term tables of the mixed epilogue; without them it gathers the entries
    P.vtables = vtables && mixed && !lno;
    if (P.vtables) {
        const size_t nb8 = (v + 7) / 8;
        P.off_ot = take(o * o * nb8 * nb8 * 64 * sizeof(float2));
        P.off_tf = take(o * nb8 * 8 * sizeof(float2));
    }
    P.off_ijk = take((size_t)P.n_ijk * 3 * sizeof(int));
    P.off_epart = take((size_t)P.group * P.n_ijk * kMaxPartials * el);
    if (P.lno) {
        // FP64 box arrays: WW (0), PQ (1), Q (2), PW / Zbar (3); the energy alone needs only 0 and 2
        const size_t box = o * o * o * (size_t)maxbox;
        P.off_L[0] = take(box * el);
        P.off_L[2] = take(box * el);
        if (want_grad) {
            P.off_L[1] = take(box * el);
            P.off_L[3] = take(box * el);
        } else {
            P.off_L[1] = P.off_L[0];
            P.off_L[3] = P.off_L[2];
        }
        P.off_lpart = take((size_t)3 * kLnoGrid * el);
    }
    P.total = off;
    return TRIPLES_OK;
}

// vtables: with the V-term tables, which only make a call faster (a problem
// that fits the fixed scratch without them goes without them when it would not
// fit it with them); most_group: chunk slots at most.
int make_plan(int precision, int nocc, int nvir, int packed, int want_grad, Plan &P, int lno,
              const triples_options *opt, bool vtables, int most_group) {
    const int rc = plan_once(precision, nocc, nvir, packed, want_grad, P, lno, opt, vtables, most_group);
    if (rc != TRIPLES_OK || !P.vtables || P.total <= TRIPLES_STATIC_SCRATCH_BYTES) return rc;
    Plan B;
    plan_once(precision, nocc, nvir, packed, want_grad, B, lno, opt, false, 1);
    if (B.total > TRIPLES_STATIC_SCRATCH_BYTES) return rc;
    return plan_once(precision, nocc, nvir, packed, want_grad, P, lno, opt, false, most_group);
}

// The plan with the most chunk slots that fits workspace_bytes; failing one,
// the plan without V-term tables.
int make_plan_for(int precision, int nocc, int nvir, int packed, int want_grad, Plan &P, const triples_options *opt,
                  size_t workspace_bytes) {
    for (int g = kMaxGroup; g >= 1; g--) {
        const int rc = plan_once(precision, nocc, nvir, packed, want_grad, P, 0, opt, true, g);
        if (rc != TRIPLES_OK) return rc;
        if (P.total <= workspace_bytes) return TRIPLES_OK;
        g = std::min(g, P.group);   // fewer slots than asked for: go on from there
    }
    return plan_once(precision, nocc, nvir, packed, want_grad, P, 0, opt, false, 1);
}

// ---------------------------------------------------------------------------
// layout kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long tri_index(int f, int y) {
    return f >= y ? (long long)f * (f + 1) / 2 + y : (long long)y * (y + 1) / 2 + f;
}

// A1[y][p][x][f] = ovvv[p,x,f,y]  (packed: unpacked symmetric [f,y] block)
__global__ void k_prep_A1(const double *__restrict__ ovvv, int packed, Dims d,
                          double *__restrict__ A1) {
    __shared__ double tile[32][33];
    const long long px = blockIdx.z;  // p*v + x
    const int f0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    const long long npair = (long long)d.v * (d.v + 1) / 2;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int f = f0 + r, y = y0 + threadIdx.x;
        double val = 0.0;
        if (f < d.v && y < d.v)
            val = packed ? ovvv[px * npair + tri_index(f, y)] : ovvv[(px * d.v + f) * d.v + y];
        tile[r][threadIdx.x] = val;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int y = y0 + r, f = f0 + threadIdx.x;
        if (y < d.v && f < d.Kp)
            A1[((long long)y * d.o * d.v + px) * d.Kp + f] = tile[threadIdx.x][r];
    }
}

// B1[q][r][z][f] = t2[r,q,z,f]
__global__ void k_prep_B1(const double *__restrict__ t2, Dims d, double *__restrict__ B1) {
    const long long row = blockIdx.x;  // (q*o + r)*v + z
    const int z = row % d.v;
    const int qr = row / d.v;
    const int r = qr % d.o, q = qr / d.o;
    const double *src = t2 + (((long long)r * d.o + q) * d.v + z) * d.v;
    for (int f = threadIdx.x; f < d.Kp; f += blockDim.x)
        B1[row * d.Kp + f] = f < d.v ? src[f] : 0.0;
}

// A2[q][p][x][m] = ovoo[p,x,m,q]
__global__ void k_prep_A2(const double *__restrict__ ovoo, Dims d, double *__restrict__ A2) {
    const long long total = (long long)d.o * d.o * d.v * d.o;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        int m = e % d.o;
        long long t = e / d.o;
        int x = t % d.v;
        t /= d.v;
        int p = t % d.o;
        int q = t / d.o;
        A2[e] = ovoo[(((long long)p * d.v + x) * d.o + m) * d.o + q];
    }
}

// B2[y][r][z][m] = t2[r,m,z,y]
__global__ void k_prep_B2(const double *__restrict__ t2, Dims d, double *__restrict__ B2) {
    const long long total = (long long)d.v * d.o * d.v * d.o;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        int m = e % d.o;
        long long t = e / d.o;
        int z = t % d.v;
        t /= d.v;
        int r = t % d.o;
        int y = t / d.o;
        B2[e] = t2[(((long long)r * d.o + m) * d.v + z) * d.v + y];
    }
}

// ---------------------------------------------------------------------------
// 16-bit split operands for the tensor-core path
// ---------------------------------------------------------------------------
// Occupied representatives i >= j >= k: first the o(o-1)(o-2)/6 with
// i > j > k (combinatorial order: neighbours share i and j, and so the tables and
// lines that they read), then the o(o-1)/2 with i == j > k, as many with
// i > j == k, and the o with i == j == k.
__host__ __device__ inline int n_distinct_ijk(int o) { return o * (o - 1) * (o - 2) / 6; }

__global__ void k_ijk_table(int o, int *ijk) {
    const int n = o * (o + 1) * (o + 2) / 6, nd = n_distinct_ijk(o), np = o * (o - 1) / 2;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        int i, j, k;
        if (r < nd) {
            i = 2;
            while ((i + 1) * i * (i - 1) / 6 <= r) i++;   // largest i with C(i,3) <= r
            int rem = r - i * (i - 1) * (i - 2) / 6;
            j = 1;
            while ((j + 1) * j / 2 <= rem) j++;             // largest j with C(j,2) <= rem
            k = rem - j * (j - 1) / 2;
        } else {
            int t = r - nd;
            const int kind = t < np ? 0 : (t < 2 * np ? 1 : 2);
            t -= kind * np;
            if (kind == 2) {
                i = j = k = t;
            } else {
                int a = 1;
                while ((a + 1) * a / 2 <= t) a++;           // pair a > b, b = t - C(a,2)
                const int b = t - a * (a - 1) / 2;
                i = a;
                j = kind == 0 ? a : b;
                k = b;
            }
        }
        ijk[3 * r] = i;
        ijk[3 * r + 1] = j;
        ijk[3 * r + 2] = k;
    }
}

__global__ void k_absmax(const double *__restrict__ x, long long n, unsigned long long *out) {
    double m = 0.0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x)
        m = fmax(m, fabs(x[e]));
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

__device__ __forceinline__ double pow2_scale(double m) {
    // largest power of two s with m * s < 2^14 (fp16 keeps headroom below 65504)
    if (!(m > 0.0) || !isfinite(m)) return 1.0;
    int e;
    frexp(m, &e);   // m < 2^e
    return ldexp(1.0, 14 - e);
}

__global__ void k_make_scales(Ctrl *ctrl, int scaled) {
    const double a = fmax(__longlong_as_double((long long)ctrl->absmax[0]),
                          __longlong_as_double((long long)ctrl->absmax[1]));
    const double b = __longlong_as_double((long long)ctrl->absmax[2]);
    const double sA = scaled ? pow2_scale(a) : 1.0;
    const double sB = scaled ? pow2_scale(b) : 1.0;
    ctrl->scale[0] = sA;
    ctrl->scale[1] = sB;
    ctrl->out_scale = (float)(1.0 / (sA * sB));
}

// What the small per-chunk kernels need: the virtual ranges for the Wbar scale,
// the energy partials of the epilogue.
struct ChunkAux {
    Ctrl *ctrl;
    ChunkSlot *slot;
    const double *mo_e;
    const double *e_part;
    double ybar;
    int o, a0, na, b0, nb, c0, nc, n_part;
    int scaled, lno;
};

// Per-chunk power-of-two scale for the split Wbar, from a bound that needs no
// pass over Wbar:  |Wbar| <= 2|ybar| (144 max|w| + 36 max|v|) / min|D| over the
// chunk (|Z| <= 12 max|X|, |X| <= 6 max|w| + 3 max|v|, |R WW| <= 72 max|w|,
// orbit weight <= 2).  Resets the running max |w| for the slot's next chunk.
// One 32-thread block per chunk.
template <typename JOBS>
__global__ void k_chunk_scale(const __grid_constant__ JOBS J) {
    const ChunkAux &A = J.job[JOBS::kOne ? 0 : blockIdx.x];
    const Ctrl *ctrl = A.ctrl;
    const int o = A.o;
    __shared__ double s_min[3], s_maxo;
    const double inf = 1e300;
    if (threadIdx.x < 4) {
        double m = (threadIdx.x < 3) ? inf : -inf;
        const int st = threadIdx.x == 0 ? A.a0 : (threadIdx.x == 1 ? A.b0 : A.c0);
        const int n = threadIdx.x == 0 ? A.na : (threadIdx.x == 1 ? A.nb : A.nc);
        if (threadIdx.x < 3) {
            for (int t = 0; t < n; t++) m = fmin(m, A.mo_e[o + st + t]);
            s_min[threadIdx.x] = m;
        } else {
            for (int t = 0; t < o; t++) m = fmax(m, A.mo_e[t]);
            s_maxo = m;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double dmin = s_min[0] + s_min[1] + s_min[2] - 3.0 * s_maxo;
        const double mw = (double)__uint_as_float(A.slot->wmax_bits);
        const double mv = __longlong_as_double((long long)ctrl->absmax[3]) * __longlong_as_double((long long)ctrl->absmax[4]) +
                          __longlong_as_double((long long)ctrl->absmax[2]) * __longlong_as_double((long long)ctrl->absmax[5]);
        // |wbar| <= 6 |WWbar|; with the LNO projector (row / column abs sums nr, nc)
        // WWbar = P^T(ybar Q / 3) + r3^T(ybar P(WW) / (3 D)), |Q| <= 12 (6 mw + 3 mv) / dmin;
        // nr = nc = 1 is the canonical bound
        const double nr = A.lno ? ctrl->lno_norm[0] : 1.0, ncl = A.lno ? ctrl->lno_norm[1] : 1.0;
        double bound = 2.0 * fabs(A.ybar) * (72.0 * (nr + ncl) * mw + 36.0 * nr * mv) / (dmin > 1e-300 ? dmin : 1e-300);
        A.slot->wscale = A.scaled ? pow2_scale(bound) : 1.0;
        A.slot->wmax_bits = 0u;
    }
}

// The chunks' energy partials, each in a fixed order; the epilogue's item
// counter goes back to zero for its next launch.  Chunks of one problem (a
// Group) are added by one block, chunk after chunk; those of a Table belong to
// different problems, one block each.
template <typename JOBS>
__global__ void k_energy_sum(const __grid_constant__ JOBS J, int per_block) {
    for (int c = blockIdx.x * per_block; c < (int)(blockIdx.x + 1) * per_block; c++) {
        const ChunkAux &A = J.job[JOBS::kOne ? 0 : c];
        energy_sum_body(A.e_part, A.n_part, &A.ctrl->e_acc);
        if (threadIdx.x == 0) A.slot->ticket = 0u;
        __syncthreads();
    }
}

template <typename H>
__device__ __forceinline__ void split16(double xs, H &hi, H &lo);
template <>
__device__ __forceinline__ void split16<__half>(double xs, __half &hi, __half &lo) {
    hi = __double2half(xs);
    lo = __double2half(xs - (double)__half2float(hi));
}
template <>
__device__ __forceinline__ void split16<__nv_bfloat16>(double xs, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
    hi = __double2bfloat16(xs);
    lo = __double2bfloat16(xs - (double)__bfloat162float(hi));
}

// A1h[h][y][p][x][f] = split(ovvv[p,x,f,y] * sA), f < Kp8 (zero beyond v)
// max abs row sum and max abs column sum of the LNO projector mat[o,o]
__global__ void k_lno_mat_norms(const double *__restrict__ mat, int o, Ctrl *ctrl) {
    __shared__ double s_r[kLnoMaxO], s_c[kLnoMaxO];
    for (int i = threadIdx.x; i < o; i += blockDim.x) {
        double r = 0.0, c = 0.0;
        for (int k = 0; k < o; k++) {
            r += fabs(mat[i * o + k]);
            c += fabs(mat[k * o + i]);
        }
        s_r[i] = r;
        s_c[i] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double mr = 0.0, mc = 0.0;
        for (int i = 0; i < o; i++) {
            mr = fmax(mr, s_r[i]);
            mc = fmax(mc, s_c[i]);
        }
        ctrl->lno_norm[0] = mr;
        ctrl->lno_norm[1] = mc;
    }
}

// Tile (row block fb >= column block yb) of a triangle of nb x nb blocks, for each px
__device__ __forceinline__ void tri_tile(long long t, int nb, long long &px, int &fb, int &yb) {
    const int per = nb * (nb + 1) / 2;
    px = t / per;
    const int e = (int)(t - px * per);
    fb = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
    while (fb * (fb + 1) / 2 > e) fb--;
    while ((fb + 1) * (fb + 2) / 2 <= e) fb++;
    yb = e - fb * (fb + 1) / 2;
}

// The same operand from the packed layout: a block reads a 64 x 64 tile f0 >= y0 of
// the triangle of one (p, x) once, rows of 512 bytes, and writes it both ways.
// Bound by HBM (nocc 40 nvir 360: 5.9 to 4.9 ms;
// with 32 x 32 tiles of both triangles half of the reads ran down columns).
template <typename H>
__global__ void __launch_bounds__(256) k_prep_A1h_packed(const double *__restrict__ ovvv, Dims d, int Kp8,
                                                         const Ctrl *ctrl, H *__restrict__ out) {
    __shared__ double tile[64][65];
    int fb, yb;
    long long px;
    tri_tile(blockIdx.x, (Kp8 + 63) / 64, px, fb, yb);
    const int f0 = fb * 64, y0 = yb * 64, lane = threadIdx.x & 63, row = threadIdx.x >> 6;
    const double sA = ctrl->scale[0];
    const double *src = ovvv + px * ((long long)d.v * (d.v + 1) / 2);
#pragma unroll 4
    for (int r = row; r < 64; r += 4) {
        const int f = f0 + r, y = y0 + lane;
        double val = 0.0;
        if (f < d.v && y <= f) {
            val = src[(long long)f * (f + 1) / 2 + y] * sA;
            if (fb == yb) tile[lane][r] = val;   // the diagonal tile holds both triangles
        }
        if (fb != yb || y <= f || f >= d.v) tile[r][lane] = val;
    }
    __syncthreads();
    const long long half = (long long)d.v * d.o * d.v * Kp8;
    for (int pass = 0; pass < (fb == yb ? 1 : 2); pass++) {
        // rows of the first pass are y with f along the lanes, of the second f with y along them
        const int a0 = pass ? f0 : y0, b0 = pass ? y0 : f0;
        const int b = b0 + lane;
#pragma unroll 4
        for (int r = row; r < 64; r += 4) {
            const int a = a0 + r;
            if (a < d.v && b < Kp8) {
                H hi, lo;
                split16<H>(pass ? tile[r][lane] : tile[lane][r], hi, lo);
                const long long e = ((long long)a * d.o * d.v + px) * Kp8 + b;
                out[e] = hi;
                out[half + e] = lo;
            }
        }
    }
}

template <typename H>
__global__ void k_prep_A1h(const double *__restrict__ ovvv, Dims d, int Kp8, const Ctrl *ctrl,
                           H *__restrict__ out) {
    __shared__ double tile[32][33];
    const long long px = blockIdx.z;
    const int f0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    const double sA = ctrl->scale[0];
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int f = f0 + r, y = y0 + threadIdx.x;
        double val = 0.0;
        if (f < d.v && y < d.v)
            val = ovvv[(px * d.v + f) * d.v + y];
        tile[r][threadIdx.x] = val;
    }
    __syncthreads();
    const long long half = (long long)d.v * d.o * d.v * Kp8;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int y = y0 + r, f = f0 + threadIdx.x;
        if (y < d.v && f < Kp8) {
            H hi, lo;
            split16<H>(tile[threadIdx.x][r] * sA, hi, lo);
            const long long e = ((long long)y * d.o * d.v + px) * Kp8 + f;
            out[e] = hi;
            out[half + e] = lo;
        }
    }
}

// B1h[h][q][r][z][f] = split(t2[r,q,z,f] * sB)
template <typename H>
__global__ void k_prep_B1h(const double *__restrict__ t2, Dims d, int Kp8, const Ctrl *ctrl,
                           H *__restrict__ out) {
    const long long row = blockIdx.x;  // (q*o + r)*v + z
    const int z = row % d.v;
    const int qr = row / d.v;
    const int r = qr % d.o, q = qr / d.o;
    const double *src = t2 + (((long long)r * d.o + q) * d.v + z) * d.v;
    const double sB = ctrl->scale[1];
    const long long half = (long long)d.o * d.o * d.v * Kp8;
    for (int f = threadIdx.x; f < Kp8; f += blockDim.x) {
        H hi, lo;
        split16<H>(f < d.v ? src[f] * sB : 0.0, hi, lo);
        out[row * Kp8 + f] = hi;
        out[half + row * Kp8 + f] = lo;
    }
}

// A2h[h][q][p][x][m] = split(-ovoo[p,x,m,q] * sA), m < Op8
template <typename H>
__global__ void k_prep_A2h(const double *__restrict__ ovoo, Dims d, int Op8, const Ctrl *ctrl,
                           H *__restrict__ out) {
    const long long total = (long long)d.o * d.o * d.v * Op8;
    const double sA = ctrl->scale[0];
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        int m = e % Op8;
        long long t = e / Op8;
        int x = t % d.v;
        t /= d.v;
        int p = t % d.o;
        int q = t / d.o;
        double val = m < d.o ? -ovoo[(((long long)p * d.v + x) * d.o + m) * d.o + q] * sA : 0.0;
        H hi, lo;
        split16<H>(val, hi, lo);
        out[e] = hi;
        out[total + e] = lo;
    }
}

// The tile of a block in an (m, y) transposition for each (r, z): 64 m by 64 y
__device__ __forceinline__ void rz_tile(const Dims &d, int nm, int &r, int &z, int &m0, int &y0) {
    const int nmb = (nm + 63) / 64, nyb = (d.v + 63) / 64;
    long long t = blockIdx.x;
    m0 = (int)(t % nmb) * 64;
    t /= nmb;
    y0 = (int)(t % nyb) * 64;
    t /= nyb;
    z = (int)(t % d.v);
    r = (int)(t / d.v);
}

// B2h[h][y][r][z][m] = split(t2[r,m,z,y] * sB), m < Op8.  Through a tile in shared
// memory, so that reads run along y and writes along m: bound by HBM (a thread per
// output element read sectors for one value each, nocc 40 nvir 360: 4.5 ms; now 0.8).
template <typename H>
__global__ void __launch_bounds__(256) k_prep_B2h(const double *__restrict__ t2, Dims d, int Op8, const Ctrl *ctrl,
                                                  H *__restrict__ out) {
    __shared__ double tile[64][65];
    int r, z, m0, y0;
    rz_tile(d, Op8, r, z, m0, y0);
    const int lane = threadIdx.x & 63, row = threadIdx.x >> 6;
    const double sB = ctrl->scale[1];
    const int mn = min(64, Op8 - m0), yn = min(64, d.v - y0);
    for (int k = row; k < mn; k += 4) {
        const int m = m0 + k;
        tile[k][lane] = (m < d.o && lane < yn) ? t2[(((long long)r * d.o + m) * d.v + z) * d.v + y0 + lane] * sB : 0.0;
    }
    __syncthreads();
    const long long half = (long long)d.v * d.o * d.v * Op8;
    for (int e = threadIdx.x; e < yn * mn; e += 256) {
        const int k = e % mn, yl = e / mn;
        H hi, lo;
        split16<H>(tile[k][yl], hi, lo);
        const long long at = (((long long)(y0 + yl) * d.o + r) * d.v + z) * Op8 + m0 + k;
        out[at] = hi;
        out[half + at] = lo;
    }
}

// ---------------------------------------------------------------------------
// FP64 contraction kernels (one GEMM problem per blockIdx.z)
// ---------------------------------------------------------------------------
struct GemmLaunch {
    Dims d;
    int n;                       // chunks
    ChunkDesc ch[kMaxGroup];
    double *S[kMaxGroup];        // staging (F1)
    double *SW[kMaxGroup];       // Wbar (adjoint kinds)
    int zstart[kMaxGroup + 1];   // GEMM problems (blockIdx.z) chunk after chunk,
    int cum[kMaxGroup][7];       // and within a chunk ordering after ordering
    int nmt, nslice;             // M tiles and K slices of blockIdx.x
    const double *A1, *B1, *A2, *B2;
    double *G;                   // gradient target
};

// The five contractions of a chunk.  F1: S_tau[p][q][y][x][r][z] = W for all
// (tau, y, q); the adjoint kinds with Wbar[y][p][x][q][r][z] in L.S:
//   B1A  ovvv: G_A1[y][p][x][f] += sum_{q,r,z} Wbar B1[q][r][z][f]   problems (tau, y)
//   B1B  t2:   G_B1[q][r][z][f] += sum_{y,p,x} Wbar A1[y][p][x][f]   problems (tau, q)
//   B1C  ovoo: G_A2[q][p][x][m] -= sum_{y,r,z} Wbar B2[y][r][z][m]   problems (tau, q)
//   B1D  t2:   G_B2[y][r][z][m] -= sum_{q,p,x} Wbar A2[q][p][x][m]   problems (tau, y)
// Orderings that share a block write the same rows in B1B and B1C, and K may
// be cut into slices, so the adjoint kinds add atomically.
enum GemmKind { GK_F1 = 0, GK_B1A, GK_B1B, GK_B1C, GK_B1D };
__host__ __device__ constexpr bool gemm_kfa(int kind) { return kind == GK_F1 || kind == GK_B1A || kind == GK_B1C; }
__host__ __device__ constexpr bool gemm_kfb(int kind) { return kind == GK_F1; }

template <int KIND, int BM, int BN>
__global__ void __launch_bounds__(kGThreads) k_chunk_fp64(const __grid_constant__ GemmLaunch L) {
    extern __shared__ __align__(16) double gemm_smem[];
    int c = 0, t = 0;
    while (c + 1 < L.n && (int)blockIdx.z >= L.zstart[c + 1]) c++;
    const int b = (int)blockIdx.z - L.zstart[c];
    while (t + 1 < L.ch[c].nperm && b >= L.cum[c][t + 1]) t++;
    const PermBlock &pb = L.ch[c].pb[t];
    const Dims &d = L.d;
    const int o = d.o, v = d.v, Kp = d.Kp, rem = b - L.cum[c][t];
    const double *SW = L.SW[c];
    const long long oTz = (long long)o * pb.Tz;
    // Wbar strides
    const long long s_q = pb.rzp, s_x = (long long)o * pb.rzp, s_p = (long long)pb.Tx * s_x, s_y = (long long)o * s_p;
    const long long ovK = (long long)o * v * Kp, vK = (long long)v * Kp, ovo = (long long)o * v * o, vo = (long long)v * o;
    GemmArgs g;
    g.K2 = 0;
    g.cn = map1(1);
    g.alpha = 1.0;
    g.alpha2 = 0.0;
    g.atomic = 1;
    if (KIND == GK_F1) {
        const int y = rem / o, q = rem % o;
        const long long yg = pb.Y0 + y;
        g.M = o * pb.Tx;
        g.N = o * pb.Tz;
        g.K = v;
        g.K2 = o;
        g.A = GOp{L.A1 + yg * ovK + (long long)pb.X0 * Kp, map2(pb.Tx, Kp, vK), map1(1)};
        g.B = GOp{L.B1 + q * ovK + (long long)pb.Z0 * Kp, map2(pb.Tz, Kp, vK), map1(1)};
        g.A2 = GOp{L.A2 + q * ovo + (long long)pb.X0 * o, map2(pb.Tx, o, vo), map1(1)};
        g.B2 = GOp{L.B2 + yg * ovo + (long long)pb.Z0 * o, map2(pb.Tz, o, vo), map1(1)};
        // staging in 8 x 8 x 8 blocks (StageRow, rows not exchanged)
        const int ex = min(8, pb.Tx), ey = min(8, pb.Ty), ez = min(8, pb.Tz), nx = pb.Tx / ex, nz = pb.Tz / ez;
        const long long es = ex * ey * ez, rs = (long long)pb.Tx * pb.Ty * pb.Tz;
        g.C = L.S[c] + pb.soff + (long long)q * o * rs + (y / ey) * nx * nz * es + (y % ey) * (ex * ez);
        g.cm = map3(ex, nx, ez, nz * es, (long long)o * o * rs);
        g.cn = map3(ez, nz, 1, es, rs);
        g.alpha2 = -1.0;
        g.atomic = 0;
    } else if (KIND == GK_B1A) {
        g.M = o * pb.Tx;
        g.N = v;
        g.K = o * o * pb.Tz;
        g.A = GOp{SW + pb.swoff + rem * s_y, map2(pb.Tx, s_x, s_p), map2((int)oTz, 1, s_q)};
        g.B = GOp{L.B1 + (long long)pb.Z0 * Kp, map1(1), map3(pb.Tz, o, Kp, vK, ovK)};
        g.C = L.G + ((long long)pb.Y0 + rem) * ovK + (long long)pb.X0 * Kp;
        g.cm = map2(pb.Tx, Kp, vK);
    } else if (KIND == GK_B1B) {
        g.M = o * pb.Tz;
        g.N = v;
        g.K = pb.Ty * o * pb.Tx;
        g.A = GOp{SW + pb.swoff + rem * s_q, map1(1), map3(pb.Tx, o, s_x, s_p, s_y)};
        g.B = GOp{L.A1 + (long long)pb.Y0 * ovK + (long long)pb.X0 * Kp, map1(1), map3(pb.Tx, o, Kp, vK, ovK)};
        g.C = L.G + rem * ovK + (long long)pb.Z0 * Kp;
        g.cm = map2(pb.Tz, Kp, vK);
    } else if (KIND == GK_B1C) {
        g.M = o * pb.Tx;
        g.N = o;
        g.K = pb.Ty * o * pb.Tz;
        g.A = GOp{SW + pb.swoff + rem * s_q, map2(pb.Tx, s_x, s_p), map2((int)oTz, 1, s_y)};
        g.B = GOp{L.B2 + (long long)pb.Y0 * ovo + (long long)pb.Z0 * o, map1(1), map3(pb.Tz, o, o, vo, ovo)};
        g.C = L.G + rem * ovo + (long long)pb.X0 * o;
        g.cm = map2(pb.Tx, o, vo);
        g.alpha = -1.0;
    } else {
        g.M = o * pb.Tz;
        g.N = o;
        g.K = o * o * pb.Tx;
        g.A = GOp{SW + pb.swoff + rem * s_y, map1(1), map3(pb.Tx, o, s_x, s_p, s_q)};
        g.B = GOp{L.A2 + (long long)pb.X0 * o, map1(1), map3(pb.Tx, o, o, vo, ovo)};
        g.C = L.G + ((long long)pb.Y0 + rem) * ovo + (long long)pb.Z0 * o;
        g.cm = map2(pb.Tz, o, vo);
        g.alpha = -1.0;
    }
    const int m0 = (blockIdx.x % L.nmt) * BM, n0 = blockIdx.y * BN;
    if (m0 >= g.M || n0 >= g.N) return;
    gemm_fp64_tile<BM, BN, gemm_kfa(KIND), gemm_kfb(KIND)>(g, m0, n0, blockIdx.x / L.nmt, L.nslice, gemm_smem);
}

// ---------------------------------------------------------------------------
// gradient fold back to the reference layouts
// ---------------------------------------------------------------------------
// full ovvv_bar[p,x,f,y] = G_A1[y][p][x][f]
__global__ void k_fold_ovvv_full(const double *__restrict__ GA1, Dims d, double *__restrict__ out) {
    __shared__ double tile[32][33];
    const long long px = blockIdx.z;
    const int y0 = blockIdx.x * 32, f0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int y = y0 + r, f = f0 + threadIdx.x;
        tile[r][threadIdx.x] = (y < d.v && f < d.v) ? GA1[((long long)y * d.o * d.v + px) * d.Kp + f] : 0.0;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int f = f0 + r, y = y0 + threadIdx.x;
        if (f < d.v && y < d.v) out[(px * d.v + f) * d.v + y] = tile[threadIdx.x][r];
    }
}

// packed ovvv_bar[p,x,tri(f,y)] = G[f,y] + G[y,f] (f != y), G[f,f]; G[f,y] = G_A1[y][p][x][f]
// (pyscfad/cc/ccsd_t.py:184-191).  A block takes a 64 x 64 tile f0 >= y0 of one
// (p, x): rows of 512 bytes of both triangles, G[f,y] transposed in shared
// memory.  Bound by HBM.  One element per thread, without tiles, read G[f,y]
// with a lane per y (nocc 40 nvir 360: 22 to 4.8 ms).
__global__ void __launch_bounds__(256) k_fold_ovvv_packed(const double *__restrict__ GA1, Dims d,
                                                          double *__restrict__ out) {
    __shared__ double tile[64][65];
    int fb, yb;
    long long px;
    tri_tile(blockIdx.x, (d.v + 63) / 64, px, fb, yb);
    const int f0 = fb * 64, y0 = yb * 64, lane = threadIdx.x & 63, row = threadIdx.x >> 6;
    const long long sy = (long long)d.o * d.v * d.Kp, npair = (long long)d.v * (d.v + 1) / 2;
    const double *src = GA1 + px * d.Kp;
#pragma unroll 4
    for (int r = row; r < 64; r += 4) {
        const int y = y0 + r, f = f0 + lane;
        tile[r][lane] = (y < d.v && f < d.v) ? src[y * sy + f] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int r = row; r < 64; r += 4) {
        const int f = f0 + r, y = y0 + lane;
        if (f < d.v && y <= f) {
            const double val = tile[lane][r] + (f != y ? src[f * sy + y] : 0.0);
            out[px * npair + (long long)f * (f + 1) / 2 + y] = val;
        }
    }
}

// t2_bar[r,q,z,f] += G_B1[q][r][z][f] + G_B2[f][r][z][q].  G_B2 through a tile in
// shared memory: read along q, added along f (nocc 40 nvir 360: 5.1 to 1.5 ms).
__global__ void __launch_bounds__(256) k_fold_t2(const double *__restrict__ GB1, const double *__restrict__ GB2, Dims d,
                                                 double *__restrict__ t2_bar) {
    __shared__ double tile[64][65];
    int r, z, q0, f0;
    rz_tile(d, d.o, r, z, q0, f0);
    const int lane = threadIdx.x & 63, row = threadIdx.x >> 6;
    const int qn = min(64, d.o - q0), fn = min(64, d.v - f0);
    for (int e = threadIdx.x; e < fn * qn; e += 256) {
        const int k = e % qn, fl = e / qn;
        tile[k][fl] = GB2[(((long long)(f0 + fl) * d.o + r) * d.v + z) * d.o + q0 + k];
    }
    __syncthreads();
    if (lane < fn)
        for (int k = row; k < qn; k += 4) {
            const int q = q0 + k, f = f0 + lane;
            t2_bar[(((long long)r * d.o + q) * d.v + z) * d.v + f] +=
                GB1[(((long long)q * d.o + r) * d.v + z) * d.Kp + f] + tile[k][lane];
        }
}

// ovoo_bar[p,x,m,q] = G_A2[q][p][x][m]
__global__ void k_fold_ovoo(const double *__restrict__ GA2, Dims d, double *__restrict__ out) {
    const long long total = (long long)d.o * d.v * d.o * d.o;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int q = e % d.o;
        long long t = e / d.o;
        const int m = t % d.o;
        t /= d.o;
        const int x = t % d.v;
        const int p = t / d.v;
        out[e] = GA2[(((long long)q * d.o + p) * d.v + x) * d.o + m];
    }
}

__global__ void k_copy_scalar(const double *src, double *dst) { dst[0] = src[0]; }

// ---------------------------------------------------------------------------
// driver
// ---------------------------------------------------------------------------
// 64 x 64 tiles of the triangle of an n x n block, for each of `count` (p, x)
static inline unsigned tri_grid(int n, size_t count) {
    const int nb = (n + 63) / 64;
    return (unsigned)((size_t)nb * (nb + 1) / 2 * count);
}

// 64 x 64 tiles of (m < nm, y < nvir) for each (r, z)
static inline unsigned rz_grid(const Dims &d, int nm) {
    return (unsigned)((size_t)((nm + 63) / 64) * ((d.v + 63) / 64) * d.o * d.v);
}

static inline unsigned grid1d(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    if (b > 148 * 64) b = 148 * 64;
    if (b < 1) b = 1;
    return (unsigned)b;
}

// ---- tensor maps (driver entry point fetched through the runtime) ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn lookup_encode_fn() {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
        return (EncodeTiledFn)ptr;
    return nullptr;
}

static EncodeTiledFn get_encode_fn() {
    static const EncodeTiledFn fn = lookup_encode_fn();   // initialised once, thread-safe
    return fn;
}

// 5-D map over a dense 16-bit array of dims[0] (innermost) to dims[4], 128B swizzle or none.
static int make_tmap5(CUtensorMap *tm, void *base, bool bf16, const uint64_t dims[5], const uint32_t box[5],
                      bool swizzle = true) {
    EncodeTiledFn enc = get_encode_fn();
    if (!enc) return TRIPLES_ERR_UNSUPPORTED;
    cuuint64_t gdim[5], gstr[4];
    uint64_t stride = 2;
    for (int i = 0; i < 5; i++) {
        gdim[i] = dims[i];
        if (i < 4) {
            stride *= dims[i];
            gstr[i] = stride;
        }
    }
    cuuint32_t bx[5], es[5] = {1, 1, 1, 1, 1};
    for (int i = 0; i < 5; i++) bx[i] = box[i];
    CUresult r = enc(tm, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, base, gdim,
                     gstr, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TRIPLES_OK : TRIPLES_ERR_CUDA;
}

// 5-D map over S_tau (FP32) as [p][q][r][y block, x block, z block][y][64], used
// by the W-contraction epilogue to store 32 x 32 pieces of full (x, z) blocks.
static int make_tmap_stage(CUtensorMap *tm, float *base, int o, int Ty) {
    EncodeTiledFn enc = get_encode_fn();
    if (!enc) return TRIPLES_ERR_UNSUPPORTED;
    const int ey = Ty < 8 ? Ty : 8;
    const cuuint64_t gdim[5] = {(cuuint64_t)ey * 64, (cuuint64_t)(Ty / ey) * 4, (cuuint64_t)o, (cuuint64_t)o, (cuuint64_t)o};
    cuuint64_t gstr[4];
    gstr[0] = gdim[0] * sizeof(float);
    for (int i = 1; i < 4; i++) gstr[i] = gstr[i - 1] * gdim[i];
    const cuuint32_t box[5] = {64, 4, 2, 1, 2}, es[5] = {1, 1, 1, 1, 1};
    CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, base, gdim, gstr, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TRIPLES_OK : TRIPLES_ERR_CUDA;
}

// SM count of the current device (cached per device; the first writers
// store the same value, so relaxed atomics suffice).
constexpr int kMaxDev = 64;
static std::atomic<int> g_num_sms[kMaxDev];

static int num_sms() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return 148;
    int n = g_num_sms[dev].load(std::memory_order_relaxed);
    if (n <= 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        g_num_sms[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// ---------------------------------------------------------------------------
// FP64 GEMM launches: tile and K-slice choice
// ---------------------------------------------------------------------------
// Of the tile shapes a contraction is built for, the one with the least padded
// area, the smaller ones charged for the operand traffic they add.  With too
// few tiles for two per SM, K is cut into slices of at least four K tiles
// (atomic adds only).
struct GemmTile {
    int bm, bn, nslice;
};

static GemmTile gemm_tile(long long M, long long N, long long K, long long batches, bool slices) {
    static const struct { int bm, bn; double w; } shapes[] = {
        {128, 128, 1.0}, {128, 64, 1.08}, {64, 64, 1.15}, {128, 48, 1.25}, {128, 32, 1.35}, {128, 16, 1.6}};
    GemmTile best{128, 128, 1};
    double cost = -1.0;
    for (const auto &s : shapes) {
        const double c = (double)((M + s.bm - 1) / s.bm * s.bm) * ((N + s.bn - 1) / s.bn * s.bn) * s.w;
        if (cost < 0 || c < cost) {
            cost = c;
            best.bm = s.bm;
            best.bn = s.bn;
        }
    }
    const long long blocks = (M + best.bm - 1) / best.bm * ((N + best.bn - 1) / best.bn) * batches;
    const long long want = 2 * num_sms(), most = (K + 4 * kGBK - 1) / (4 * kGBK);
    if (slices && blocks < want) {
        const long long n = (want + blocks - 1) / blocks;
        best.nslice = (int)(n < most ? n : most);
        if (best.nslice < 1) best.nslice = 1;
    }
    return best;
}

// f(BM, BN) as compile-time constants for a tile of gemm_tile
template <typename F>
static int gemm_dispatch(const GemmTile &t, F &&f) {
    using std::integral_constant;
    if (t.bn == 128) return f(integral_constant<int, 128>{}, integral_constant<int, 128>{});
    if (t.bn == 64 && t.bm == 128) return f(integral_constant<int, 128>{}, integral_constant<int, 64>{});
    if (t.bn == 64) return f(integral_constant<int, 64>{}, integral_constant<int, 64>{});
    if (t.bn == 48) return f(integral_constant<int, 128>{}, integral_constant<int, 48>{});
    if (t.bn == 32) return f(integral_constant<int, 128>{}, integral_constant<int, 32>{});
    return f(integral_constant<int, 128>{}, integral_constant<int, 16>{});
}

// Shared memory above the default 48 KB needs an opt-in per kernel and device
// (the attribute call is idempotent and cheap next to a launch).  `bytes` is the same
// in every call for a kernel: host threads share the limit.
template <typename K>
static int smem_optin(K kernel, size_t bytes) {
    TB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return TRIPLES_OK;
}

// One contraction of the launch's chunks; tiles from the largest M, N and K.
template <int KIND>
static int chunk_gemm(cudaStream_t st, int cat, GemmLaunch &L) {
    const long long o = L.d.o, v = L.d.v;
    long long M = 0, N = 0, K = 0;
    L.zstart[0] = 0;
    for (int c = 0; c < L.n; c++) {
        L.cum[c][0] = 0;
        for (int t = 0; t < L.ch[c].nperm; t++) {
            const PermBlock &pb = L.ch[c].pb[t];
            const long long m = o * (KIND == GK_F1 || KIND == GK_B1A || KIND == GK_B1C ? pb.Tx : pb.Tz);
            const long long n = KIND == GK_F1 ? o * pb.Tz : (KIND == GK_B1A || KIND == GK_B1B ? v : o);
            const long long k = KIND == GK_F1 ? v
                                : KIND == GK_B1A ? o * o * pb.Tz
                                : KIND == GK_B1B ? o * pb.Ty * pb.Tx
                                : KIND == GK_B1C ? o * pb.Ty * pb.Tz
                                                 : o * o * pb.Tx;
            M = std::max(M, m);
            N = std::max(N, n);
            K = std::max(K, k);
            L.cum[c][t + 1] = L.cum[c][t] + (KIND == GK_F1 ? pb.Ty * L.d.o
                                             : KIND == GK_B1A || KIND == GK_B1D ? pb.Ty : L.d.o);
        }
        L.zstart[c + 1] = L.zstart[c] + L.cum[c][L.ch[c].nperm];
    }
    const GemmTile tile = gemm_tile(M, N, K, L.zstart[L.n], KIND != GK_F1);
    return gemm_dispatch(tile, [&](auto bm, auto bn) -> int {
        constexpr int BM = decltype(bm)::value, BN = decltype(bn)::value;
        using C = GemmCfg<BM, BN, gemm_kfa(KIND), gemm_kfb(KIND)>;
        const int rc = smem_optin(k_chunk_fp64<KIND, BM, BN>, C::SMEM);
        if (rc != TRIPLES_OK) return rc;
        L.nmt = (int)((M + BM - 1) / BM);
        L.nslice = tile.nslice;
        const dim3 grid((unsigned)(L.nmt * L.nslice), (unsigned)((N + BN - 1) / BN), (unsigned)L.zstart[L.n]);
        TB_KLAUNCH(cat, (k_chunk_fp64<KIND, BM, BN><<<grid, kGThreads, C::SMEM, st>>>(L)));
        return TRIPLES_OK;
    });
}

// plain FP64 GEMM through the multi-index tile (DF factor products)
template <int BM, int BN, bool KFA, bool KFB>
__global__ void __launch_bounds__(kGThreads) k_gemm_plain(const __grid_constant__ GemmArgs g) {
    extern __shared__ __align__(16) double gemm_smem[];
    gemm_fp64_tile<BM, BN, KFA, KFB>(g, blockIdx.x * BM, blockIdx.y * BN, 0, 1, gemm_smem);
}

// C[m*cms + n*cns] = sum_k A[m*ams + k*aks] B[n*bms + k*bks]; KFA / KFB: the
// operand is contiguous along k
template <bool KFA, bool KFB>
static int gemm_plain(cudaStream_t st, int M, int N, int K, const double *A, long long ams, long long aks,
                      const double *B, long long bms, long long bks, double *C, long long cms, long long cns) {
    GemmArgs g;
    g.M = M;
    g.N = N;
    g.K = K;
    g.K2 = 0;
    g.A = GOp{A, map1(ams), map1(aks)};
    g.B = GOp{B, map1(bms), map1(bks)};
    g.A2 = g.A;
    g.B2 = g.B;
    g.C = C;
    g.cm = map1(cms);
    g.cn = map1(cns);
    g.alpha = 1.0;
    g.alpha2 = 0.0;
    g.atomic = 0;
    constexpr int BM = 128, BN = 128;
    using Cfg = GemmCfg<BM, BN, KFA, KFB>;
    const dim3 grid((unsigned)((M + BM - 1) / BM), (unsigned)((N + BN - 1) / BN));
    if (grid.y > 65535) return TRIPLES_ERR_UNSUPPORTED;
    const int rc = smem_optin(k_gemm_plain<BM, BN, KFA, KFB>, Cfg::SMEM);
    if (rc != TRIPLES_OK) return rc;
    TB_KLAUNCH(P_PREP, (k_gemm_plain<BM, BN, KFA, KFB><<<grid, kGThreads, Cfg::SMEM, st>>>(g)));
    return TRIPLES_OK;
}

// One-time set-up per device and kind of work (shared-memory opt-ins), under a
// lock so that host threads making their first
// call at the same time do it once.  Assumes the device's primary context
// lives as long as the process (a cudaDeviceReset would need it again).
enum InitKind { INIT_F2_F32 = 0, INIT_F2_F64, INIT_TC, INIT_LNO, INIT_LNO64, INIT_NKINDS };
static std::mutex g_init_mu;
static bool g_init_done[kMaxDev][INIT_NKINDS];

template <typename F>
static int once_per_device(int kind, F &&setup) {
    int dev = 0;
    TB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDev) return TRIPLES_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lk(g_init_mu);
    if (g_init_done[dev][kind]) return TRIPLES_OK;
    const int rc = setup();
    if (rc == TRIPLES_OK) g_init_done[dev][kind] = true;
    return rc;
}

static ChunkAux chunk_aux(const Plan &P, const ChunkDesc &ch, int slot, const TriplesIO &io, int n_part) {
    char *ws = (char *)io.workspace;
    ChunkAux A;
    A.ctrl = (Ctrl *)(ws + P.off_ctrl);
    A.slot = &A.ctrl->slot[slot];
    A.mo_e = io.mo_energy;
    A.e_part = (const double *)(ws + P.off_epart) + (size_t)slot * P.n_ijk * kMaxPartials;
    A.ybar = io.ybar;
    A.o = P.d.o;
    A.a0 = ch.base[0]; A.na = ch.nabc[0];
    A.b0 = ch.base[1]; A.nb = ch.nabc[1];
    A.c0 = ch.base[2]; A.nc = ch.nabc[2];
    A.n_part = n_part;
    A.scaled = P.prec == TRIPLES_PRECISION_MIXED ? 1 : 0;
    A.lno = P.lno;
    return A;
}

// ---------------------------------------------------------------------------
// one-time device set-up and the mixed-precision kernel parameters of a call
// and of one chunk, shared by the single-problem and the batched drivers
// ---------------------------------------------------------------------------
// f(JOBS{}) for each way a launch gets its jobs
template <typename T, typename F>
static void for_job_kinds(F &&f) {
    f(Group<T, 1>{});
    f(Group<T, kMaxGroup>{});
    f(Table<T>{});
}

// once per device and precision: shared-memory opt-ins
static int setup_epilogue(bool mixed) {
    return once_per_device(mixed ? INIT_F2_F32 : INIT_F2_F64, [&]() -> int {
        if (mixed) {
            int rc = TRIPLES_OK;
            for_job_kinds<F2M>([&](auto jobs) {
                using J = decltype(jobs);
                for (auto k : {k_f2m<1, J>, k_f2m<2, J>})
                    if (rc == TRIPLES_OK) rc = smem_optin(k, F2mSmem::BYTES);
            });
            return rc;
        }
        int rc = smem_optin(k_f2t<Group<F2P, 1>>, F2Smem<0>::BYTES);
        if (rc == TRIPLES_OK) rc = smem_optin(k_f2t<Group<F2P, kMaxGroup>>, F2Smem<0>::BYTES);
        return rc;
    });
}

static int setup_tensor_cores() {
    return once_per_device(INIT_TC, [&]() -> int {
        int rc = TRIPLES_OK;
        auto opt = [&](auto kernel, size_t bytes) {
            if (rc == TRIPLES_OK) rc = smem_optin(kernel, bytes);
        };
        for_job_kinds<F1Job>([&](auto jobs) {
            using J = decltype(jobs);
            opt(k_f1_tc<128, J>, TcCfg<128>::SMEM);
            opt(k_f1_tc<256, J>, TcCfg<256>::SMEM);
        });
        for_job_kinds<TcB1Params>([&](auto jobs) {
            using J = decltype(jobs);
            opt(k_b1_tc<false, 128, J>, TcB1Cfg<false, 128>::SMEM);
            opt(k_b1_tc<true, 128, J>, TcB1Cfg<true, 128>::SMEM);
            opt(k_b1_tc<false, 64, J>, TcB1Cfg<false, 64>::SMEM);
            opt(k_b1_tc<true, 64, J>, TcB1Cfg<true, 64>::SMEM);
        });
        return rc;
    });
}

// Tensor maps over one call's 16-bit operands (built on the host).
struct OperandMaps {
    CUtensorMap tmA1, tmB1, tmA2, tmB2;             // W contraction, K-major boxes
    CUtensorMap tmA1m, tmA2m, tmB1z[5], tmB2z[5];   // adjoint contractions, MN-major boxes
};

// The W contraction's N tile is 16 * P.f1_rt columns (occupied r values x 16 z).
static int build_operand_maps(const Plan &P, char *ws, OperandMaps &M) {
    const uint64_t o = P.d.o, v = P.d.v;
    const bool bf16 = P.prec == TRIPLES_PRECISION_MIXED_BF16;
    const uint64_t dA1[5] = {(uint64_t)P.Kp8, v, o, v, 2};
    const uint32_t bA[5] = {64, 16, 8, 1, 1};
    const uint64_t dB1[5] = {(uint64_t)P.Kp8, v, o, o, 2};
    const uint32_t bB[5] = {64, 16, (uint32_t)P.f1_rt, 1, 1};
    const uint64_t dA2[5] = {(uint64_t)P.Op8, v, o, o, 2};
    const uint64_t dB2[5] = {(uint64_t)P.Op8, v, o, v, 2};
    int rc;
    if ((rc = make_tmap5(&M.tmA1, ws + P.off_A1h, bf16, dA1, bA)) != TRIPLES_OK) return rc;
    if ((rc = make_tmap5(&M.tmB1, ws + P.off_B1h, bf16, dB1, bB)) != TRIPLES_OK) return rc;
    if ((rc = make_tmap5(&M.tmA2, ws + P.off_A2h, bf16, dA2, bA)) != TRIPLES_OK) return rc;
    if ((rc = make_tmap5(&M.tmB2, ws + P.off_B2h, bf16, dB2, bB)) != TRIPLES_OK) return rc;
    if (P.want_grad) {
        const uint64_t dA1mn[5] = {(uint64_t)P.Kp8, v, o, v, 2};
        const uint64_t dA2mn[5] = {(uint64_t)P.Op8, v, o, o, 2};
        const uint64_t dB1mn[5] = {(uint64_t)P.Kp8, v, o, o, 2};
        const uint64_t dB2mn[5] = {(uint64_t)P.Op8, v, o, v, 2};
        const uint32_t bX[5] = {64, 16, 4, 1, 1};
        if ((rc = make_tmap5(&M.tmA1m, ws + P.off_A1h, bf16, dA1mn, bX)) != TRIPLES_OK) return rc;
        if ((rc = make_tmap5(&M.tmA2m, ws + P.off_A2h, bf16, dA2mn, bX)) != TRIPLES_OK) return rc;
        for (int lt = 0; lt < 5; lt++) {
            const uint32_t tz = 1u << lt;
            const uint32_t bZ[5] = {64, tz, 64 / tz, 1, 1};
            if ((rc = make_tmap5(&M.tmB1z[lt], ws + P.off_B1h, bf16, dB1mn, bZ)) != TRIPLES_OK) return rc;
            if ((rc = make_tmap5(&M.tmB2z[lt], ws + P.off_B2h, bf16, dB2mn, bZ)) != TRIPLES_OK) return rc;
        }
    }
    return TRIPLES_OK;
}

// W-contraction parameters of one chunk (tiles ordering by ordering).
static int f1_params(const Plan &P, const ChunkDesc &ch, int slot, char *ws, TcF1Params &T) {
    const Dims &d = P.d;
    Ctrl *ctrl = (Ctrl *)(ws + P.off_ctrl);
    float *S = (float *)(ws + P.off_S) + (size_t)slot * P.stage_slot;
    T.d = d;
    T.ch = ch;
    T.mt_count = (d.o + 7) / 8;
    T.rt = P.f1_rt;
    T.nt_count = (d.o + T.rt - 1) / T.rt;
    T.cum[0] = 0;
    for (int t = 0; t < ch.nperm; t++) T.cum[t + 1] = T.cum[t] + ch.pb[t].Ty * d.o * T.mt_count * T.nt_count;
    T.nkb1 = (P.Kp8 + kTcBK - 1) / kTcBK;
    T.nkb2 = (P.Op8 + kTcBK - 1) / kTcBK;
    T.k1 = P.Kp8;
    T.k2 = P.Op8;
    T.S = S;
    T.out_scale = &ctrl->out_scale;
    T.wmax_bits = &ctrl->slot[slot].wmax_bits;
    T.err = &ctrl->err;
    T.bf16 = P.prec == TRIPLES_PRECISION_MIXED_BF16 ? 1 : 0;
    T.kseg = P.kseg;
    for (int t = 0; t < 6; t++) T.tmS_ok[t] = 0;
    for (int t = 0; t < ch.nperm; t++) {
        const PermBlock &pb = ch.pb[t];
        if (pb.Tx == 16 && pb.Tz == 16 && d.o >= 2) {
            const int trc = make_tmap_stage(&T.tmS[t], S + pb.soff, d.o, pb.Ty);
            if (trc != TRIPLES_OK) return trc;
            T.tmS_ok[t] = 1;
        }
    }
    return TRIPLES_OK;
}

// Triples of 8-wide sub-ranges of a chunk, one per orbit of orderings: f(start, length).
template <typename F>
static void for_sub_ranges(const ChunkDesc &ch, F &&f) {
    constexpr int sb = 8;
    int n[3];
    for (int t = 0; t < 3; t++) n[t] = (ch.nabc[t] + sb - 1) / sb;
    for (int ia = 0; ia < n[0]; ia++)
        for (int ib = 0; ib < n[1]; ib++) {
            if (ch.blk[0] == ch.blk[1] && ib > ia) continue;
            for (int ic = 0; ic < n[2]; ic++) {
                if (ch.blk[1] == ch.blk[2] && ic > ib) continue;
                const int idx[3] = {ia, ib, ic};
                int st[3], len[3];
                for (int t = 0; t < 3; t++) {
                    st[t] = ch.base[t] + idx[t] * sb;
                    len[t] = ch.nabc[t] - idx[t] * sb < sb ? ch.nabc[t] - idx[t] * sb : sb;
                }
                f(st, len);
            }
        }
}

// Elements of one sub-range triple of a chunk (all of them have the same lengths), 512 if they are full
static int chunk_elems(const ChunkDesc &ch) {
    return std::min(8, ch.nabc[0]) * std::min(8, ch.nabc[1]) * std::min(8, ch.nabc[2]);
}
// CTAs of an element kernel over a chunk, warps (energy partials) of one of its items
template <typename ARGS>
static int elem_ctas(const Plan &P, const ARGS &A) {
    const long long n = (long long)P.n_ijk * A.nsub * A.sub[0].len[0] * A.sub[0].len[1] * A.sub[0].len[2];
    return (int)((n + kElemThreads - 1) / kElemThreads);
}
static int elem_warps(int elems) { return elems > 32 ? elems / 32 : 1; }

// Chunks that go to the element kernel (k_f2e).  FP64, instead of the orbit kernel (k_f2t): a short
// sub-range, and enough items that the orbit kernel's CTAs would not run side by side (n_ijk 56 is nocc 6;
// E + VJP in blocks of 2, nvir 30, element against orbit kernel: nocc 5 7.43 / 7.14 ms, nocc 7 8.2 / 10.1).
// With the adjoint, items of 256 elements fill the orbit kernel's CTA well enough (nocc 16 nvir 36 =
// 2 x 16 + 4: 8.5 / 8.35 ms; the energy alone 3.12 / 3.29) and those of 128 need more of them (nvir 34:
// nocc 7 1.10 / 1.10 ms, nocc 12 3.76 / 3.86, nocc 16 7.64 / 7.95).
// Mixed modes (k_f2em): items of up to 32 elements, 64 without the adjoint, in place of k_f2m, which
// evaluates 512 slots of every item; its FP32 values are the same (energy nocc 64 nvir 3 0.84 / 7.4 ms,
// nocc 200 nvir 4 23 / 59, nocc 20 nvir 17 0.59 / 0.87; E + VJP nocc 16 nvir 17 0.95 / 1.03, nocc 300 nvir 2
// 72 / 275).
static bool by_element(const Plan &P, const ChunkDesc &ch) {
    const int e = chunk_elems(ch);
    if (P.prec != TRIPLES_PRECISION_FP64) return e <= (P.want_grad ? 32 : 64) && P.n_ijk >= 500;
    if (!P.want_grad) return e < 512 && P.n_ijk >= 56;
    return e <= 64 ? P.n_ijk >= 56 : e <= 128 && P.n_ijk >= 300;
}

// Where the regions of a sub-range triple lie in the (blocked) staging and in
// Wbar (wmul: 2 for the 16-bit hi and lo planes, 1 for FP64).
static void sub_regions(const ChunkDesc &ch, int o, const int *st, const int *len, int wmul, int elem, F2mSub &u) {
    u.full = 1;
    for (int t = 0; t < 3; t++) {
        u.st[t] = st[t];
        u.len[t] = len[t];
        if (len[t] != 8) u.full = 0;
    }
    u.bulk = u.bulk_bytes = 0;
    for (int pi = 0; pi < 6; pi++) {
        int pp[3];
        perm_of(pi, pp);
        int t = 0;
        while (t + 1 < ch.nperm && !(ch.pb[t].bx == ch.blk[pp[0]] && ch.pb[t].by == ch.blk[pp[1]] &&
                                     ch.pb[t].bz == ch.blk[pp[2]]))
            t++;
        const PermBlock &pb = ch.pb[t];
        const int xs = st[pp[0]] - pb.X0, ys = st[pp[1]] - pb.Y0, zs = st[pp[2]] - pb.Z0;
        F2mPi &D = u.pi[pi];
        D.s0 = f2m_stage_offset(pb, o, 0, 0, 0, ys, xs, zs);   // (y, x, z) at a block's origin: no exchange
        D.rs = pb.Tx * pb.Ty * pb.Tz;
        D.tz = pb.Tz;
        D.zs = zs;
        D.tiled = wmul == 2 && wbar_tiled(pb) ? 1 : 0;
        if (D.tiled) {
            const int tile_row = 8 * pb.rzp;   // the tiles of 8 x values
            D.wx = 8;
            D.wp = pb.Tx / 8 * tile_row;
            D.wq = o * D.wp;
            D.wy = o * D.wq;
            D.w0 = wmul * pb.swoff + (long long)ys * D.wy + xs / 8 * tile_row;
        } else {
            D.wq = pb.rzp;
            D.wx = o * D.wq;
            D.wp = pb.Tx * D.wx;
            D.wy = o * D.wp;
            D.w0 = wmul * pb.swoff + (long long)ys * D.wy + (long long)xs * D.wx;
        }
        D.half = (long long)pb.Ty * D.wy;
        D.bytes = elem * len[0] * len[1] * len[2];
        if (D.bytes % 16 == 0) {
            u.bulk |= 1 << pi;
            u.bulk_bytes += D.bytes;
        }
    }
}

// Parameters of one chunk for the FP64 epilogue and for the element kernel of any mode.
static void f2_params(const Plan &P, const ChunkDesc &ch, int slot, char *ws, const TriplesIO &io, F2P &F) {
    const bool mixed = P.prec != TRIPLES_PRECISION_FP64;
    const size_t el = mixed ? 4 : 8;   // bytes of a staged value, of a Wbar value (hi and lo)
    F.o = P.d.o;
    F.v = P.d.v;
    F.nsub = 0;
    for_sub_ranges(ch, [&](const int *st, const int *len) {
        F2mSub &u = F.sub[F.nsub++];
        sub_regions(ch, F.o, st, len, mixed ? 2 : 1, (int)el, u);
        u.pat = st[0] == st[2] ? 3 : (st[0] == st[1] ? 1 : (st[1] == st[2] ? 2 : 0));
    });
    F.n_ijk = P.n_ijk;
    F.ijk = (int *)(ws + P.off_ijk);
    F.mo_e = io.mo_energy; F.t1 = io.t1; F.t2 = io.t2; F.ovov = io.ovov; F.fvo = io.fvo;
    F.S = ws + P.off_S + (size_t)slot * P.stage_slot * el;
    F.SW = P.want_grad ? ws + P.off_SW + (size_t)slot * P.wbar_slot * el : nullptr;
    F.wscale = &((Ctrl *)(ws + P.off_ctrl))->slot[slot].wscale;
    F.ybar = io.ybar;
    F.want_grad = P.want_grad;
    F.e_part = (double *)(ws + P.off_epart) + (size_t)slot * P.n_ijk * kMaxPartials;
    F.mo_bar = io.mo_energy_bar;
    F.t1_bar = io.t1_bar; F.fvo_bar = io.fvo_bar; F.ovov_bar = io.ovov_bar; F.t2_bar = io.t2_bar;
}

// Mixed-precision epilogue parameters of one chunk.
static void f2m_params(const Plan &P, const ChunkDesc &ch, int slot, char *ws, const TriplesIO &io, bool whole, F2M &F) {
    Ctrl *ctrl = (Ctrl *)(ws + P.off_ctrl);
    const int o = P.d.o;
    F.o = o;
    F.v = P.d.v;
    F.nb8 = (P.d.v + 7) / 8;
    F.nsub = 0;
    F.n_ijk = P.n_ijk;
    F.whole = whole ? 1 : 0;
    for_sub_ranges(ch, [&](const int *st, const int *len) {
        F2mSub &u = F.sub[F.nsub++];
        sub_regions(ch, o, st, len, 2, 4, u);
        u.pat = st[0] == st[2] ? 3 : (st[0] == st[1] ? 1 : (st[1] == st[2] ? 2 : 0));
    });
    F.ijk = (int *)(ws + P.off_ijk);
    F.mo_e = io.mo_energy; F.t1 = io.t1; F.t2 = io.t2; F.ovov = io.ovov; F.fvo = io.fvo;
    F.ot = P.vtables ? (const float2 *)(ws + P.off_ot) : nullptr;
    F.tf = P.vtables ? (const float2 *)(ws + P.off_tf) : nullptr;
    F.S = (const float *)(ws + P.off_S) + (size_t)slot * P.stage_slot;
    F.SW = P.want_grad ? (uint16_t *)(ws + P.off_SW) + (size_t)slot * 2 * P.wbar_slot : nullptr;
    F.wscale = &ctrl->slot[slot].wscale;
    F.ybar = io.ybar;
    F.want_grad = P.want_grad;
    F.e_part = (double *)(ws + P.off_epart) + (size_t)slot * P.n_ijk * kMaxPartials;
    F.mo_bar = io.mo_energy_bar;
    F.t1_bar = io.t1_bar; F.fvo_bar = io.fvo_bar; F.ovov_bar = io.ovov_bar; F.t2_bar = io.t2_bar;
    F.err = &ctrl->err;
    F.ticket = &ctrl->slot[slot].ticket;
}

// LNO chunk epilogue: energy of the projected amplitudes and, with want_grad,
// mat_bar, the orbital-energy and V-term gradients and the Wbar staging that
// the adjoint contractions read next (lno.cuh).
template <int COLS, bool FULL>
static int lno_projections(const LnoArgs &A, cudaStream_t st, unsigned &grid) {
    const long long tiles = ((long long)A.o * A.o * A.ne + COLS - 1) / COLS;   // (a CTA has one tile at least)
    grid = (unsigned)std::min({tiles, (long long)2 * num_sms(), (long long)kLnoGrid});
    const size_t smem = LnoProj<COLS>::smem(A.o);
    for (int slot = 2; slot >= 0; slot--)
        TB_KLAUNCH(P_LNO_PROJ, (k_lno_proj<COLS, FULL><<<grid, kLnoThreads, smem, st>>>(A, slot, slot == 2 ? 1 : 0)));
    return TRIPLES_OK;
}

template <typename StageT>
static int lno_chunk(const Plan &P, const ChunkDesc &ch, cudaStream_t st, const TriplesIO &io, char *ws) {
    const bool mixed = sizeof(StageT) == 4, bf16 = P.prec == TRIPLES_PRECISION_MIXED_BF16;
    {
        const int rc = once_per_device(mixed ? INIT_LNO : INIT_LNO64, [&]() -> int {
            int rc = smem_optin(k_lno_fwd<StageT>, F2Smem<0>::TABLES);
            // the projections for the largest nocc of each: a limit set per call would be changed
            // by another host thread between that and the launch
            auto proj = [&](auto cols) {
                using C = LnoProj<decltype(cols)::value>;
                if (rc == TRIPLES_OK) rc = smem_optin(k_lno_proj<decltype(cols)::value, true>, C::smem(C::MAXO));
                if (rc == TRIPLES_OK) rc = smem_optin(k_lno_proj<decltype(cols)::value, false>, C::smem(C::MAXO));
            };
            proj(std::integral_constant<int, 128>{});
            proj(std::integral_constant<int, 64>{});
            proj(std::integral_constant<int, 32>{});
            if (rc != TRIPLES_OK) return rc;
            if (!mixed) return smem_optin(k_lno_adj<0>, F2Smem<0>::BYTES);
            if ((rc = smem_optin(k_lno_adj<1>, F2Smem<1>::BYTES)) != TRIPLES_OK) return rc;
            return smem_optin(k_lno_adj<2>, F2Smem<2>::BYTES);
        });
        if (rc != TRIPLES_OK) return rc;
    }
    const int o = P.d.o;
    Ctrl *ctrl = (Ctrl *)(ws + P.off_ctrl);
    LnoArgs A;
    A.o = o;
    A.v = P.d.v;
    A.nsub = 0;
    int n[3];
    for (int t = 0; t < 3; t++) n[t] = (ch.nabc[t] + 7) / 8;
    for (int c = 0; c < n[0] * n[1] * n[2]; c++) {
        const int idx[3] = {c / (n[1] * n[2]), c / n[2] % n[1], c % n[2]};
        int sst[3], len[3];
        for (int t = 0; t < 3; t++) {
            sst[t] = ch.base[t] + 8 * idx[t];
            len[t] = std::min(8, ch.nabc[t] - 8 * idx[t]);
        }
        F2mSub &u = A.sub[A.nsub++];
        sub_regions(ch, o, sst, len, mixed ? 2 : 1, (int)sizeof(StageT), u);
        u.pat = ch.blk[0] == ch.blk[2] ? 3 : (ch.blk[0] == ch.blk[1] ? 1 : (ch.blk[1] == ch.blk[2] ? 2 : 0));
    }
    A.kn = 0;
    while ((1 << A.kn) < chunk_elems(ch)) A.kn++;
    A.ne = box_slots(ch);
    A.n_ijk = P.n_ijk;
    A.ijk = (int *)(ws + P.off_ijk);
    A.S = ws + P.off_S;
    A.WW = (double *)(ws + P.off_L[0]);
    A.PQ = (double *)(ws + P.off_L[1]);
    A.Q = (double *)(ws + P.off_L[2]);
    A.PW = (double *)(ws + P.off_L[3]);
    A.mat = io.mat; A.mo_e = io.mo_energy; A.t1 = io.t1; A.t2 = io.t2; A.ovov = io.ovov; A.fvo = io.fvo;
    A.SW = P.want_grad ? (void *)(ws + P.off_SW) : nullptr;
    A.wscale = &ctrl->slot[0].wscale;
    A.mat_bar = io.mat_bar; A.mo_bar = io.mo_energy_bar; A.t1_bar = io.t1_bar; A.t2_bar = io.t2_bar;
    A.ovov_bar = io.ovov_bar; A.fvo_bar = io.fvo_bar;
    A.ybar = io.ybar;
    A.f = 2.0 * io.ybar / 3.0;
    A.g = ch.nperm / 9.0;
    A.want_grad = P.want_grad;
    A.part = (double *)(ws + P.off_lpart);
    const unsigned items = (unsigned)(P.n_ijk * A.nsub);
    const bool full = A.kn == 9;
    const unsigned elems = (unsigned)elem_ctas(P, A);
    if (full) TB_KLAUNCH(P_LNO, (k_lno_fwd<StageT><<<items, kLnoThreads, F2Smem<0>::TABLES, st>>>(A)));
    else TB_KLAUNCH(P_LNO, (k_lno_fwd_e<StageT><<<elems, kElemThreads, 0, st>>>(A)));
    // columns per tile: 128 while two buffers of all rows leave room for two CTAs per SM
    unsigned parts = 0;
    const int prc = o <= 16   ? (full ? lno_projections<128, true>(A, st, parts) : lno_projections<128, false>(A, st, parts))
                    : o <= 32 ? (full ? lno_projections<64, true>(A, st, parts) : lno_projections<64, false>(A, st, parts))
                              : (full ? lno_projections<32, true>(A, st, parts) : lno_projections<32, false>(A, st, parts));
    if (prc != TRIPLES_OK) return prc;
    Group<ChunkAux, 1> G;
    G.n = 1;
    G.job[0] = chunk_aux(P, ch, 0, io, 3 * (int)parts);
    G.job[0].e_part = A.part;
    TB_KLAUNCH(P_PREP, (k_energy_sum<<<1, 256, 0, st>>>(G, 1)));
    if (!P.want_grad) return TRIPLES_OK;
    if (!mixed) {
        if (full) TB_KLAUNCH(P_LNO_ADJ, (k_lno_adj<0><<<items, kLnoThreads, F2Smem<0>::BYTES, st>>>(A)));
        else TB_KLAUNCH(P_LNO_ADJ, (k_lno_adj_e<0><<<elems, kElemThreads, 0, st>>>(A)));
        return TRIPLES_OK;
    }
    // fp16: power-of-two scale of the split Wbar; bf16: scale 1 (both read by the contractions)
    TB_KLAUNCH(P_PREP, (k_chunk_scale<<<1, 32, 0, st>>>(G)));
    if (!full && bf16) TB_KLAUNCH(P_LNO_ADJ, (k_lno_adj_e<2><<<elems, kElemThreads, 0, st>>>(A)));
    else if (!full) TB_KLAUNCH(P_LNO_ADJ, (k_lno_adj_e<1><<<elems, kElemThreads, 0, st>>>(A)));
    else if (bf16) TB_KLAUNCH(P_LNO_ADJ, (k_lno_adj<2><<<items, kLnoThreads, F2Smem<2>::BYTES, st>>>(A)));
    else TB_KLAUNCH(P_LNO_ADJ, (k_lno_adj<1><<<items, kLnoThreads, F2Smem<1>::BYTES, st>>>(A)));
    return TRIPLES_OK;
}

// Adjoint-contraction parameters of one chunk and kind (0: ovvv_bar, 1: t2_bar
// ovvv term, 2: ovoo_bar, 3: t2_bar ooov term), tiles ordering by ordering.
static int b1_params(const Plan &P, const ChunkDesc &ch, int slot, char *ws, const OperandMaps &M, int kind, TcB1Params &B) {
    const Dims &d = P.d;
    const uint64_t o = d.o;
    const bool bf16 = P.prec == TRIPLES_PRECISION_MIXED_BF16;
    Ctrl *ctrl = (Ctrl *)(ws + P.off_ctrl);
    char *SW = ws + P.off_SW + (size_t)slot * P.wbar_slot * 4;
    const uint32_t bK[5] = {64, 1, 16, 8, 1};   // Wbar K-major (kinds 0, 2)
    const uint32_t bM[5] = {64, 1, 16, 4, 1};   // Wbar MN-major (kinds 1, 3)
    B.d = d;
    B.nperm = ch.nperm;
    for (int t = 0; t < ch.nperm; t++) B.pb[t] = ch.pb[t];
    B.wscale = &ctrl->slot[slot].wscale;
    B.err = &ctrl->err;
    B.bf16 = bf16 ? 1 : 0;
    B.kseg = P.kseg;
    B.kind = kind;
    {
        const int most = kind <= 1 ? 128 : 64;
        B.ncol = kind <= 1 ? d.v : d.o;
        B.ntile_n = (B.ncol + most - 1) / most;
        B.nw = B.ntile_n > 1 ? most : (B.ncol + 15) / 16 * 16;
    }
    B.G = (double *)(ws + (kind == 0 ? P.off_GA1 : kind == 1 ? P.off_GB1 : kind == 2 ? P.off_GA2 : P.off_GB2));
    B.oscale = &ctrl->scale[(kind == 0 || kind == 2) ? 1 : 0];
    B.sign = kind == 2 ? -1.0 : 1.0;
    for (int t = 0; t < ch.nperm; t++) {
        const PermBlock &pb = ch.pb[t];
        const bool kmajor = kind == 0 || kind == 2;
        int rc;
        if (wbar_tiled(pb)) {
            // [h y q][p, x tile][rz tile][64]; boxes of 128 rows x 64 K values (K = 4 p in the MN-major kinds)
            const uint64_t nxb = pb.Tx / 8;
            const uint64_t dT[5] = {64, (uint64_t)pb.rzp / 8, o * nxb, 2 * pb.Ty * o, 1};
            const uint32_t bTK[5] = {64, 8, 16, 1, 1}, bTM[5] = {64, 16, (uint32_t)(4 * nxb), 1, 1};
            rc = make_tmap5(&B.tmA[t], SW + 2 * pb.swoff * 2, bf16, dT, kmajor ? bTK : bTM, false);
        } else {
            const uint64_t dW[5] = {(uint64_t)pb.rzp, o, (uint64_t)pb.Tx, o, (uint64_t)(2 * pb.Ty)};
            rc = make_tmap5(&B.tmA[t], SW + 2 * pb.swoff * 2, bf16, dW, kmajor ? bK : bM);
        }
        if (rc != TRIPLES_OK) return rc;
        const int mt_px = (d.o * (pb.Tx == 8 ? 8 : 16) + kTcBM - 1) / kTcBM;   // M tiles over (p, x)
        int lz = 0;
        while ((1 << lz) < pb.Tz) lz++;
        switch (kind) {
        case 0:
            B.tmB[t] = M.tmB1z[lz];
            B.nbatch[t] = pb.Ty; B.ntile_m[t] = mt_px;
            B.nk_outer[t] = d.o; B.nk_inner[t] = (d.o * pb.Tz + 63) / 64;
            break;
        case 1:
            B.tmB[t] = M.tmA1m;
            B.nbatch[t] = d.o; B.ntile_m[t] = (d.o * pb.Tz + 127) / 128;
            B.nk_outer[t] = pb.Ty; B.nk_inner[t] = (d.o + 3) / 4;
            break;
        case 2:
            B.tmB[t] = M.tmB2z[lz];
            B.nbatch[t] = d.o; B.ntile_m[t] = mt_px;
            B.nk_outer[t] = pb.Ty; B.nk_inner[t] = (d.o * pb.Tz + 63) / 64;
            break;
        default:
            B.tmB[t] = M.tmA2m;
            B.nbatch[t] = pb.Ty; B.ntile_m[t] = (d.o * pb.Tz + 127) / 128;
            B.nk_outer[t] = d.o; B.nk_inner[t] = (d.o + 3) / 4;
            break;
        }
    }
    B.cum[0] = 0;
    for (int t = 0; t < ch.nperm; t++) B.cum[t + 1] = B.cum[t] + B.nbatch[t] * B.ntile_m[t] * B.ntile_n;
    return TRIPLES_OK;
}

// Per-call preparation: control block, occupied table, zeroed gradients, and
// the operand layouts (FP64 copies, or 16-bit splits with their scales).
template <typename StageT>
static int prep_launches(const Plan &P, cudaStream_t st, const TriplesIO &io) {
    const Dims d = P.d;
    const bool mixed = P.prec != TRIPLES_PRECISION_FP64;
    const bool bf16 = P.prec == TRIPLES_PRECISION_MIXED_BF16;
    char *ws = (char *)io.workspace;
    Ctrl *ctrl = (Ctrl *)(ws + P.off_ctrl);
    double *A1 = (double *)(ws + P.off_A1);
    double *B1 = (double *)(ws + P.off_B1);
    double *A2 = (double *)(ws + P.off_A2);
    double *B2 = (double *)(ws + P.off_B2);
    void *SW = P.want_grad ? (void *)(ws + P.off_SW) : nullptr;
    double *GA1 = P.want_grad ? (double *)(ws + P.off_GA1) : nullptr;
    double *GB1 = P.want_grad ? (double *)(ws + P.off_GB1) : nullptr;
    double *GA2 = P.want_grad ? (double *)(ws + P.off_GA2) : nullptr;
    double *GB2 = P.want_grad ? (double *)(ws + P.off_GB2) : nullptr;
    int *ijk = (int *)(ws + P.off_ijk);
    const size_t o = d.o, v = d.v, n = d.n;

    TB_CUDA(cudaMemsetAsync(ctrl, 0, kCtrlBytes, st));
    TB_KLAUNCH(P_PREP, k_ijk_table<<<grid1d(P.n_ijk, 128), 128, 0, st>>>(d.o, ijk));
    if (P.want_grad) {
        TB_CUDA(cudaMemsetAsync(GA1, 0, v * o * v * d.Kp * sizeof(double), st));
        TB_CUDA(cudaMemsetAsync(GB1, 0, o * o * v * d.Kp * sizeof(double), st));
        TB_CUDA(cudaMemsetAsync(GA2, 0, o * o * v * o * sizeof(double), st));
        TB_CUDA(cudaMemsetAsync(GB2, 0, v * o * v * o * sizeof(double), st));
        TB_CUDA(cudaMemsetAsync(io.mo_energy_bar, 0, n * sizeof(double), st));
        TB_CUDA(cudaMemsetAsync(io.t1_bar, 0, o * v * sizeof(double), st));
        TB_CUDA(cudaMemsetAsync(io.t2_bar, 0, o * o * v * v * sizeof(double), st));
        TB_CUDA(cudaMemsetAsync(io.ovov_bar, 0, o * v * o * v * sizeof(double), st));
        TB_CUDA(cudaMemsetAsync(io.fvo_bar, 0, v * o * sizeof(double), st));
        if (P.lno) {
            TB_CUDA(cudaMemsetAsync(io.mat_bar, 0, o * o * sizeof(double), st));
            if (mixed) TB_KLAUNCH(P_PREP, k_lno_mat_norms<<<1, 64, 0, st>>>(io.mat, d.o, ctrl));
        }
    }

    // FP64 operand layouts (used by the FP64 contractions only)
    if (!mixed) {
        TB_KLAUNCH(P_PREP, k_prep_A1<<<dim3((d.Kp + 31) / 32, (d.v + 31) / 32, (unsigned)(o * v)), dim3(32, 8), 0, st>>>(
            io.ovvv, P.packed, d, A1));
        TB_KLAUNCH(P_PREP, k_prep_B1<<<(unsigned)(o * o * v), 128, 0, st>>>(io.t2, d, B1));
        TB_KLAUNCH(P_PREP, k_prep_A2<<<grid1d((long long)o * o * v * o, 256), 256, 0, st>>>(io.ovoo, d, A2));
        TB_KLAUNCH(P_PREP, k_prep_B2<<<grid1d((long long)v * o * v * o, 256), 256, 0, st>>>(io.t2, d, B2));
    }

    // 16-bit split operands (tensor-core path)
    if (mixed) {
        const long long npair = (long long)v * (v + 1) / 2;
        TB_KLAUNCH(P_PREP, k_absmax<<<grid1d((long long)o * v * (P.packed ? npair : (long long)v * v), 256), 256, 0, st>>>(
            io.ovvv, (long long)o * v * (P.packed ? npair : (long long)v * v), &ctrl->absmax[0]));
        TB_KLAUNCH(P_PREP, k_absmax<<<grid1d((long long)o * v * o * o, 256), 256, 0, st>>>(io.ovoo, (long long)o * v * o * o,
                                                                         &ctrl->absmax[1]));
        TB_KLAUNCH(P_PREP, k_absmax<<<grid1d((long long)o * o * v * v, 256), 256, 0, st>>>(io.t2, (long long)o * o * v * v,
                                                                         &ctrl->absmax[2]));
        TB_KLAUNCH(P_PREP, k_absmax<<<grid1d((long long)o * v * o * v, 256), 256, 0, st>>>(io.ovov, (long long)o * v * o * v, &ctrl->absmax[3]));
        TB_KLAUNCH(P_PREP, k_absmax<<<grid1d((long long)o * v, 256), 256, 0, st>>>(io.t1, (long long)o * v, &ctrl->absmax[4]));
        TB_KLAUNCH(P_PREP, k_absmax<<<grid1d((long long)o * v, 256), 256, 0, st>>>(io.fvo, (long long)o * v, &ctrl->absmax[5]));
        TB_KLAUNCH(P_PREP, k_make_scales<<<1, 1, 0, st>>>(ctrl, bf16 ? 0 : 1));
        if (bf16) {
            if (P.packed)
                TB_KLAUNCH(P_PREP, k_prep_A1h_packed<__nv_bfloat16><<<tri_grid(P.Kp8, o * v), 256, 0, st>>>(
                    io.ovvv, d, P.Kp8, ctrl, (__nv_bfloat16 *)(ws + P.off_A1h)));
            else
                TB_KLAUNCH(P_PREP, k_prep_A1h<__nv_bfloat16><<<dim3((P.Kp8 + 31) / 32, (d.v + 31) / 32, (unsigned)(o * v)), dim3(32, 8), 0, st>>>(
                    io.ovvv, d, P.Kp8, ctrl, (__nv_bfloat16 *)(ws + P.off_A1h)));
            TB_KLAUNCH(P_PREP, k_prep_B1h<__nv_bfloat16><<<(unsigned)(o * o * v), 128, 0, st>>>(io.t2, d, P.Kp8, ctrl,
                                                                            (__nv_bfloat16 *)(ws + P.off_B1h)));
            TB_KLAUNCH(P_PREP, k_prep_A2h<__nv_bfloat16><<<grid1d((long long)o * o * v * P.Op8, 256), 256, 0, st>>>(
                io.ovoo, d, P.Op8, ctrl, (__nv_bfloat16 *)(ws + P.off_A2h)));
            TB_KLAUNCH(P_PREP, k_prep_B2h<__nv_bfloat16><<<rz_grid(d, P.Op8), 256, 0, st>>>(
                io.t2, d, P.Op8, ctrl, (__nv_bfloat16 *)(ws + P.off_B2h)));
        } else {
            if (P.packed)
                TB_KLAUNCH(P_PREP, k_prep_A1h_packed<__half><<<tri_grid(P.Kp8, o * v), 256, 0, st>>>(
                    io.ovvv, d, P.Kp8, ctrl, (__half *)(ws + P.off_A1h)));
            else
                TB_KLAUNCH(P_PREP, k_prep_A1h<__half><<<dim3((P.Kp8 + 31) / 32, (d.v + 31) / 32, (unsigned)(o * v)), dim3(32, 8), 0, st>>>(
                    io.ovvv, d, P.Kp8, ctrl, (__half *)(ws + P.off_A1h)));
            TB_KLAUNCH(P_PREP, k_prep_B1h<__half><<<(unsigned)(o * o * v), 128, 0, st>>>(io.t2, d, P.Kp8, ctrl,
                                                                     (__half *)(ws + P.off_B1h)));
            TB_KLAUNCH(P_PREP, k_prep_A2h<__half><<<grid1d((long long)o * o * v * P.Op8, 256), 256, 0, st>>>(
                io.ovoo, d, P.Op8, ctrl, (__half *)(ws + P.off_A2h)));
            TB_KLAUNCH(P_PREP, k_prep_B2h<__half><<<rz_grid(d, P.Op8), 256, 0, st>>>(
                io.t2, d, P.Op8, ctrl, (__half *)(ws + P.off_B2h)));
        }
        if (P.vtables) {
            const int nb8 = (d.v + 7) / 8;
            TB_KLAUNCH(P_PREP, k_prep_vtables<<<grid1d((long long)o * o * nb8 * nb8 * 64, 256), 256, 0, st>>>(
                io.ovov, io.t2, io.t1, io.fvo, d.o, d.v, nb8, (float2 *)(ws + P.off_ot), (float2 *)(ws + P.off_tf)));
        }
        TB_LAUNCH_CHECK();
        if (P.want_grad) TB_CUDA(cudaMemsetAsync(SW, 0, ((P.group - 1) * P.wbar_slot + P.wbar_elems) * 4, st));
    }
    return TRIPLES_OK;

}

// Gradients back to the reference layouts, and the energy out.
static int fold_launches(const Plan &P, cudaStream_t st, const TriplesIO &io) {
    const Dims d = P.d;
    char *ws = (char *)io.workspace;
    Ctrl *ctrl = (Ctrl *)(ws + P.off_ctrl);
    const double *GA1 = (const double *)(ws + P.off_GA1), *GB1 = (const double *)(ws + P.off_GB1);
    const double *GA2 = (const double *)(ws + P.off_GA2), *GB2 = (const double *)(ws + P.off_GB2);
    const size_t o = d.o, v = d.v;
    if (P.want_grad) {
        if (P.packed) {
            TB_KLAUNCH(P_FOLD, k_fold_ovvv_packed<<<tri_grid(d.v, o * v), 256, 0, st>>>(GA1, d, io.ovvv_bar));
        } else {
            TB_KLAUNCH(P_FOLD, k_fold_ovvv_full<<<dim3((d.v + 31) / 32, (d.v + 31) / 32, (unsigned)(o * v)), dim3(32, 8), 0, st>>>(
                GA1, d, io.ovvv_bar));
        }
        TB_LAUNCH_CHECK();
        TB_KLAUNCH(P_FOLD, k_fold_t2<<<rz_grid(d, d.o), 256, 0, st>>>(GB1, GB2, d, io.t2_bar));
        TB_KLAUNCH(P_FOLD, k_fold_ovoo<<<grid1d((long long)o * v * o * o, 256), 256, 0, st>>>(GA2, d, io.ovoo_bar));
    }
    TB_KLAUNCH(P_FOLD, k_copy_scalar<<<1, 1, 0, st>>>(&ctrl->e_acc, io.e_out));
    return TRIPLES_OK;
}

// The work units of a group: start[] from per-job counts.
template <typename G, typename F>
static int group_starts(G &g, int n, F &&count) {
    g.n = n;
    g.start[0] = 0;
    for (int j = 0; j < n; j++) g.start[j + 1] = g.start[j] + count(g.job[j]);
    return g.start[n];
}

template <typename JOBS>
static void launch_f1(const Plan &P, cudaStream_t st, int tiles, const JOBS &J) {
    const int grid = std::min(tiles, num_sms());
    if (P.f1_bn == 128) k_f1_tc<128, JOBS><<<grid, kF1Threads, TcCfg<128>::SMEM, st>>>(J);
    else k_f1_tc<256, JOBS><<<grid, kF1Threads, TcCfg<256>::SMEM, st>>>(J);
}

template <typename JOBS>
static void launch_f2m(bool bf16, cudaStream_t st, int items, const JOBS &J) {
    const int grid = std::min(items, 2 * num_sms());
    if (bf16) k_f2m<2, JOBS><<<grid, kF2mThreads, F2mSmem::BYTES, st>>>(J);
    else k_f2m<1, JOBS><<<grid, kF2mThreads, F2mSmem::BYTES, st>>>(J);
}

constexpr int kB1Cat[4] = {P_B1A, P_B1B, P_B1C, P_B1D};

template <typename JOBS>
static void launch_b1(int kind, cudaStream_t st, int tiles, const JOBS &J) {
    const int grid = std::min(tiles, num_sms());
    switch (kind) {
    case 0: k_b1_tc<false, 128, JOBS><<<grid, kB1Threads, TcB1Cfg<false, 128>::SMEM, st>>>(J); break;
    case 1: k_b1_tc<true, 128, JOBS><<<grid, kB1Threads, TcB1Cfg<true, 128>::SMEM, st>>>(J); break;
    case 2: k_b1_tc<false, 64, JOBS><<<grid, kB1Threads, TcB1Cfg<false, 64>::SMEM, st>>>(J); break;
    default: k_b1_tc<true, 64, JOBS><<<grid, kB1Threads, TcB1Cfg<true, 64>::SMEM, st>>>(J); break;
    }
}

// n chunks of one call in the mixed modes: W contraction, epilogue (energy and
// adjoint of the raw amplitudes), adjoint contractions.
template <int NG>
static int mixed_chunks(const Plan &P, const ChunkDesc *ch, int n, cudaStream_t st, const TriplesIO &io,
                        const OperandMaps &M) {
    const bool bf16 = P.prec == TRIPLES_PRECISION_MIXED_BF16;
    char *ws = (char *)io.workspace;
    {
        Group<F1Job, NG> G;
        for (int c = 0; c < n; c++) {
            G.job[c].m = F1Maps{M.tmA1, M.tmB1, M.tmA2, M.tmB2};
            const int rc = f1_params(P, ch[c], c, ws, G.job[c].P);
            if (rc != TRIPLES_OK) return rc;
        }
        const int tiles = group_starts(G, n, [](const F1Job &j) { return j.P.cum[j.P.ch.nperm]; });
        TB_KLAUNCH(P_F1, launch_f1(P, st, tiles, G));
    }
    if (P.lno) {
        // projected energy: whole-chunk epilogue instead of the orbit tiles (one chunk at a time)
        const int rc = lno_chunk<float>(P, ch[0], st, io, ws);
        if (rc != TRIPLES_OK) return rc;
    } else {
        // chunks for the persistent epilogue and for the element kernel
        Group<F2M, NG> G;
        Group<F2P, NG> H;
        Group<ChunkAux, NG> X;
        int nf2m = 0, nelem = 0;
        for (int c = 0; c < n; c++) {
            if (by_element(P, ch[c])) {
                F2P &j = H.job[nelem++];
                f2_params(P, ch[c], c, ws, io, j);
                X.job[c] = chunk_aux(P, ch[c], c, io, P.n_ijk * j.nsub * elem_warps(chunk_elems(ch[c])));
            } else {
                F2M &j = G.job[nf2m++];
                f2m_params(P, ch[c], c, ws, io, false, j);
                X.job[c] = chunk_aux(P, ch[c], c, io, P.n_ijk * j.nsub);
            }
        }
        X.n = n;
        if (P.want_grad) TB_KLAUNCH(P_PREP, (k_chunk_scale<<<n, 32, 0, st>>>(X)));
        if (nf2m > 0) {
            const int items = group_starts(G, nf2m, [&](const F2M &j) { return P.n_ijk * j.nsub; });
            TB_KLAUNCH(P_F2, launch_f2m(bf16, st, items, G));
        }
        if (nelem > 0) {
            const int ctas = group_starts(H, nelem, [&](const F2P &j) { return elem_ctas(P, j); });
            if (bf16) TB_KLAUNCH(P_F2, (k_f2em<2><<<(unsigned)ctas, kElemThreads, 0, st>>>(H)));
            else TB_KLAUNCH(P_F2, (k_f2em<1><<<(unsigned)ctas, kElemThreads, 0, st>>>(H)));
        }
        TB_KLAUNCH(P_F2, (k_energy_sum<<<1, 256, 0, st>>>(X, n)));
    }
    if (!P.want_grad) return TRIPLES_OK;
    for (int kind = 0; kind < 4; kind++) {
        Group<TcB1Params, NG> G;
        for (int c = 0; c < n; c++) {
            const int rc = b1_params(P, ch[c], c, ws, M, kind, G.job[c]);
            if (rc != TRIPLES_OK) return rc;
        }
        const int tiles = group_starts(G, n, [](const TcB1Params &j) { return j.cum[j.nperm]; });
        TB_KLAUNCH(kB1Cat[kind], launch_b1(kind, st, tiles, G));
    }
    return TRIPLES_OK;
}

// The same in FP64.
template <int NG>
static int fp64_chunks(const Plan &P, const ChunkDesc *ch, int n, cudaStream_t st, const TriplesIO &io) {
    char *ws = (char *)io.workspace;
    GemmLaunch L;
    L.d = P.d;
    L.n = n;
    L.A1 = (const double *)(ws + P.off_A1);
    L.B1 = (const double *)(ws + P.off_B1);
    L.A2 = (const double *)(ws + P.off_A2);
    L.B2 = (const double *)(ws + P.off_B2);
    L.G = nullptr;
    for (int c = 0; c < n; c++) {
        L.ch[c] = ch[c];
        L.S[c] = (double *)(ws + P.off_S) + c * P.stage_slot;
        L.SW[c] = P.want_grad ? (double *)(ws + P.off_SW) + c * P.wbar_slot : nullptr;
    }
    int rc;
    if ((rc = chunk_gemm<GK_F1>(st, P_F1, L)) != TRIPLES_OK) return rc;
    if (P.lno) {
        rc = lno_chunk<double>(P, ch[0], st, io, ws);
        if (rc != TRIPLES_OK) return rc;
    } else {
        // chunks for the orbit kernel and for the element kernel
        Group<F2P, NG> G, H;
        Group<ChunkAux, NG> X;
        int norb = 0, nelem = 0;
        for (int c = 0; c < n; c++) {
            const bool elem = by_element(P, ch[c]);
            F2P &j = elem ? H.job[nelem++] : G.job[norb++];
            f2_params(P, ch[c], c, ws, io, j);
            X.job[c] = chunk_aux(P, ch[c], c, io, P.n_ijk * j.nsub * (elem ? elem_warps(chunk_elems(ch[c])) : 1));
        }
        X.n = n;
        if (norb > 0) {
            const int items = group_starts(G, norb, [&](const F2P &j) { return P.n_ijk * j.nsub; });
            TB_KLAUNCH(P_F2, (k_f2t<<<(unsigned)items, kF2Threads, F2Smem<0>::BYTES, st>>>(G)));
        }
        if (nelem > 0) {
            const int ctas = group_starts(H, nelem, [&](const F2P &j) { return elem_ctas(P, j); });
            TB_KLAUNCH(P_F2, (k_f2e<<<(unsigned)ctas, kElemThreads, 0, st>>>(H)));
        }
        TB_KLAUNCH(P_F2, (k_energy_sum<<<1, 256, 0, st>>>(X, n)));
    }
    if (!P.want_grad) return TRIPLES_OK;
    L.G = (double *)(ws + P.off_GA1);
    if ((rc = chunk_gemm<GK_B1A>(st, P_B1A, L)) != TRIPLES_OK) return rc;
    L.G = (double *)(ws + P.off_GB2);
    if ((rc = chunk_gemm<GK_B1D>(st, P_B1D, L)) != TRIPLES_OK) return rc;
    L.G = (double *)(ws + P.off_GB1);
    if ((rc = chunk_gemm<GK_B1B>(st, P_B1B, L)) != TRIPLES_OK) return rc;
    L.G = (double *)(ws + P.off_GA2);
    return chunk_gemm<GK_B1C>(st, P_B1C, L);
}

template <typename StageT>
static int run_impl(const Plan &P, cudaStream_t st, const TriplesIO &io) {
    const bool mixed = P.prec != TRIPLES_PRECISION_FP64;
    int prc = setup_epilogue(mixed);
    if (prc != TRIPLES_OK) return prc;
    if ((prc = prep_launches<StageT>(P, st, io)) != TRIPLES_OK) return prc;
    const Dims d = P.d;
    char *ws = (char *)io.workspace;
    OperandMaps M;
    if (mixed) {
        if ((prc = build_operand_maps(P, ws, M)) != TRIPLES_OK) return prc;
        if ((prc = setup_tensor_cores()) != TRIPLES_OK) return prc;
    }

    // the chunks of a group (P.group at most) run in one launch per kernel
    ChunkDesc ch[kMaxGroup];
    int n = 0;
    auto run_group = [&]() -> int {
        if (n == 0) return TRIPLES_OK;
        const int rc = mixed ? (n == 1 ? mixed_chunks<1>(P, ch, n, st, io, M) : mixed_chunks<kMaxGroup>(P, ch, n, st, io, M))
                             : (n == 1 ? fp64_chunks<1>(P, ch, n, st, io) : fp64_chunks<kMaxGroup>(P, ch, n, st, io));
        n = 0;
        return rc;
    };
    for (int A = P.a0; A < P.nb && (P.a1 <= 0 || A < P.a1); A++)
        for (int B = 0; B <= A; B++)
            for (int C = 0; C <= B; C++) {
                make_chunk(d, A, B, C, ch[n++]);
                if (n == P.group && (prc = run_group()) != TRIPLES_OK) return prc;
            }
    if ((prc = run_group()) != TRIPLES_OK) return prc;
    return fold_launches(P, st, io);
}

int run_triples(const Plan &P, cudaStream_t st, const TriplesIO &io) {
    if (P.prec == TRIPLES_PRECISION_FP64) return run_impl<double>(P, st, io);
    return run_impl<float>(P, st, io);
}

// ---------------------------------------------------------------------------
// batched calls: many problems of uneven size.  Every problem keeps its own
// workspace (operands, one chunk's staging, gradient accumulators); chunk
// step c launches each kernel kind ONCE over the c-th chunk of every problem
// that has one (tiles / CTAs numbered problem after problem, parameters in
// job tables built on the host when the batch is created and stored after
// the problems' workspaces).  Mixed precision only; an FP64 batch runs the
// problems one after another.
// ---------------------------------------------------------------------------
struct BatchStep {
    size_t f1_jobs[2], f1_start[2];   // [0]: W-contraction N tile 256, [1]: 128
    int f1_n[2], f1_tiles[2];
    size_t aux;                       // ChunkAux per problem of the step
    int naux;
    size_t f2_jobs, f2_start;
    int f2_items;
    size_t b1_jobs[4], b1_start[4];   // per adjoint kind
    int b1_tiles[4];
};

struct Batch {
    int prec = 0, nprob = 0;
    char *ws = nullptr;
    std::vector<Plan> plans;
    std::vector<TriplesIO> ios;
    std::vector<size_t> ws_off;
    std::vector<BatchStep> steps;
    size_t tables_off = 0, total = 0;
};

static void batch_chunks(const Plan &P, std::vector<ChunkDesc> &out) {
    out.clear();
    for (int A = 0; A < P.nb; A++)
        for (int B = 0; B <= A; B++)
            for (int C = 0; C <= B; C++) {
                ChunkDesc ch;
                make_chunk(P.d, A, B, C, ch);
                out.push_back(ch);
            }
}

// Plans, workspace offsets and (with image != nullptr) the job tables of a
// batch; B.ws must then be the device workspace the tables point into.
static int batch_build(Batch &B, int prec, int nprob, const triples_problem *probs, double ybar,
                       std::vector<char> *image, bool vtables) {
    if (nprob < 1 || !probs) return TRIPLES_ERR_INVALID_ARGUMENT;
    B.prec = prec;
    B.nprob = nprob;
    B.plans.assign(nprob, Plan{});
    B.ios.assign(nprob, TriplesIO{});
    B.ws_off.assign(nprob, 0);
    size_t off = 0;
    for (int p = 0; p < nprob; p++) {
        const triples_problem &q = probs[p];
        triples_options opt{};
        opt.block_size = q.block_size;
        opt.tile_n = q.tile_n;
        const int rc = make_plan(prec, q.nocc, q.nvir, q.ovvv_packed, 1, B.plans[p], 0, &opt, vtables);
        if (rc != TRIPLES_OK) return rc;
        B.ws_off[p] = off;
        off = align256(off + B.plans[p].total);
        TriplesIO &io = B.ios[p];
        io.mo_energy = q.mo_energy; io.t1 = q.t1; io.t2 = q.t2; io.ovoo = q.ovoo; io.ovov = q.ovov;
        io.ovvv = q.ovvv; io.fvo = q.fvo; io.ybar = ybar; io.e_out = q.e_out;
        io.mo_energy_bar = q.mo_energy_bar; io.t1_bar = q.t1_bar; io.t2_bar = q.t2_bar; io.ovoo_bar = q.ovoo_bar;
        io.ovov_bar = q.ovov_bar; io.ovvv_bar = q.ovvv_bar; io.fvo_bar = q.fvo_bar;
        io.workspace = B.ws ? B.ws + B.ws_off[p] : nullptr;
        if (image && (!io.mo_energy || !io.t1 || !io.t2 || !io.ovoo || !io.ovov || !io.ovvv || !io.fvo || !io.e_out ||
                      !io.mo_energy_bar || !io.t1_bar || !io.t2_bar || !io.ovoo_bar || !io.ovov_bar ||
                      !io.ovvv_bar || !io.fvo_bar))
            return TRIPLES_ERR_INVALID_ARGUMENT;
    }
    B.tables_off = off;
    B.steps.clear();
    if (prec == TRIPLES_PRECISION_FP64) {
        B.total = off;
        return TRIPLES_OK;
    }
    std::vector<std::vector<ChunkDesc>> chunks(nprob);
    std::vector<OperandMaps> maps(image ? nprob : 0);
    size_t nsteps = 0;
    for (int p = 0; p < nprob; p++) {
        batch_chunks(B.plans[p], chunks[p]);
        if (chunks[p].size() > nsteps) nsteps = chunks[p].size();
        if (image) {
            const int rc = build_operand_maps(B.plans[p], B.ws + B.ws_off[p], maps[p]);
            if (rc != TRIPLES_OK) return rc;
        }
    }
    // table layout: per step, 256-byte aligned arrays
    size_t t = 0;
    auto take = [&](size_t bytes) {
        const size_t at = t;
        t = align256(t + bytes);
        return at;
    };
    B.steps.resize(nsteps);
    for (size_t c = 0; c < nsteps; c++) {
        BatchStep &S = B.steps[c];
        std::vector<int> who, who_bn[2];
        for (int p = 0; p < nprob; p++)
            if (c < chunks[p].size()) {
                who.push_back(p);
                who_bn[B.plans[p].f1_bn == 256 ? 0 : 1].push_back(p);
            }
        const int n = (int)who.size();
        for (int g = 0; g < 2; g++) {
            S.f1_n[g] = (int)who_bn[g].size();
            S.f1_jobs[g] = take(sizeof(F1Job) * S.f1_n[g]);
            S.f1_start[g] = take(sizeof(int) * (S.f1_n[g] + 1));
        }
        S.naux = n;
        S.aux = take(sizeof(ChunkAux) * n);
        S.f2_jobs = take(sizeof(F2M) * n);
        S.f2_start = take(sizeof(int) * (n + 1));
        for (int k = 0; k < 4; k++) {
            S.b1_jobs[k] = take(sizeof(TcB1Params) * n);
            S.b1_start[k] = take(sizeof(int) * (n + 1));
        }
        if (!image) continue;
        if (image->size() < t) image->resize(t);
        char *img = image->data();
        for (int g = 0; g < 2; g++) {
            int *start = (int *)(img + S.f1_start[g]);
            start[0] = 0;
            for (int j = 0; j < S.f1_n[g]; j++) {
                const int p = who_bn[g][j];
                F1Job job;
                std::memset(&job, 0, sizeof(job));
                const OperandMaps &M = maps[p];
                job.m = F1Maps{M.tmA1, M.tmB1, M.tmA2, M.tmB2};
                const int rc = f1_params(B.plans[p], chunks[p][c], 0, B.ws + B.ws_off[p], job.P);
                if (rc != TRIPLES_OK) return rc;
                std::memcpy(img + S.f1_jobs[g] + sizeof(F1Job) * j, &job, sizeof(job));
                start[j + 1] = start[j] + job.P.cum[job.P.ch.nperm];
            }
            S.f1_tiles[g] = start[S.f1_n[g]];
        }
        int *f2s = (int *)(img + S.f2_start);
        f2s[0] = 0;
        int *b1s[4];
        for (int k = 0; k < 4; k++) {
            b1s[k] = (int *)(img + S.b1_start[k]);
            b1s[k][0] = 0;
        }
        for (int j = 0; j < n; j++) {
            const int p = who[j];
            const Plan &P = B.plans[p];
            const ChunkDesc &ch = chunks[p][c];
            char *wsp = B.ws + B.ws_off[p];
            F2M F;
            std::memset(&F, 0, sizeof(F));
            f2m_params(P, ch, 0, wsp, B.ios[p], true, F);
            std::memcpy(img + S.f2_jobs + sizeof(F) * j, &F, sizeof(F));
            f2s[j + 1] = f2s[j] + P.n_ijk * F.nsub;
            const ChunkAux A = chunk_aux(P, ch, 0, B.ios[p], P.n_ijk * F.nsub);
            std::memcpy(img + S.aux + sizeof(A) * j, &A, sizeof(A));
            for (int k = 0; k < 4; k++) {
                TcB1Params Bp;
                std::memset(&Bp, 0, sizeof(Bp));
                const int rc = b1_params(P, ch, 0, wsp, maps[p], k, Bp);
                if (rc != TRIPLES_OK) return rc;
                std::memcpy(img + S.b1_jobs[k] + sizeof(Bp) * j, &Bp, sizeof(Bp));
                b1s[k][j + 1] = b1s[k][j] + Bp.cum[ch.nperm];
            }
        }
        S.f2_items = f2s[n];
        for (int k = 0; k < 4; k++) S.b1_tiles[k] = b1s[k][n];
    }
    if (image) image->resize(t);
    B.total = B.tables_off + t;
    return TRIPLES_OK;
}

static int run_batch(const Batch &B, cudaStream_t st) {
    if (B.prec == TRIPLES_PRECISION_FP64) {
        for (int p = 0; p < B.nprob; p++) {
            const int rc = run_impl<double>(B.plans[p], st, B.ios[p]);
            if (rc != TRIPLES_OK) return rc;
        }
        return TRIPLES_OK;
    }
    int rc;
    if ((rc = setup_epilogue(true)) != TRIPLES_OK) return rc;
    if ((rc = setup_tensor_cores()) != TRIPLES_OK) return rc;
    for (int p = 0; p < B.nprob; p++)
        if ((rc = prep_launches<float>(B.plans[p], st, B.ios[p])) != TRIPLES_OK) return rc;
    const char *tab = B.ws + B.tables_off;
    const bool bf16 = B.prec == TRIPLES_PRECISION_MIXED_BF16;
    for (const BatchStep &S : B.steps) {
        for (int g = 0; g < 2; g++) {
            if (S.f1_n[g] == 0) continue;
            const Table<F1Job> J{S.f1_n[g], (const int *)(tab + S.f1_start[g]), (const F1Job *)(tab + S.f1_jobs[g])};
            Plan W;   // only the tile width matters to the launch
            W.f1_bn = g == 0 ? 256 : 128;
            TB_KLAUNCH(P_F1, launch_f1(W, st, S.f1_tiles[g], J));
        }
        const Table<ChunkAux> X{S.naux, nullptr, (const ChunkAux *)(tab + S.aux)};
        TB_KLAUNCH(P_PREP, (k_chunk_scale<<<S.naux, 32, 0, st>>>(X)));
        const Table<F2M> F{S.naux, (const int *)(tab + S.f2_start), (const F2M *)(tab + S.f2_jobs)};
        TB_KLAUNCH(P_F2, launch_f2m(bf16, st, S.f2_items, F));
        TB_KLAUNCH(P_F2, (k_energy_sum<<<S.naux, 256, 0, st>>>(X, 1)));
        for (int k = 0; k < 4; k++) {
            const Table<TcB1Params> J{S.naux, (const int *)(tab + S.b1_start[k]), (const TcB1Params *)(tab + S.b1_jobs[k])};
            TB_KLAUNCH(kB1Cat[k], launch_b1(k, st, S.b1_tiles[k], J));
        }
    }
    for (int p = 0; p < B.nprob; p++)
        if ((rc = fold_launches(B.plans[p], st, B.ios[p])) != TRIPLES_OK) return rc;
    return TRIPLES_OK;
}

void profile_enable(int on) {
    g_prof = on != 0;
    g_prof_recs.clear();
    g_pool_used = 0;
}

int profile_read(int max_cats, double *ms, int *launches) {
    for (int c = 0; c < max_cats && c < P_NCAT; c++) {
        ms[c] = 0.0;
        launches[c] = 0;
    }
    for (const ProfRec &r : g_prof_recs) {
        float t = 0.f;
        if (cudaEventSynchronize(r.b) != cudaSuccess) return -1;
        cudaEventElapsedTime(&t, r.a, r.b);
        if (r.cat < max_cats) {
            ms[r.cat] += t;
            launches[r.cat] += 1;
        }
    }
    return P_NCAT;
}

const char *profile_name(int cat) { return (cat >= 0 && cat < P_NCAT) ? kProfNames[cat] : ""; }
int last_cuda_error() { return g_last_cuda_error; }
void set_last_cuda_error(int e) { g_last_cuda_error = e; }

}  // namespace tb

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

size_t triples_workspace_size(int precision, int nocc, int nvir, int ovvv_packed, int want_grad) {
    return triples_workspace_size_ex(precision, nocc, nvir, ovvv_packed, want_grad, nullptr);
}

size_t triples_workspace_size_ex(int precision, int nocc, int nvir, int ovvv_packed, int want_grad,
                                 const triples_options *opt) {
    tb::Plan P;
    if (tb::make_plan(precision, nocc, nvir, ovvv_packed, want_grad, P, 0, opt) != TRIPLES_OK) return 0;
    return P.total;
}

size_t triples_workspace_extra(int precision, int nocc, int nvir, int ovvv_packed, int want_grad,
                               const triples_options *opt) {
    tb::Plan P, Q;
    if (tb::make_plan(precision, nocc, nvir, ovvv_packed, want_grad, P, 0, opt) != TRIPLES_OK) return 0;
    if (tb::make_plan(precision, nocc, nvir, ovvv_packed, want_grad, Q, 0, opt, true, tb::kMaxGroup) != TRIPLES_OK) return 0;
    return Q.total > P.total ? Q.total - P.total : 0;
}

size_t triples_workspace_least(int precision, int nocc, int nvir, int ovvv_packed, int want_grad,
                               const triples_options *opt) {
    tb::Plan P;
    if (tb::make_plan(precision, nocc, nvir, ovvv_packed, want_grad, P, 0, opt, false) != TRIPLES_OK) return 0;
    return P.total;
}

// The kernels read and write the workspace in 16-byte pieces (vectors, bulk and tensor copies).
static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

static int triples_call(void *stream, int precision, int nocc, int nvir, int ovvv_packed, int want_grad,
                        const triples_options *opt, const tb::TriplesIO &io, size_t workspace_bytes) {
    tb::Plan P;
    int rc = tb::make_plan_for(precision, nocc, nvir, ovvv_packed, want_grad, P, opt, workspace_bytes);
    if (rc != TRIPLES_OK) return rc;
    if (!io.workspace || workspace_bytes < P.total) return TRIPLES_ERR_WORKSPACE;
    if (!aligned16(io.workspace)) return TRIPLES_ERR_INVALID_ARGUMENT;
    if (!io.mo_energy || !io.t1 || !io.t2 || !io.ovoo || !io.ovov || !io.ovvv || !io.fvo || !io.e_out)
        return TRIPLES_ERR_INVALID_ARGUMENT;
    if (want_grad && (!io.mo_energy_bar || !io.t1_bar || !io.t2_bar || !io.ovoo_bar || !io.ovov_bar ||
                      !io.ovvv_bar || !io.fvo_bar))
        return TRIPLES_ERR_INVALID_ARGUMENT;
    return tb::run_triples(P, (cudaStream_t)stream, io);
}

int triples_energy(void *stream, int precision, int nocc, int nvir, int ovvv_packed,
                   const double *mo_energy, const double *t1, const double *t2, const double *ovoo,
                   const double *ovov, const double *ovvv, const double *fvo, void *workspace,
                   size_t workspace_bytes, double *e_out) {
    tb::TriplesIO io{};
    io.mo_energy = mo_energy; io.t1 = t1; io.t2 = t2; io.ovoo = ovoo; io.ovov = ovov;
    io.ovvv = ovvv; io.fvo = fvo; io.ybar = 1.0; io.workspace = workspace; io.e_out = e_out;
    return triples_call(stream, precision, nocc, nvir, ovvv_packed, 0, nullptr, io, workspace_bytes);
}

int triples_energy_vjp(void *stream, int precision, int nocc, int nvir, int ovvv_packed,
                       const double *mo_energy, const double *t1, const double *t2, const double *ovoo,
                       const double *ovov, const double *ovvv, const double *fvo, double ybar,
                       void *workspace, size_t workspace_bytes, double *e_out, double *mo_energy_bar,
                       double *t1_bar, double *t2_bar, double *ovoo_bar, double *ovov_bar,
                       double *ovvv_bar, double *fvo_bar) {
    return triples_energy_vjp_ex(stream, precision, nocc, nvir, ovvv_packed, mo_energy, t1, t2, ovoo, ovov,
                                 ovvv, fvo, ybar, 1, nullptr, workspace, workspace_bytes, e_out, mo_energy_bar,
                                 t1_bar, t2_bar, ovoo_bar, ovov_bar, ovvv_bar, fvo_bar);
}

int triples_energy_vjp_ex(void *stream, int precision, int nocc, int nvir, int ovvv_packed,
                          const double *mo_energy, const double *t1, const double *t2, const double *ovoo,
                          const double *ovov, const double *ovvv, const double *fvo, double ybar,
                          int want_grad, const triples_options *opt, void *workspace, size_t workspace_bytes,
                          double *e_out, double *mo_energy_bar, double *t1_bar, double *t2_bar,
                          double *ovoo_bar, double *ovov_bar, double *ovvv_bar, double *fvo_bar) {
    tb::TriplesIO io{};
    io.mo_energy = mo_energy; io.t1 = t1; io.t2 = t2; io.ovoo = ovoo; io.ovov = ovov;
    io.ovvv = ovvv; io.fvo = fvo; io.ybar = want_grad ? ybar : 1.0; io.workspace = workspace; io.e_out = e_out;
    if (want_grad) {
        io.mo_energy_bar = mo_energy_bar; io.t1_bar = t1_bar; io.t2_bar = t2_bar; io.ovoo_bar = ovoo_bar;
        io.ovov_bar = ovov_bar; io.ovvv_bar = ovvv_bar; io.fvo_bar = fvo_bar;
    }
    return triples_call(stream, precision, nocc, nvir, ovvv_packed, want_grad ? 1 : 0, opt, io, workspace_bytes);
}

// ---- LNO (projected) energy ----
size_t triples_lno_workspace_size(int precision, int nocc, int nvir, int ovvv_packed, int want_grad) {
    return triples_lno_workspace_size_ex(precision, nocc, nvir, ovvv_packed, want_grad, nullptr);
}

size_t triples_lno_workspace_size_ex(int precision, int nocc, int nvir, int ovvv_packed, int want_grad,
                                     const triples_options *opt) {
    tb::Plan P;
    if (tb::make_plan(precision, nocc, nvir, ovvv_packed, want_grad, P, 1, opt) != TRIPLES_OK) return 0;
    return P.total;
}

static int triples_lno_call(void *stream, int precision, int nocc, int nvir, int ovvv_packed, int want_grad,
                            const triples_options *opt, const tb::TriplesIO &io, size_t workspace_bytes) {
    tb::Plan P;
    int rc = tb::make_plan(precision, nocc, nvir, ovvv_packed, want_grad, P, 1, opt);
    if (rc != TRIPLES_OK) return rc;
    if (!io.workspace || workspace_bytes < P.total) return TRIPLES_ERR_WORKSPACE;
    if (!aligned16(io.workspace)) return TRIPLES_ERR_INVALID_ARGUMENT;
    if (!io.mat || !io.mo_energy || !io.t1 || !io.t2 || !io.ovoo || !io.ovov || !io.ovvv || !io.fvo || !io.e_out)
        return TRIPLES_ERR_INVALID_ARGUMENT;
    if (want_grad && (!io.mat_bar || !io.mo_energy_bar || !io.t1_bar || !io.t2_bar || !io.ovoo_bar ||
                      !io.ovov_bar || !io.ovvv_bar || !io.fvo_bar))
        return TRIPLES_ERR_INVALID_ARGUMENT;
    return tb::run_triples(P, (cudaStream_t)stream, io);
}

int triples_lno_energy(void *stream, int precision, int nocc, int nvir, int ovvv_packed, const double *mat,
                       const double *mo_energy, const double *t1, const double *t2, const double *ovoo,
                       const double *ovov, const double *ovvv, const double *fvo, void *workspace,
                       size_t workspace_bytes, double *e_out) {
    return triples_lno_energy_vjp_ex(stream, precision, nocc, nvir, ovvv_packed, mat, mo_energy, t1, t2, ovoo, ovov,
                                     ovvv, fvo, 1.0, 0, nullptr, workspace, workspace_bytes, e_out, nullptr,
                                     nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
}

int triples_lno_energy_vjp(void *stream, int precision, int nocc, int nvir, int ovvv_packed, const double *mat,
                           const double *mo_energy, const double *t1, const double *t2, const double *ovoo,
                           const double *ovov, const double *ovvv, const double *fvo, double ybar,
                           void *workspace, size_t workspace_bytes, double *e_out, double *mat_bar,
                           double *mo_energy_bar, double *t1_bar, double *t2_bar, double *ovoo_bar,
                           double *ovov_bar, double *ovvv_bar, double *fvo_bar) {
    return triples_lno_energy_vjp_ex(stream, precision, nocc, nvir, ovvv_packed, mat, mo_energy, t1, t2, ovoo, ovov,
                                     ovvv, fvo, ybar, 1, nullptr, workspace, workspace_bytes, e_out, mat_bar,
                                     mo_energy_bar, t1_bar, t2_bar, ovoo_bar, ovov_bar, ovvv_bar, fvo_bar);
}

int triples_lno_energy_vjp_ex(void *stream, int precision, int nocc, int nvir, int ovvv_packed, const double *mat,
                              const double *mo_energy, const double *t1, const double *t2, const double *ovoo,
                              const double *ovov, const double *ovvv, const double *fvo, double ybar,
                              int want_grad, const triples_options *opt, void *workspace, size_t workspace_bytes,
                              double *e_out, double *mat_bar, double *mo_energy_bar, double *t1_bar,
                              double *t2_bar, double *ovoo_bar, double *ovov_bar, double *ovvv_bar,
                              double *fvo_bar) {
    tb::TriplesIO io{};
    io.mat = mat;
    io.mo_energy = mo_energy; io.t1 = t1; io.t2 = t2; io.ovoo = ovoo; io.ovov = ovov;
    io.ovvv = ovvv; io.fvo = fvo; io.ybar = want_grad ? ybar : 1.0; io.workspace = workspace; io.e_out = e_out;
    if (want_grad) {
        io.mat_bar = mat_bar;
        io.mo_energy_bar = mo_energy_bar; io.t1_bar = t1_bar; io.t2_bar = t2_bar; io.ovoo_bar = ovoo_bar;
        io.ovov_bar = ovov_bar; io.ovvv_bar = ovvv_bar; io.fvo_bar = fvo_bar;
    }
    return triples_lno_call(stream, precision, nocc, nvir, ovvv_packed, want_grad ? 1 : 0, opt, io,
                            workspace_bytes);
}

// ---- LNO host tables (introspection) ----
size_t triples_lno_tables(void *out, size_t bytes) {
    const size_t need = sizeof(tb::LnoTables) + 16 * sizeof(tb::LnoPattern);
    if (out && bytes >= need) {
        tb::LnoTables t;
        tb::LnoPattern pats[16];
        tb::lno_build_tables(t);
        tb::lno_build_patterns(pats);
        std::memcpy(out, &t, sizeof(t));
        std::memcpy((char *)out + sizeof(t), pats, sizeof(pats));
    }
    return need;
}

// ---- density-fitted ERI producer ----
// ovvv[(p,x), pair] = sum_P Lov[P,(p,x)] Lvv[P,pair]  (pyscfad/cc/dfccsd.py:77-88), packed
// pairs f >= y at f(f+1)/2 + y, built on the device by one FP64 GEMM; the (T)
// path then runs on it with packed ovvv, and the packed ovvv cotangent maps
// back to
//   Lov_bar[P,(p,x)] = sum_pair ovvv_bar[(p,x),pair] Lvv[P,pair]
//   Lvv_bar[P,pair]  = sum_(p,x) ovvv_bar[(p,x),pair] Lov[P,(p,x)]
// (two more GEMMs, the same FP64 tile as the FP64 contractions).
struct DfLayout {
    tb::Plan P;
    size_t off_ovvv, off_gvvv, total;
};

// workspace_bytes: what the caller has (SIZE_MAX: the size to ask for)
static int df_layout(int precision, int nocc, int nvir, int naux, int want_grad, DfLayout &L, size_t workspace_bytes) {
    if (naux < 1) return TRIPLES_ERR_INVALID_ARGUMENT;
    const size_t nov = (size_t)nocc * nvir, npair = (size_t)nvir * (nvir + 1) / 2;
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t own = al(nov * npair * sizeof(double)) * (want_grad ? 2 : 1);
    int rc;
    if (workspace_bytes == SIZE_MAX)
        rc = tb::make_plan(precision, nocc, nvir, 1, want_grad, L.P);
    else
        rc = tb::make_plan_for(precision, nocc, nvir, 1, want_grad, L.P, nullptr,
                               workspace_bytes > own ? workspace_bytes - own : 0);
    if (rc != TRIPLES_OK) return rc;
    L.off_ovvv = al(L.P.total);
    L.off_gvvv = L.off_ovvv + al(nov * npair * sizeof(double));
    L.total = L.off_ovvv + own;
    return TRIPLES_OK;
}

size_t triples_df_workspace_size(int precision, int nocc, int nvir, int naux, int want_grad) {
    DfLayout L;
    if (df_layout(precision, nocc, nvir, naux, want_grad, L, SIZE_MAX) != TRIPLES_OK) return 0;
    return L.total;
}

static int triples_df_call(void *stream, int precision, int nocc, int nvir, int naux, int want_grad,
                           const double *Lov, const double *Lvv, tb::TriplesIO io, size_t workspace_bytes,
                           double *Lov_bar, double *Lvv_bar) {
    DfLayout L;
    int rc = df_layout(precision, nocc, nvir, naux, want_grad, L, workspace_bytes);
    if (rc != TRIPLES_OK) return rc;
    if (!io.workspace || workspace_bytes < L.total) return TRIPLES_ERR_WORKSPACE;
    if (!aligned16(io.workspace)) return TRIPLES_ERR_INVALID_ARGUMENT;
    if (!Lov || !Lvv || !io.mo_energy || !io.t1 || !io.t2 || !io.ovoo || !io.ovov || !io.fvo || !io.e_out)
        return TRIPLES_ERR_INVALID_ARGUMENT;
    if (want_grad && (!Lov_bar || !Lvv_bar || !io.mo_energy_bar || !io.t1_bar || !io.t2_bar || !io.ovoo_bar ||
                      !io.ovov_bar || !io.fvo_bar))
        return TRIPLES_ERR_INVALID_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    char *ws = (char *)io.workspace;
    double *ovvv = (double *)(ws + L.off_ovvv), *gvvv = (double *)(ws + L.off_gvvv);
    const long long nov = (long long)nocc * nvir, npair = (long long)nvir * (nvir + 1) / 2;
    // ovvv[px][pair] = sum_P Lov[P][px] Lvv[P][pair]
    if ((rc = tb::gemm_plain<false, false>(st, (int)nov, (int)npair, naux, Lov, 1, nov, Lvv, 1, npair, ovvv, npair, 1)) !=
        TRIPLES_OK)
        return rc;
    io.ovvv = ovvv;
    io.ovvv_bar = want_grad ? gvvv : nullptr;
    if ((rc = tb::run_triples(L.P, st, io)) != TRIPLES_OK) return rc;
    if (!want_grad) return TRIPLES_OK;
    // Lov_bar[P][px] = sum_pair G[px][pair] Lvv[P][pair]
    if ((rc = tb::gemm_plain<true, true>(st, (int)nov, naux, (int)npair, gvvv, npair, 1, Lvv, npair, 1, Lov_bar, 1, nov)) !=
        TRIPLES_OK)
        return rc;
    // Lvv_bar[P][pair] = sum_px G[px][pair] Lov[P][px]
    return tb::gemm_plain<false, true>(st, (int)npair, naux, (int)nov, gvvv, 1, npair, Lov, nov, 1, Lvv_bar, 1, npair);
}

int triples_energy_df(void *stream, int precision, int nocc, int nvir, int naux, const double *mo_energy,
                      const double *t1, const double *t2, const double *ovoo, const double *ovov, const double *Lov,
                      const double *Lvv, const double *fvo, void *workspace, size_t workspace_bytes, double *e_out) {
    tb::TriplesIO io{};
    io.mo_energy = mo_energy; io.t1 = t1; io.t2 = t2; io.ovoo = ovoo; io.ovov = ovov;
    io.fvo = fvo; io.ybar = 1.0; io.workspace = workspace; io.e_out = e_out;
    return triples_df_call(stream, precision, nocc, nvir, naux, 0, Lov, Lvv, io, workspace_bytes, nullptr, nullptr);
}

int triples_energy_vjp_df(void *stream, int precision, int nocc, int nvir, int naux, const double *mo_energy,
                          const double *t1, const double *t2, const double *ovoo, const double *ovov,
                          const double *Lov, const double *Lvv, const double *fvo, double ybar, void *workspace,
                          size_t workspace_bytes, double *e_out, double *mo_energy_bar, double *t1_bar,
                          double *t2_bar, double *ovoo_bar, double *ovov_bar, double *Lov_bar, double *Lvv_bar,
                          double *fvo_bar) {
    tb::TriplesIO io{};
    io.mo_energy = mo_energy; io.t1 = t1; io.t2 = t2; io.ovoo = ovoo; io.ovov = ovov;
    io.fvo = fvo; io.ybar = ybar; io.workspace = workspace; io.e_out = e_out;
    io.mo_energy_bar = mo_energy_bar; io.t1_bar = t1_bar; io.t2_bar = t2_bar; io.ovoo_bar = ovoo_bar;
    io.ovov_bar = ovov_bar; io.fvo_bar = fvo_bar;
    return triples_df_call(stream, precision, nocc, nvir, naux, 1, Lov, Lvv, io, workspace_bytes, Lov_bar, Lvv_bar);
}

// Fixed scratch for callers that may not allocate device memory themselves
// (for example code running inside another framework's memory pool or a
// host program that must keep its device footprint fixed).  Every device
// that loads this library holds the array until the process exits.  The
// call clears what must start at zero (its control block and gradient
// accumulators) on each use, so the last call's leftovers do no harm; two
// calls whose GPU work overlaps share the array and race.
static constexpr size_t kStaticScratchBytes = TRIPLES_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
static constexpr int kStaticMaxDevices = 64;
// Device address of the array per device, looked up once with that device
// current.  Host threads making their first call on a device at the same
// time both store the same address; the cache assumes the device's primary
// context lives as long as the process.
static std::atomic<void *> g_static_scratch_addr[kStaticMaxDevices];

static int static_scratch_address(void **addr_out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        tb::set_last_cuda_error((int)e);
        return TRIPLES_ERR_CUDA;
    }
    if (dev < 0 || dev >= kStaticMaxDevices) return TRIPLES_ERR_UNSUPPORTED;
    void *addr = g_static_scratch_addr[dev].load(std::memory_order_acquire);
    if (addr == nullptr) {
        // the array's host-side name is only a stand-in for the symbol
        e = cudaGetSymbolAddress(&addr, g_static_scratch);
        if (e != cudaSuccess || addr == nullptr) {
            tb::set_last_cuda_error((int)e);
            return TRIPLES_ERR_CUDA;
        }
        g_static_scratch_addr[dev].store(addr, std::memory_order_release);
    }
    *addr_out = addr;
    return TRIPLES_OK;
}

int triples_energy_vjp_static(void *stream, int precision, int nocc, int nvir, int ovvv_packed,
                              const double *mo_energy, const double *t1, const double *t2,
                              const double *ovoo, const double *ovov, const double *ovvv,
                              const double *fvo, double ybar, double *e_out, double *mo_energy_bar,
                              double *t1_bar, double *t2_bar, double *ovoo_bar, double *ovov_bar,
                              double *ovvv_bar, double *fvo_bar) {
    const size_t need = triples_workspace_size(precision, nocc, nvir, ovvv_packed, 1);
    if (need == 0) return TRIPLES_ERR_INVALID_ARGUMENT;
    if (need > kStaticScratchBytes) return TRIPLES_ERR_WORKSPACE;   // problem too large for the fixed scratch
    void *scratch = nullptr;
    const int rc = static_scratch_address(&scratch);
    if (rc != TRIPLES_OK) return rc;
    return triples_energy_vjp(stream, precision, nocc, nvir, ovvv_packed, mo_energy, t1, t2, ovoo, ovov, ovvv,
                              fvo, ybar, scratch, kStaticScratchBytes, e_out, mo_energy_bar, t1_bar, t2_bar,
                              ovoo_bar, ovov_bar, ovvv_bar, fvo_bar);
}

int triples_static_scratch(void **ptr, size_t *bytes) {
    if (!ptr) return TRIPLES_ERR_INVALID_ARGUMENT;
    const int rc = static_scratch_address(ptr);
    if (rc == TRIPLES_OK && bytes) *bytes = kStaticScratchBytes;
    return rc;
}

int triples_static_check_device_status(void *stream) {
    void *scratch = nullptr;
    const int rc = static_scratch_address(&scratch);
    if (rc != TRIPLES_OK) return rc;
    return triples_check_device_status(stream, scratch);
}

int triples_check_device_status(void *stream, const void *workspace) {
    if (!workspace) return TRIPLES_ERR_INVALID_ARGUMENT;
    tb::Ctrl c;
    cudaError_t e = cudaMemcpyAsync(&c, workspace, sizeof(c), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) {
        tb::set_last_cuda_error((int)e);
        return TRIPLES_ERR_CUDA;
    }
    return c.err ? TRIPLES_ERR_DEVICE_TIMEOUT : TRIPLES_OK;
}

// ---- batched calls ----
struct triples_batch {
    tb::Batch b;
};

size_t triples_batch_workspace_size(int precision, int nprob, const triples_problem *probs) {
    tb::Batch B;
    if (tb::batch_build(B, precision, nprob, probs, 1.0, nullptr, true) != TRIPLES_OK) return 0;
    return B.total;
}

size_t triples_batch_workspace_least(int precision, int nprob, const triples_problem *probs) {
    tb::Batch B;
    if (tb::batch_build(B, precision, nprob, probs, 1.0, nullptr, false) != TRIPLES_OK) return 0;
    return B.total;
}

int triples_batch_create(int precision, int nprob, const triples_problem *probs, double ybar, void *workspace,
                         size_t workspace_bytes, triples_batch **batch) {
    if (!batch) return TRIPLES_ERR_INVALID_ARGUMENT;
    *batch = nullptr;
    if (!workspace) return TRIPLES_ERR_WORKSPACE;
    if (!aligned16(workspace)) return TRIPLES_ERR_INVALID_ARGUMENT;
    // the workspace must hold the batch before any table points into it
    bool vtables = true;
    for (;; vtables = false) {
        tb::Batch sizing;
        const int rc = tb::batch_build(sizing, precision, nprob, probs, ybar, nullptr, vtables);
        if (rc != TRIPLES_OK) return rc;
        if (workspace_bytes >= sizing.total) break;
        if (!vtables) return TRIPLES_ERR_WORKSPACE;
    }
    triples_batch *h = new (std::nothrow) triples_batch;
    if (!h) return TRIPLES_ERR_INVALID_ARGUMENT;
    h->b.ws = (char *)workspace;
    std::vector<char> image;
    int rc = tb::batch_build(h->b, precision, nprob, probs, ybar, &image, vtables);
    if (rc == TRIPLES_OK && !image.empty()) {
        const cudaError_t e = cudaMemcpy(h->b.ws + h->b.tables_off, image.data(), image.size(), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            tb::set_last_cuda_error((int)e);
            rc = TRIPLES_ERR_CUDA;
        }
    }
    if (rc != TRIPLES_OK) {
        delete h;
        return rc;
    }
    *batch = h;
    return TRIPLES_OK;
}

int triples_batch_run(triples_batch *batch, void *stream) {
    if (!batch) return TRIPLES_ERR_INVALID_ARGUMENT;
    return tb::run_batch(batch->b, (cudaStream_t)stream);
}

int triples_batch_check_device_status(triples_batch *batch, void *stream) {
    if (!batch) return TRIPLES_ERR_INVALID_ARGUMENT;
    int status = TRIPLES_OK;
    for (int p = 0; p < batch->b.nprob; p++) {
        const int rc = triples_check_device_status(stream, batch->b.ws + batch->b.ws_off[p]);
        if (rc == TRIPLES_ERR_CUDA) return rc;
        if (rc != TRIPLES_OK) status = rc;
    }
    return status;
}

void triples_batch_destroy(triples_batch *batch) { delete batch; }

const char *triples_status_string(int status) {
    switch (status) {
    case TRIPLES_OK: return "ok";
    case TRIPLES_ERR_INVALID_ARGUMENT: return "invalid argument";
    case TRIPLES_ERR_WORKSPACE: return "workspace too small";
    case TRIPLES_ERR_CUDA: return "CUDA error";
    case TRIPLES_ERR_UNSUPPORTED: return "unsupported precision or device";
    case TRIPLES_ERR_DEVICE_TIMEOUT: return "device-side wait timed out";
    default: return "unknown status";
    }
}

int triples_last_cuda_error(void) { return tb::last_cuda_error(); }

const char *triples_version(void) { return "0.1.0"; }

void triples_profile_enable(int on) { tb::profile_enable(on); }

int triples_profile_read(int max_categories, double *ms, int *launches) {
    if (max_categories < 0 || (max_categories > 0 && (!ms || !launches))) return -1;
    return tb::profile_read(max_categories, ms, launches);
}

const char *triples_profile_name(int category) { return tb::profile_name(category); }

}  // extern "C"
