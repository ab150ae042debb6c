// Shared definitions for the (T) kernels.
//
// Index conventions (o = nocc, v = nvir, Kp = padded virtual length of the
// contraction axis):
//   raw triples amplitude, the quantity the reference builds per job in
//   get_wv (pyscfadlib/pyscfadlib/vjp/cc/ccsd_t.c:121-152):
//     w^{pqr}_{xyz} = sum_f ovvv[p,x,f,y] t2[r,q,z,f] - sum_m ovoo[p,x,m,q] t2[r,m,z,y]
//     v^{pqr}_{xyz} = ovov[p,x,q,y] t1[r,z] + t2[q,p,y,x] fvo[z,r]
//   Device operand layouts built once per call (prep kernels):
//     A1[y][p][x][f] = ovvv[p,x,f,y]     B1[q][r][z][f] = t2[r,q,z,f]
//     A2[q][p][x][m] = ovoo[p,x,m,q]     B2[y][r][z][m] = t2[r,m,z,y]
//   so that, for fixed (y,q), w is the two-term GEMM
//     W[(p,x),(r,z)] = A1[y][(p,x),:] . B1[q][(r,z),:]^T - A2[q][(p,x),:] . B2[y][(r,z),:]^T
//
// Work is split into "chunks": a triple of virtual blocks A >= B >= C (block
// size Tv) together with ALL occupied indices.  A chunk is closed under the
// simultaneous (occupied, virtual) index permutations that couple raw
// amplitudes in the energy, so its epilogue needs nothing outside the chunk.
// For each distinct ordering tau = (X,Y,Z) of (A,B,C) the raw amplitudes are
// staged as S_tau[p][q][y][x][r][z] (x in X, y in Y, z in Z, local indices).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tb {

constexpr int kBig = 1 << 30;

// idx -> (i0,i1,i2,i3), i0 = idx % e0, i1 = (idx/e0) % e1, i2 = (idx/e0/e1) % e2,
// i3 = rest; offset = sum i_k * s_k (elements).
struct Map4 {
    int e0, e1, e2;
    long long s0, s1, s2, s3;
};

__host__ __device__ inline Map4 map1(long long s0) { return Map4{kBig, 1, 1, s0, 0, 0, 0}; }
__host__ __device__ inline Map4 map2(int e0, long long s0, long long s1) {
    return Map4{e0, kBig, 1, s0, s1, 0, 0};
}
__host__ __device__ inline Map4 map3(int e0, int e1, long long s0, long long s1, long long s2) {
    return Map4{e0, e1, kBig, s0, s1, s2, 0};
}
__device__ __forceinline__ long long apply(const Map4 &m, int idx) {
    int i0 = idx % m.e0;
    int t = idx / m.e0;
    int i1 = t % m.e1;
    t /= m.e1;
    int i2 = t % m.e2;
    int i3 = t / m.e2;
    return (long long)i0 * m.s0 + (long long)i1 * m.s1 + (long long)i2 * m.s2 +
           (long long)i3 * m.s3;
}

// One distinct ordering (X,Y,Z) of a chunk's virtual blocks.
struct PermBlock {
    int bx, by, bz;        // block indices
    int X0, Tx, Y0, Ty, Z0, Tz;
    long long soff;        // offset of S_tau in the staging buffer (elements)
    int rzp;               // o*Tz rounded up to 8 (16-byte rows of 16-bit Wbar)
    long long swoff;       // offset of Wbar_tau (values) in the Wbar buffer
};

// *p += v in global memory.  atomicAdd through a pointer that the compiler does not
// know to be global (one read from a job table or from shared memory) first tests for
// shared memory and carries the code for it: 265 to 242 ms of the mixed epilogue at
// nocc 20 nvir 180.
__device__ __forceinline__ void red_add(double *p, double v) {
    asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "d"(v) : "memory");
}

// 16-bit Wbar_tau: blocks of at least 8 x values are stored as 8 x 8 tiles
// [h][y][q][p][x / 8][rz / 8][x % 8][rz % 8] (rz = r Tz + z), smaller ones as rows
// [h][y][p][x][q][rz].  A tile is one 128-byte line, the 8 z runs of eight x that
// one epilogue region holds for a y: as rows they were 16-byte halves of 32-byte
// sectors whose other half came from another work item.  It is also a core
// matrix of the adjoint contractions' first operand, K- or MN-major.
__host__ __device__ inline bool wbar_tiled(const PermBlock &pb) { return pb.Tx >= 8; }

struct ChunkDesc {
    int nperm;
    int blk[3];            // A >= B >= C block indices
    int nabc[3];           // sizes of blocks A, B, C
    int base[3];           // first virtual index of A, B, C
    PermBlock pb[6];
};

struct Dims {
    int o, v, n, Kp, Tv;   // Tv: power-of-two block size
};

// Virtual blocks: v / Tv full blocks of Tv, then the remainder split into
// descending powers of two (so every block size divides 64).
__host__ __device__ inline int num_blocks(const Dims &d) {
    int nfull = d.v / d.Tv, rem = d.v - nfull * d.Tv, n = nfull;
    for (int bit = d.Tv >> 1; bit > 0; bit >>= 1)
        if (rem & bit) n++;
    return n;
}
__host__ __device__ inline int block_size(const Dims &d, int b) {
    int nfull = d.v / d.Tv;
    if (b < nfull) return d.Tv;
    int rem = d.v - nfull * d.Tv, k = b - nfull;
    for (int bit = d.Tv >> 1; bit > 0; bit >>= 1)
        if (rem & bit) {
            if (k == 0) return bit;
            --k;
        }
    return 0;
}
__host__ __device__ inline int block_start(const Dims &d, int b) {
    int nfull = d.v / d.Tv;
    if (b <= nfull) return b * d.Tv;
    int s = nfull * d.Tv, rem = d.v - s, k = b - nfull;
    for (int bit = d.Tv >> 1; bit > 0; bit >>= 1)
        if (rem & bit) {
            if (k == 0) return s;
            s += bit;
            --k;
        }
    return s;
}

// The six orderings of three slots, lexicographic: index = 2*first + (second is
// the larger of the two remaining).
__host__ __device__ constexpr inline void perm_of(int s, int out[3]) {
    const int first = s >> 1;
    const int lo = (first == 0) ? 1 : 0;
    const int hi = (first == 2) ? 1 : 2;
    out[0] = first;
    out[1] = (s & 1) ? hi : lo;
    out[2] = (s & 1) ? lo : hi;
}

__host__ __device__ constexpr inline int perm_index(int a, int b) {
    int lo = (a == 0) ? 1 : 0;  // smallest remaining slot
    return 2 * a + (b == lo ? 0 : 1);
}

// index of the ordering t -> P[s][P[pi][t]]
__host__ __device__ constexpr inline int perm_compose(int s, int pi) {
    int ps[3] = {0, 0, 0}, pp[3] = {0, 0, 0};
    perm_of(s, ps);
    perm_of(pi, pp);
    return perm_index(ps[pp[0]], ps[pp[1]]);
}

// Staging layout of the mixed epilogue: S_tau[p][q][r][y block][x block][z block]
// and, inside a block of (ey, ex, ez) = (min(8, Ty), ...) values, [y][x][z];
// rows of 64 values (ex = ez = 8) are stored with bit 2 of the slot x*8+z
// exchanged by y's bit 0 and bit 4 by y's bit 1.  Block sizes are powers of
// two up to 16, so a block of fewer than 8 is one block.
__host__ __device__ inline int f2m_row_swizzle(int y) { return ((y & 1) << 2) | ((y & 2) << 3); }

struct StageRow {         // the z run of one (p, q, y, x): offset of r, z = base + r rs + z part
    long long base;
    int rs, ez, es, slot, swz;   // stride of r, z extent and size of a block, slot of z = 0, exchange
    __host__ __device__ int at(int z) const { return (z >> 3) * es + ((slot + (z & 7)) ^ swz); }
};

__host__ __device__ inline StageRow f2m_stage_row(const PermBlock &pb, int o, int p, int q, int y, int x) {
    const int ex = pb.Tx < 8 ? pb.Tx : 8, ey = pb.Ty < 8 ? pb.Ty : 8, ez = pb.Tz < 8 ? pb.Tz : 8;
    const int nx = pb.Tx > 8 ? 2 : 1, nz = pb.Tz > 8 ? 2 : 1;
    StageRow R;
    R.ez = ez;
    R.es = ex * ey * ez;
    R.rs = pb.Tx * pb.Ty * pb.Tz;
    R.slot = (x & 7) * ez;
    R.swz = (ex == 8 && ez == 8) ? f2m_row_swizzle(y & 7) : 0;
    R.base = pb.soff + (long long)(p * o + q) * o * R.rs + ((y >> 3) * nx + (x >> 3)) * nz * R.es + (y & 7) * (ex * ez);
    return R;
}

__host__ __device__ inline long long f2m_stage_offset(const PermBlock &pb, int o, int p, int q, int r, int y, int x,
                                                      int z) {
    const StageRow R = f2m_stage_row(pb, o, p, q, y, x);
    return R.base + (long long)r * R.rs + R.at(z);
}

// The jobs of one launch: chunks of one problem by value (Group), or chunks of
// many problems in device memory (Table).  Work units (tiles, items) are
// numbered job after job: job j has [start[j], start[j + 1]).  Group<T, 1> is
// the single-chunk kernel, its parameters compile-time constant addresses.
constexpr int kMaxGroup = 8;

template <typename T, int N>
struct Group {
    static constexpr bool kOne = N == 1;
    int n;
    int start[N + 1];
    T job[N];
};

template <typename T>
struct Table {
    static constexpr bool kOne = false;
    int n;
    const int *start;
    const T *job;
};

// Job of unit t, for a caller whose t only grows: a binary search once, then
// the index moves forward.
struct JobCursor {
    int j = -1;
    template <typename JOBS>
    __device__ __forceinline__ int at(const JOBS &J, int t, int &local) {
        if constexpr (JOBS::kOne) {
            local = t;
            return 0;
        } else {
            if (j < 0) {
                int lo = 0, hi = J.n - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (J.start[mid] <= t) lo = mid;
                    else hi = mid - 1;
                }
                j = lo;
            }
            while (j + 1 < J.n && J.start[j + 1] <= t) j++;
            local = t - J.start[j];
            return j;
        }
    }
};

}  // namespace tb
