// Internal planning structures shared by the (T) drivers.
#pragma once
#include <cstddef>

#include "common.cuh"
#include "pyscfad_b200.h"

namespace tb {

constexpr int kMaxTv = 16;        // largest virtual block
constexpr int kMaxPartials = 32;  // energy partials per occupied representative: 8 sub-range triples, or 4 of 8 warps
constexpr int kMaxCols = 1024;    // largest nocc * Tv (one staged (r, z) row)
constexpr int kCtrlBytes = 256;   // control block at workspace offset 0
// Chunk slots of a call: most bytes of staging and Wbar.  A chunk of nocc 5 has
// a few tens of tiles per kernel, one of nocc 13 fills the chip once or twice
// with a nearly empty last wave; from nocc 20 (1.6 GB a chunk) on a chunk is
// enough alone.  One chunk at a time / within 1 GB / within 2 GB, E + VJP: nocc
// 5 nvir 19 mixed 1.26 / 0.45 / 0.45 ms, FP64 kernels 0.95 / 0.45 / 0.45 ms, nocc
// 13 nvir 83 bf16 41.4 / 35.2 / 33.0 ms, nocc 12 nvir 100 FP64 112 / 112 / 104 ms.
constexpr size_t kGroupBytes = (size_t)2 << 30;
constexpr int kLnoGrid = 1024;    // LNO projection: most blocks (an energy partial each and slot)
constexpr int kLnoArrays = 4;     // LNO box arrays (with the adjoint)
constexpr double kLnoBudgetBytes = 96e9;   // block size rule of the LNO plan (plan_once)

// State of one chunk slot
struct ChunkSlot {
    double wscale;                // power-of-two scale of the split Wbar
    unsigned wmax_bits;           // bit pattern of max |W| (F1)
    unsigned ticket;              // work items handed out by the mixed epilogue (first slot of a launch)
};

// Control block (workspace offset 0)
struct Ctrl {
    int err;                      // device-side error bits: bounded waits that gave up (1, 2, 4: W contraction's
                                  // producer, MMA, epilogue; 8, 16, 32: adjoint contractions'; 64: mixed
                                  // epilogue), 128: misaligned shared memory of the adjoint contractions
    double e_acc;                 // E(T) accumulator
    double scale[2];              // operand scales (A: ovvv/ovoo, B: t2), powers of two
    float out_scale;              // 1 / (scale[0] * scale[1])
    float pad_;
    unsigned long long absmax[6]; // bit patterns of max |ovvv|, |ovoo|, |t2|, |ovov|, |t1|, |fvo|
    double lno_norm[2];           // LNO projector: max abs row sum, max abs column sum
    ChunkSlot slot[kMaxGroup];
};

static_assert(sizeof(Ctrl) <= kCtrlBytes, "control block too large");

struct Plan {
    Dims d;
    int a0, a1;      // chunk slice by largest virtual block (a1 <= 0: no upper bound)
    int kseg;        // 64-wide K blocks per FP32 accumulation segment (mixed precision)
    int f1_bn;       // widest N tile of the tensor-core W contraction (128 or 256)
    int f1_rt;       // occupied r values of its N tiles (16 columns each)
    int prec, want_grad, packed;
    int lno;         // projected (LNO) energy: box arrays off_L
    int nb;          // number of virtual blocks
    int n_ijk;       // occupied triplet representatives i >= j >= k
    int Kp8, Op8;    // 16-byte padded contraction lengths of the 16-bit operands
    size_t stage_elems, stage_bytes, wbar_elems;
    size_t stage_slot, wbar_slot;   // elements from one chunk slot to the next
    size_t off_ctrl;
    size_t off_A1, off_B1, off_A2, off_B2, off_S, off_SW;
    size_t off_A1h, off_B1h, off_A2h, off_B2h;
    size_t off_GA1, off_GB1, off_GA2, off_GB2;
    int group;       // chunk slots: chunks whose kernels run in one launch each
    bool vtables;    // the workspace holds the epilogue's FP32 V-term tables
    size_t off_ot, off_tf;
    size_t off_ijk, off_epart;
    size_t off_L[4], off_lpart;
    size_t total;
};

struct TriplesIO {
    const double *mo_energy, *t1, *t2, *ovoo, *ovov, *ovvv, *fvo;
    const double *mat;             // LNO projector [o,o] (lno plans only)
    double ybar;
    void *workspace;
    double *e_out;
    double *mo_energy_bar, *t1_bar, *t2_bar, *ovoo_bar, *ovov_bar, *ovvv_bar, *fvo_bar;
    double *mat_bar;
};

int make_plan(int precision, int nocc, int nvir, int packed, int want_grad, Plan &P, int lno = 0,
              const triples_options *opt = nullptr, bool vtables = true, int most_group = 1);
int make_plan_for(int precision, int nocc, int nvir, int packed, int want_grad, Plan &P, const triples_options *opt,
                  size_t workspace_bytes);
int run_triples(const Plan &P, cudaStream_t st, const TriplesIO &io);

}  // namespace tb
