// Host-side launchers of the statevector kernels (kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "engine.h"

namespace qsv {

constexpr int EXPECT_BATCH = 8;     // Pauli terms of one flip mask reduced per kernel launch
constexpr int EXPECT_Z_BATCH = 16;  // Z-only terms (24 more would not fit the accumulators in 128 registers)
constexpr int REDUCE_BLOCKS = 152 * 4;

bool pass_shape_supported(int precision, int T, int R);
// Shape of a pass kind (0 one-state, 1 two-state reverse sweep) for n qubits:
// the autotuned one if set, else the built-in default.
void resolve_shape(int arith, int kind, int n, int* T, int* R);
bool set_tuned_shape(int arith, int kind, int n, int T, int R);
// One-state shape of a batch group's forward plan (T = 0 asked for): the tuned
// one if set; else the default, but (12, 4) for complex64 groups of at most 14
// qubits (6 layers, 2048 items: 12 qubits 334 us, 3.6 ms on the whole-state
// kernel of a 13-qubit tile; 14 qubits 1185 us, 1236 at (13, 5)) and for those
// that fill less than one tile of 13 qubits an SM (19 items of 15 qubits: 72 us,
// 87 at (13, 5)).  Larger ones have fewer passes at (13, 5): 1024 items of 16
// qubits, 12 layers, 3.99 ms, 4.36 at (12, 4).
void batch_forward_shape(int arith, int n, int64_t items, int* T, int* R);
bool pass_shape_c128(int T, int R);
bool pass_shape_c64(int T, int R);
bool pass_shape_ds(int T, int R);
bool pass_shape_ds_r5(int T, int R);  // pass_ds_r5.cu
cudaError_t launch_pass_ds(int T, int R, void* state, const PassDesc* dpass, const StepDesc* dsteps,
                           const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride,
                            const uint8_t* active, cudaStream_t st);
cudaError_t launch_pass_ds_r5(int T, int R, void* state, const PassDesc* dpass, const StepDesc* dsteps,
                              const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride,
                              const uint8_t* active, cudaStream_t st);
cudaError_t launch_pass_c128(int T, int R, void* state, const PassDesc* dpass, const StepDesc* dsteps,
                             const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride,
                            const uint8_t* active, cudaStream_t st);
cudaError_t launch_pass_c64(int T, int R, void* state, const PassDesc* dpass, const StepDesc* dsteps,
                            const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride,
                            const uint8_t* active, cudaStream_t st);

cudaError_t launch_tile_pass(int precision, int T, int R, void* state, const PassDesc* dpass,
                             const StepDesc* dsteps, const KOp* dops, const void* dcoef, int n, int H,
                             int items, uint64_t cstride, const uint8_t* active, cudaStream_t st);
cudaError_t launch_small(int precision, void* state, uint64_t stride, int batch, int n, const KOp* dops, int nops,
                         const void* dcoef, uint64_t cstride, const uint8_t* active, cudaStream_t st);
// k: the op's dense target count (host copy of dop->k; selects the wide kernel)
cudaError_t launch_globalop(int precision, void* state, int n, int k, const KOp* dop, const void* dcoef, int items,
                            uint64_t cstride, const uint8_t* active, cudaStream_t st);
cudaError_t launch_set_basis(int precision, void* state, uint64_t N, uint64_t index, cudaStream_t st);
cudaError_t launch_convert(bool to64, const void* in, void* out, uint64_t n, cudaStream_t st);
cudaError_t launch_expect_z(int precision, const void* state, uint64_t N, const uint64_t* dzm, int nterms,
                            double* dpartial, int nblocks, cudaStream_t st);
cudaError_t launch_expect_x(int precision, const void* state, uint64_t N, uint64_t xmask, int flip_q,
                            const uint64_t* dzm, const int32_t* dny, int nterms, double* dpartial, int nblocks,
                            cudaStream_t st);
cudaError_t launch_reduce_partials(const double* dpartial, int nblocks, int stride, int nterms, double* dout,
                                   cudaStream_t st);
// Exact parallel sampling (sample.cu) in blocks of SAMPLE_BS amplitudes.
constexpr int SAMPLE_BS = 4096;
constexpr int SAMPLE_SLOTS = 64;  // blocks whose inner running sums are kept for the shots
struct SampleBlock {
    uint64_t cnt[2];  // grid counts at binades e and (two) e + 1
    int32_t e, two;
};
struct SampleScratch {
    float* bsum;       // nb approximate block sums
    double* pre;       // nb + 1: their exclusive prefix
    SampleBlock* blk;  // nb
    double* start;     // nb + 1: the exact running sum at every block start
    int32_t* slot;     // nb
    double* fine;      // SAMPLE_SLOTS * 1024 running sums
    int64_t* seq;      // blocks resolved element by element
};
// Lays the scratch out from `base` (256-byte aligned) and returns its size.
size_t sample_scratch(uint64_t N, void* base, SampleScratch* w);
size_t sample_scratch_bytes(uint64_t N);
cudaError_t launch_sample(int precision, const void* state, uint64_t N, const SampleScratch& w, const double* uni,
                          int64_t shots, uint64_t* out, cudaStream_t st);

}  // namespace qsv

namespace qsv {
// adjoint.cu
void adjoint_shape(int arith, int* T, int* R);
int adjoint_small_max(int arith);
bool pass2_shape_supported(int arith, int T, int R);
cudaError_t launch_pass2(int arith, int T, int R, void* psi, void* lam, const PassDesc* dpass, const StepDesc* dsteps,
                         const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride, int per_tile,
                         double* partial, int* grid_out, cudaStream_t st);
int pass2_grid_cap();
// adjoint_c128.cu, adjoint_ds.cu (+ adjoint_ds_r4.cu), adjoint_c64.cu: the tiled two-state
// pass per arithmetic
bool pass2_shape_c128(int T, int R);
bool pass2_shape_ds(int T, int R);
bool pass2_shape_ds_r4(int T, int R);  // adjoint_ds_r4.cu
bool pass2_shape_c64(int T, int R);
cudaError_t launch_pass2_c128(int T, int R, void* psi, void* lam, const PassDesc* dpass, const StepDesc* dsteps,
                              const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride,
                              int per_tile, double* partial, int* grid_out, cudaStream_t st);
cudaError_t launch_pass2_ds(int T, int R, void* psi, void* lam, const PassDesc* dpass, const StepDesc* dsteps,
                            const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride,
                            int per_tile, double* partial, int* grid_out, cudaStream_t st);
cudaError_t launch_pass2_ds_r4(int T, int R, void* psi, void* lam, const PassDesc* dpass, const StepDesc* dsteps,
                               const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride,
                               int per_tile, double* partial, int* grid_out, cudaStream_t st);
cudaError_t launch_pass2_c64(int T, int R, void* psi, void* lam, const PassDesc* dpass, const StepDesc* dsteps,
                             const KOp* dops, const void* dcoef, int n, int H, int items, uint64_t cstride,
                             int per_tile, double* partial, int* grid_out, cudaStream_t st);
cudaError_t launch_small2(int arith, void* psi, void* lam, int n, const KOp* dops, int nops, const void* dcoef,
                          int items, uint64_t cstride, double* probe_out, uint64_t pstride, cudaStream_t st);
cudaError_t launch_hamiltonian(int storage, const void* psi, void* lam, uint64_t N, const uint64_t* dx,
                               const uint64_t* dz, const int32_t* dny, const double* dc, int nterms, cudaStream_t st);
cudaError_t launch_probe_reduce(const double* partial, int grid, int np, double* out, cudaStream_t st);
}  // namespace qsv

namespace qsv {
// batch.cu
cudaError_t launch_bind(int arith, void* pool, uint64_t cstride, const Bind* dbinds, int nb, const double* dvals,
                        int nslots, int items, cudaStream_t st);
cudaError_t launch_replicate(int arith, void* pool, uint64_t cstride, uint64_t len, int items, cudaStream_t st);
cudaError_t launch_zero_items(int storage, void* state, int n, int items, cudaStream_t st);
uint64_t hamiltonian_chunk(int n);
// Expectation values per item; npart / inv (complex64; null: as they are):
// divided by the item's <psi|psi>, inv[item] = 1 / <psi|psi>.
cudaError_t launch_expect_seg(int storage, const void* psi, int n, int items, const uint64_t* dx, const uint64_t* dz,
                              const int32_t* dny, const double* dc, const int32_t* doptr, int nobs, double* epart,
                              double* out, double* npart, double* inv, cudaStream_t st);
cudaError_t launch_lambda_seg(int storage, const void* psi, void* lam, int n, int items, const uint64_t* dx,
                              const uint64_t* dz, const int32_t* dny, const double* dc, const int32_t* dtobs,
                              int nterms, int nobs, const double* dw, cudaStream_t st);
cudaError_t launch_probe_reduce_seg(const double* partial, uint64_t ntiles, int tpi, int items, int np, double* out,
                                    int ostride, int ooff, cudaStream_t st);
cudaError_t launch_slot_gather(const double* vals, int nprobe, int items, const int32_t* sptr, const int32_t* sidx,
                               int nslots, const double* inv, double* grads, cudaStream_t st);
}  // namespace qsv

namespace qsv {
// shots.cu: per-shot trajectories (mid-circuit measure / reset / cif)
struct MeasureSpec {
    uint8_t q[8];    // measured qubits, outcome bit order
    uint8_t srt[8];  // the same, ascending
    uint8_t cb[8];   // classical bits written (measure)
    int32_t k;       // qubits measured
    int32_t reset;   // 1: reset (final block 0), 0: measure
};
struct CifSpec {
    uint8_t cb[16];
    int32_t nc;
    uint64_t condition;
};
int outcome_blocks_per_item(int n, int k);
// Measures or resets every item; the states of items c_begin .. items-1 are
// collapsed (the outcomes alone matter for the others).  With `shared`, every
// item's state is that one state and `state` receives the collapsed copies.
cudaError_t launch_measure(const void* shared, void* state, int n, const MeasureSpec& ms, int items, int c_begin,
                           const double* duni, int draw, int ndraws, uint8_t* dcreg, int ncb, double* dpart,
                           int32_t* doutcome, double* dscale, cudaStream_t st);
cudaError_t launch_cif_mask(const uint8_t* dcreg, int ncb, int items, const CifSpec& cs, uint8_t* dactive,
                            cudaStream_t st);
cudaError_t launch_items_copy(void* state, int n, int items, const void* psi0, cudaStream_t st);
}  // namespace qsv

namespace qsv {
// noise.cu: per-shot noise channels on one qubit, per-item final sample
constexpr int MAX_CHANNEL_OPS = 8;
int channel_blocks_per_item(int n);  // CTAs per item of the Kraus-norm reduction
// cross: some Kraus operator's Gram matrix K^dagger K has a nonzero
// off-diagonal entry (the norms then need sum conj(a) c as well)
// One channel on every item.  A Kraus channel leaves the item's state
// unnormalised by 1 / dscale[item] where that factor is moderate.
cudaError_t launch_channel(void* state, int n, int q, int m, int kraus, int cross, const double* dmats,
                           const double* dprobs, int items, const double* duni, int draw, int ndraws, double* dpart,
                           double* dimat, double* dscale, cudaStream_t st);
cudaError_t launch_fill_ones(double* d, int count, cudaStream_t st);
// values[item * per + t] *= scale[item]^2
cudaError_t launch_scale_items(double* values, int items, int per, const double* dscale, cudaStream_t st);
cudaError_t launch_item_sample(const void* state, int n, int items, const double* dscale, const double* duni, int draw,
                               int ndraws, uint64_t* dout, cudaStream_t st);
}  // namespace qsv
