// ltl_kernels.h -- host-side launchers of the libltl_b200 kernels (internal).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "ltl_internal.cuh"

namespace ltl {

struct GridBarrier;  // grid_barrier.cuh

// Limit of a barrier wait.  missing = 1: the barrier expects one CTA more than there are,
// so that every wait runs out (how the failure path is tested).
struct BarrierLimit {
    unsigned long long ns = 2000000000ull;  // far above any generation's time
    unsigned int missing = 0;
};

// K5: refresh the torus halo of a frame (every halo cell <- its inner source).
cudaError_t launch_halo_fill(const Frame& f, cudaStream_t s);

// K1 fast path: SWAR 8-bit lanes, warp-shuffle row sums; R <= 5.
bool plain_swar8_supported(int radius);
// One-time function attributes (dynamic shared memory) so that launches can be
// captured in CUDA graphs without configuration calls.
cudaError_t plain_prepare(int radius);
// wrap: read every cell from its inner position (torus wrap inside the kernel),
// so the frame halo is neither read nor needed; requires plain_wrap_supported(n).
bool plain_wrap_supported(int n, int rows);
cudaError_t launch_plain_swar8(const Frame& cur, const Frame& nxt, const Rule& rule, int band_rows, bool wrap,
                               cudaStream_t s);
// Built-in shape: generations per pass, and rows per work item at that depth.
int plain_swar8_depth(int radius);
int plain_swar8_band_rows(int rows, int n, int radius, int depth, int device);
// Temporally blocked SWAR step: `depth` (2 or 3, depth * R <= 16) generations per
// pass; the frames' halo must be at least depth * R.
bool plain_tb_supported(int radius, int depth);
cudaError_t plain_tb_prepare(int radius);
cudaError_t launch_plain_tb(const Frame& cur, const Frame& nxt, const Rule& rule, int band_rows, int depth,
                            bool wrap, cudaStream_t s);

// K1 generic path (R up to 2038): one fused kernel (vertical window sums in
// registers, a prefix scan per row, or per pair of rows, in shared memory, the
// rule); needs a halo of at least R rounded up to plain_wide_cols_per_thread(R).
// band_rows: rows per CTA (plain_generic_band_rows: built-in choice).
bool plain_generic_supported(int radius);
int plain_generic_band_rows(int rows, int n, int radius, int device);
int plain_wide_cols_per_thread(int radius);
cudaError_t launch_plain_generic(const Frame& cur, const Frame& nxt, const Rule& rule, int band_rows,
                                 cudaStream_t s);

// K3: bit-packed variant.  Packed frame: 32-bit words, cell (i, j) is bit j % 32
// of word j / 32 (LSB first; two consecutive words are one little-endian uint64
// of the PACK codec).  Inner row i is frame row HR + i, inner word w is frame
// column HW + w.  No step reads a halo: rows and words wrap in the loads.  Bits
// past n in a row's last word are copies of the row's first cells where n >= 64
// (joined rows, see packed_core.cuh; uploads make them, the packed step keeps
// them), else anything; other readers mask them.
struct PackedFrame {
    uint32_t* words;
    int n;          // cells per side
    int nw;         // inner words per row = ceil(n / 32)
    int HR;         // rows before inner row 0
    int HW;         // words before inner word 0 (packed step: 0, 16-byte aligned rows)
    size_t wpitch;  // words per frame row
    int rows = 0;   // inner rows of a rectangular torus (0: square, n rows)
    __host__ __device__ int nrows() const { return rows ? rows : n; }
};
bool packed_supported(int n, int radius);
// as plain_prepare, for a grid's frames: before the first launch_packed_step (walk) or
// launch_packed_run
cudaError_t packed_prepare(const PackedFrame& f, int radius, bool walk);
// band_rows <= 0: built-in heuristic; > 0: rows per work item (tuning table / ltl_set_param)
cudaError_t launch_packed_step(const PackedFrame& cur, const PackedFrame& nxt, const Rule& rule, int band_rows,
                               cudaStream_t s);
// Grids that are advanced many generations per launch (packed_runs: small ones, by
// sides and radius alone): `steps` generations from cur, to nxt if `steps` is odd,
// else back in cur; both frames are written.
struct PackedRun {
    GridBarrier* barrier = nullptr;  // device, zero at first; one per grid, which always has the same CTAs
    unsigned int* err = nullptr;     // device, zero at first; set if a barrier wait ran out: the grid
                                     // is then unspecified and the barrier has to be zeroed
    BarrierLimit limit{};
};
bool packed_runs(const PackedFrame& f, int radius);
cudaError_t launch_packed_run(const PackedFrame& cur, const PackedFrame& nxt, const Rule& rule, int steps,
                              const PackedRun& run, cudaStream_t s);

// Transfers between codings and reductions (k_transfer.cu).  Callers' byte
// buffers are dense cells, `pitch` bytes per row, any alignment.
// Byte frame <- / -> caller's buffer; in, every byte that is not 0 becomes 1.
cudaError_t launch_copy_in(const Frame& f, const uint8_t* src, size_t src_pitch, cudaStream_t s);
cudaError_t launch_copy_out(const Frame& f, uint8_t* dst, size_t dst_pitch, cudaStream_t s);
// Inner rows [row0, row0 + nrows) of a packed frame from / to a buffer whose row
// i is frame row row0 + i.  nonzero: a cell is alive if its byte is not 0, else
// by its bit 0.  barrier (where a whole grid comes in, else null): zeroed, since a run
// whose wait ran out leaves it at some count in between.
cudaError_t launch_pack_rows(const uint8_t* src, size_t pitch, bool nonzero, const PackedFrame& dst, int row0,
                             int nrows, GridBarrier* barrier, cudaStream_t s);
// err (or null): if that word is set, dst's first cell becomes kMarkCell.
constexpr uint8_t kMarkCell = 0xff;
constexpr uint32_t kMarkCells = 0x5ac3a53cu;
cudaError_t launch_unpack_rows(const PackedFrame& src, int row0, int nrows, uint8_t* dst, size_t pitch,
                               const unsigned int* err, cudaStream_t s);
// A packed frame's inner words as PACK-coded rows (bits past n cleared); err as above, the
// first 32 cells become kMarkCells.
cudaError_t launch_frame_to_pack64(const PackedFrame& f, uint64_t* dst, size_t dst_pitch_words, const unsigned int* err,
                                   cudaStream_t s);
// PACK-coded rows into a packed frame (barrier as in launch_pack_rows).
cudaError_t launch_pack64_to_frame(const uint64_t* src, size_t src_pitch_words, const PackedFrame& f,
                                   GridBarrier* barrier, cudaStream_t s);
// PACK codec on callers' buffers (not 0 -> 1).
cudaError_t launch_pack(const uint8_t* cells, size_t cell_pitch, int rows, int cols, uint64_t* words,
                        size_t word_pitch_words, cudaStream_t s);
cudaError_t launch_unpack(const uint64_t* words, size_t word_pitch_words, int rows, int cols, uint8_t* cells,
                          size_t cell_pitch, cudaStream_t s);
// K6: population and comparison over the inner cells.  `scratch` holds two
// uint64 (count, first index) in device memory.
cudaError_t launch_population(const Frame& f, unsigned long long* scratch, cudaStream_t s);
cudaError_t launch_population(const PackedFrame& f, unsigned long long* scratch, cudaStream_t s);
cudaError_t launch_compare(const Frame& f, const uint8_t* other, size_t other_pitch, unsigned long long* scratch,
                           cudaStream_t s);
cudaError_t launch_compare(const PackedFrame& f, const uint8_t* other, size_t other_pitch, unsigned long long* scratch,
                           cudaStream_t s);

// K2: tcgen05 banded-product step on packed frames (the tensor variant keeps
// its grid in the packed layout of K3; the kernel wraps rows and words modulo n
// itself, so the packed halo is never read).  The frames need HW >= 1.
struct TensorPlan;
bool tensor_supported(int n, int radius, char* why, size_t why_len);
// barrier, err: device words, zero before the plan's first launch; err is set when a
// wait runs out, and both have to be zeroed then.
TensorPlan* tensor_plan_create(const PackedFrame& a, const PackedFrame& b, const Rule& rule, int device,
                               GridBarrier* barrier, unsigned int* err, char* why, size_t why_len);
void tensor_plan_destroy(TensorPlan* p);
int tensor_plan_depth(const TensorPlan* p);
int tensor_plan_operand_bits(const TensorPlan* p);
// Advance `steps` generations in one launch, from packed frame `src_is_a ? a : b`
// (steps > 1 only where tensor_plan_runs).
bool tensor_plan_runs(const TensorPlan* p);
cudaError_t launch_tensor_steps(TensorPlan* p, bool src_is_a, int steps, cudaStream_t s);
// Limit of the kernel's bounded waits, and a test hook that withholds one
// completion signal so that the waits run out (no fault, no hang: the kernel
// returns after the limit with an error bit set).
void tensor_plan_set_wait(TensorPlan* p, unsigned long long ns, int inject_missing_commit);

// Tuning table (written by cat_cpu_b200/autotune.py): the value of `param` for
// (variant name, radius, n), or `fallback` when no line matches.  Lines look like
//   variant=plain radius=5 nmin=8192 nmax=65536 band_rows=128
// radius=* matches every radius.  The file is $LTL_TUNING_FILE, else
// tuning/ltl_tuning.txt next to libltl_b200.so.
long long tuning_lookup(const char* variant, int radius, long long n, const char* param, long long fallback);

}  // namespace ltl
