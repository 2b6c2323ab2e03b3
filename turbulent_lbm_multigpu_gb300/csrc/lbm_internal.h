// lbm_internal.h -- host runtime shared by the translation units of
// liblbm_gb300.so (not part of the public C ABI).
#pragma once
#include <cstdio>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "lbm_gb300.h"
#include "lbm_kernels.cuh"

namespace lbm_rt {
using namespace lbm;

// Records the message returned by lbm_cu_last_error() on this thread; -1.
int fail(const std::string &m);

#define CU(call)                                                                                \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess) return ::lbm_rt::fail(std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

inline cudaStream_t S(void *s) { return (cudaStream_t)s; }

// Launch of a kernel that begins with follow_previous_grid(): its blocks are
// set up before the grid before it on the stream has written back its results.
// Measured on runs launched step by step (us per step, plain -> this): float
// 24^3 5.12 -> 2.83, 64^3 9.22 -> 6.64, 128^3 55.6 -> 52.6; half 24^3 5.12 ->
// 2.64, 128^3 33.0 -> 30.3; double 64^3 56.9 -> 54.5: about 2.5 us a launch.
// Also faster in a graph that a caller captures (float 64^3 6.84 -> 6.41) and
// between lbm_cu_halo copies (four 64^3 lattices, step and exchange: 71.0 ->
// 60.1 us).  Not used for the steps of several subdomains (domain_one_step).
struct Dep {
    bool on = true;  // false: an ordinary launch
};
template <typename... P, typename... A>
inline int launch_dep(Dep dep, void (*kernel)(P...), dim3 grid, int threads, size_t shared, cudaStream_t st,
                      const A &...args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = dep.on ? 1 : 0;
    CU(cudaLaunchKernelEx(&cfg, kernel, args...));
    return 0;
}

constexpr int kBlock = 256;

inline size_t storage_bytes(int st) { return st == kF64 ? 8 : st == kF32 ? 4 : 2; }
inline size_t real_bytes(int st) { return st == kF64 ? 8 : 4; }
inline int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }
inline int grid_for(int64_t work) { return (int)((work + kBlock - 1) / kBlock); }

// Kernel arguments of a lattice, rounded to its arithmetic type.
void set_params_desc(LatDesc &h, int storage, const lbm_params &p);
inline bool uses_les(const LatDesc &h) { return h.pd[P_LES] != 0.0; }

// The two-cell kernels apply when every lattice has an even x extent and a
// float arithmetic type.
bool pair_shape(int storage, const LatDesc *tab, int ntab);
inline int cells_per_block(bool pair) { return pair ? kPairCells : kBlock; }

// Kernel shapes of a step: 1 one cell per thread, 2 two cells per thread,
// 3 tiles staged through shared memory by bulk copies, 0 automatic: for the
// 16-bit storage types 3 where both kinds of step are the faster staged
// (staged_pays), the staged alpha and the one-cell beta step where only the
// alpha step is (kShapeStagedAlpha), 1 otherwise.  The shape a set of lattices runs: 2 needs
// float arithmetic and even nx, 3 float or 16-bit storage; otherwise 1.
//
// Small launches do not fill the staged kernel's persistent blocks with
// tiles, and a tile's way through the ring is longer than a load and a store.
// Measured (half, us per step launched one by one, one-cell / staged): 24^3
// 3.15 / 5.23, 64^3 6.16 / 8.55, 96^3 15.2 / 16.1, 112^3 (1.40 M cells) 22.7 /
// 22.3, 128^3 33.3 / 30.9, 144^3 55.7 / 43.9, 176^3 101 / 75.6; rows that are
// not whole 16-byte units: 121x99x87 (1.04 M) 17.4 / 18.3, 129x128x128 33.7 /
// 32.2 (its beta kernels 41.3 / 41.8), 177x176x176 102.5 / 77.9; c16 64^3 6.76 / 8.69, 112^3 26.9 / 26.9,
// 176^3 111 / 92.9.  The alpha kernels alone cross earlier (half, us): 64^3
// 10.5 / 10.7, 96^3 18.6 / 17.5, 121x99x87 20.7 / 18.8.  The lines are cell
// counts where this GPU's two kernels cross, not multiples of its resident
// blocks.
constexpr int64_t kStagedAlphaCells = 786432;    // alpha steps
constexpr int64_t kStagedCells = 1310720;        // beta steps, every row whole 16-byte units
constexpr int64_t kStagedRaggedCells = 2359296;  // beta steps, other rows
inline bool staged_pays(bool beta, bool ragged, int64_t cells) {
    return cells >= (!beta ? kStagedAlphaCells : ragged ? kStagedRaggedCells : kStagedCells);
}
int effective_shape(int storage, int shape, const LatDesc *tab, int ntab);

// Internal kernel shape of double lattices that run the contracted FP64
// kernels (lbm_cu_set_fp64_contraction): one cell per thread, fused
// multiply-adds (lbm_f64fma.cu).
constexpr int kShapeF64Fma = 4;
// Internal kernel shape between 1 and 3: staged alpha, one-cell beta steps.
constexpr int kShapeStagedAlpha = 5;
// One step of up to kParamLattices double lattices with the contracted
// kernels (lbm_f64fma.cu); blocks of kBlock cells.
int launch_step_f64_fma(int parity, bool les, const DomainArgs &a, int blocks, Dep dep, cudaStream_t st);

// Streaming multiprocessors of the current device (cached per device).
int sm_count();
// A lattice's population, flag and velocity planes in one device block of
// lattice_block_bytes (a pool's; the lattice does not free it).
size_t lattice_block_bytes(int nx, int ny, int nz, int storage, int store_v);
int lattice_in_block(int nx, int ny, int nz, int storage, int store_v, void *block, lbm_lattice **out);
// Grow a lattice's staging buffer to at least `bytes`.
int ensure_stage(lbm_lattice *l, size_t bytes);

// One step over `ntab` lattices of one storage type, kParamLattices
// descriptors per launch.
int launch_step(int storage, int shape, int parity, bool les, const LatDesc *htab, int ntab, int sv, int sr,
                Dep dep, cudaStream_t st);
// One step of a lattice in its own kernel shape; store: write u and rho, if
// the lattice keeps them.
int step_lattice(const lbm_lattice *l, int parity, bool store, cudaStream_t st);
// Cells per staged tile of a storage type (0: not staged).
int staged_cells(int storage);
// One step of up to kBatchLattices 16-bit lattices of any row length, all at
// an alpha step or all at a beta step, through the staged tiles (first_block /
// nblocks of the descriptors count tiles of staged_cells).
int launch_staged_batch(int storage, bool beta, bool les, const BatchArgs &a, int tiles, Dep dep, cudaStream_t st);
// One lattice block of a checkpoint file (lbm_io.cu).
int ckpt_write_lattice(FILE *f, lbm_lattice *l, int64_t counter);
int ckpt_read_lattice(FILE *f, lbm_lattice *l, int64_t *counter);
}  // namespace lbm_rt

struct lbm_lattice {
    int nx, ny, nz;
    int64_t n, pstride;
    int storage;
    int store_v, store_rho;
    void *dd = nullptr;
    uint8_t *flags = nullptr;
    void *vel = nullptr;
    void *rho = nullptr;
    lbm::LatDesc h{};
    bool pooled = false;  // the fields lie in a block that the lattice's owner keeps
    void *stage = nullptr;  // staging for host copies and reduction partials
    size_t stage_bytes = 0;
    int shape = 0;  // requested kernel shape (0: per storage type, see effective_shape)
    int fma64 = 0;  // double storage: contracted FP64 kernels (lbm_cu_set_fp64_contraction)
};
