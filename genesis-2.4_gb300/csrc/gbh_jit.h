// gbh_jit.h -- per-program kernel specialisation (see gbh_jit.cu).
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "gbh_devfn.cuh"
#include "gbh_level.cuh"
#include "gbh_rows.cuh"

namespace gbh {

struct JitKernel {
    void *module = nullptr;   // CUmodule
    void *fn = nullptr;       // CUfunction
};

// CUDA source of the step kernel specialised to one tile type; empty if the
// program holds an op the generator does not emit. uniform_parent: the tree
// shared by every neuron of the type (elimination unrolled in registers), or
// null (per-neuron trees, shared-memory columns). compact: runs of identical
// compartment programs become loops and the rows stay in shared memory
// (smaller code; the autotuner decides which form runs). smem_rows: the
// unrolled form of a uniform tree keeps the eliminated rows (D, R) in
// shared-memory columns instead of registers, which frees ~4 registers a
// compartment for loads in flight.
std::string jit_source(const TileType &tt, const std::vector<int> &prog, const TableGeom &tg, bool mixed, bool giv,
                       const std::vector<int> *uniform_parent, int min_blocks = 4, bool compact = false,
                       bool smem_rows = false, int warps = 4);

// Which operands of a micro-op are field rows (bit i: operand i).
int field_operands(int code);

// The rows above a type's static ones as the level-elimination kernel runs
// them (gbh_level.cuh): their programs and the pool program with field rows
// relative to `f0`, so that types which differ only in their dendrites share
// one kernel (equal `key`). ok: the generator emits every op of them.
struct LevelProg {
    bool ok = false;
    int ntop = 0, f0 = 0;
    std::vector<int> prog;   // ntop slot programs, then the 0-terminated pool program
    int pool_off = 0;
    std::string key;
};
LevelProg level_prog(const TileType &tt, const std::vector<int> &prog);
// Source of the level-elimination kernel (entry gbh_jit) for one such program.
// resident: the block keeps its rows' constants in shared memory; io: with
// per-step inputs and outputs.
std::string jit_level_source(const LevelProg &lp, const TileType &tt, const TableGeom &tg, bool mixed, bool resident,
                             bool io);
cudaError_t jit_level_launch(const JitKernel &k, const DevView &v, const LevelView &lv, int g0, int ngroups, int warps,
                             int nsteps, long long step, size_t smem, cudaStream_t st);
// A type's compartments as the row-parallel kernel runs them (gbh_rows.cuh):
// their programs, grouped into classes of equal ones (field rows relative to
// the compartment's first). ok: the generator emits every op and no compartment
// reads what another leaves but the table bracket.
struct RowsProg {
    bool ok = false;
    std::vector<std::vector<int>> cls;   // one program per class
    std::vector<int> of, f0, prev;       // per slot: class, first field row, previous slot with a voltage lookup (-1 none, -2 has none)
    std::vector<int> pool;               // 0-terminated pool program
    std::string key;
};
RowsProg rows_prog(const TileType &tt, const std::vector<int> &prog);
std::string jit_rows_source(const RowsProg &rp, const TileType &tt, const TableGeom &tg, bool mixed);
cudaError_t jit_rows_launch(const JitKernel &k, const DevView &v, const RowView &rv, int g0, int ngroups, int warps,
                            int nsteps, long long step, size_t smem, cudaStream_t st);
// Largest dynamic shared memory the kernel may be launched with.
bool jit_allow_smem(const JitKernel &k, size_t smem);

bool jit_available(std::string *why);
int jit_compile(const std::string &src, bool fp64_exact, int device_major, int device_minor, JitKernel *out,
                std::string *log);
cudaError_t jit_launch(const JitKernel &k, const DevView &v, int tile0, int tile1, int smax, int warps, int nsteps,
                       long long step, size_t smem, bool coop, cudaStream_t st);
void jit_release(JitKernel &k);

}  // namespace gbh
