/* dsh_tb.h — the temporally blocked pass of small elastic grids
 * (dsh_tblock.cuh): its launch shape for a context and its launch. */
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "dsh_tblock.cuh"

namespace dsh {
/* the kernel of one build: each order is a module of its own (dsh_tb2.cu to
 * dsh_tb8.cu), loaded when it is first needed: 2.7 ms, all orders in one 17.5 */
using TbFn = void (*)(StepArgs, TbGeom, TbExchange, int, int);
TbFn tb_kernel_fd2(int mode, bool p2, int nthr);
TbFn tb_kernel_fd4(int mode, bool p2, int nthr);
TbFn tb_kernel_fd6(int mode, bool p2, int nthr);
TbFn tb_kernel_fd8(int mode, bool p2, int nthr);

/* what decides whether and how the kernel serves a pass of an elastic context */
struct TbProblem {
    int fdorder, p2, mode, nx, ny, fw;
    int nb;                      /* shot slots */
    int min_k = 1;               /* fewest steps per round */
    int max_entries, max_members, max_receivers;   /* per slot: sources, sources at one point, receivers */
};

struct TbCfg {
    TbGeom geo;
    int tiles = 0;               /* blocks of the launch: tiles of all slots */
    size_t smem = 0;             /* dynamic shared memory per block in bytes */
};

/* The launch shape on the current device: among tiles 32 or 64 points wide and
 * a multiple of 8 rows high that give at most one block per SM, and k = 1 to
 * 4 (FDORDER 2: 8, 4: 4, 6: 3, 8: 2) steps per round, the one with the least
 * estimated time per step (tb_config in dsh_tb.cu); DSH_TB_STEPS pins k (lowered
 * where the region does not fit a block) and DSH_TB_ROWS the height.  false
 * when the kernel cannot serve the problem: FDORDER > 8, more sources or
 * receivers per slot than its lists hold, NX or NY below 2 FW, or no shape
 * with every block resident. */
bool tb_config(const TbProblem &pb, TbCfg *cfg);

/* Launches steps n0 .. n0 + count - 1 for the configured slots (cooperative). */
cudaError_t tb_launch(const TbCfg &cfg, const TbProblem &pb, const StepArgs &a, const TbExchange &x, int n0, int count,
                      cudaStream_t st);
}  // namespace dsh
