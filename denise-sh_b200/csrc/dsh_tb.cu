/* Launch shape and launch of the temporally blocked pass of small elastic
 * grids (dsh_tblock.cuh), FDORDER 2..8. */
#include <algorithm>
#include <cstdlib>

#include "dsh_tb.h"

namespace dsh {
static TbFn tb_fn(const TbProblem &pb, int nthr)
{
    switch (pb.fdorder) {
    case 2: return tb_kernel_fd2(pb.mode, pb.p2, nthr);
    case 4: return tb_kernel_fd4(pb.mode, pb.p2, nthr);
    case 6: return tb_kernel_fd6(pb.mode, pb.p2, nthr);
    case 8: return tb_kernel_fd8(pb.mode, pb.p2, nthr);
    default: return nullptr;
    }
}

static int env_int(const char *name, int lo, int hi)
{
    const char *e = getenv(name);
    const int v = e ? atoi(e) : 0;
    return v >= lo && v <= hi ? v : 0;
}

bool tb_config(const TbProblem &pb, TbCfg *cfg)
{
    if (pb.fdorder < 2 || pb.fdorder > 8 || (pb.fdorder & 1) || pb.nb < 1 || pb.nx < 1 || pb.ny < 1 || pb.nx > 0xffff || pb.ny > 0x7fff) return false;
    if (pb.max_entries > TB_MAX_ENT || pb.max_members > TB_MAX_MEM || pb.max_receivers > TB_MAX_REC) return false;
    if (pb.fw > 0 && (pb.nx < 2 * pb.fw || pb.ny < 2 * pb.fw)) return false;
    int dev = 0, maxsm = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if ((long long)pb.nx * pb.ny * pb.nb > 4LL * TB_MAX_THREADS * nsm) return false;     /* more vectors than threads */
    const int H = pb.fdorder / 2, R = pb.fdorder - 1;
    const int kmax = pb.fdorder == 2 ? 8 : pb.fdorder == 4 ? 4 : pb.fdorder == 6 ? 3 : 2;
    const int kpin = env_int("DSH_TB_STEPS", 1, 64), rows = env_int("DSH_TB_ROWS", 1, 256);
    double best = 0.0;
    TbCfg c;
    auto consider = [&](int tw, int th, int k) {
        TbGeom g;
        g.tw = tw; g.th = th; g.k = k;
        g.gy = k * R; g.gx = (g.gy + 3) / 4 * 4;
        g.nv = (tw + 2 * g.gx) / 4; g.eh = th + 2 * g.gy;
        g.ntx = (pb.nx + tw - 1) / tw; g.nty = (pb.ny + th - 1) / th;
        g.nthr = (g.nv * g.eh + 31) / 32 * 32;
        g.nent = std::max(4, (pb.max_entries + 3) / 4 * 4);
        g.nrec = std::max(4, (pb.max_receivers + 3) / 4 * 4);
        const long long tiles = (long long)g.ntx * g.nty * pb.nb;
        const long long bytes = 4LL * tb_smem(g, H, pb.mode).total;
        if (g.nthr > TB_MAX_THREADS || tiles > nsm || bytes > maxsm) return false;
        /* us: per step one vector of a thread, slower with the fewer registers of
           larger blocks (the storing and adjoint modes spill more there), per
           round the exchange, longer among more tiles; fitted to 60 shapes of
           FDORDER 4, 6 and 8, 50 to 144 tiles, 384 to 1024 threads, 0.13 rms.
           Against one rate per thread and 2.8 per round: 600 x 250, FDORDER 4: 3.46 ->
           3.21; 14 shots of 160 x 80: 3.65 -> 3.32; FDORDER 6, 8 shots: 4.22 -> 3.93, 500
           x 200: 3.80 -> 3.39 */
        const double large = pb.mode == TB_FWD ? 0.0023 : 0.0028;
        const double per = g.nthr <= TB_FEW_THREADS ? 0.0012 : g.nthr <= TB_MID_THREADS ? 0.0019 : large;
        const double t = 0.1 + per * g.nthr + (3.85 + 0.0069 * (double)tiles) / k;
        if (best == 0.0 || t < best) {
            best = t;
            c.geo = g;
            c.tiles = (int)tiles;
            c.smem = (size_t)bytes;
        }
        return true;
    };
    for (int tw = 32; tw <= 64; tw += 32)
        for (int th = rows ? rows : 8; th <= (rows ? rows : 128); th += 8) {
            if (kpin) {
                for (int k = kpin; k >= 1 && !consider(tw, th, k); k--) {}
            } else {
                for (int k = kmax; k >= pb.min_k; k--) consider(tw, th, k);
            }
        }
    if (best == 0.0) return false;
    const TbFn fk = tb_fn(pb, c.geo.nthr);
    /* the opt-in maximum, not this problem's size: contexts of other sizes
       may launch the same kernel concurrently */
    if (cudaFuncSetAttribute((const void *)fk, cudaFuncAttributeMaxDynamicSharedMemorySize, maxsm) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    *cfg = c;
    return true;
}

cudaError_t tb_launch(const TbCfg &cfg, const TbProblem &pb, const StepArgs &a, const TbExchange &x, int n0, int count,
                      cudaStream_t st)
{
    const TbFn fk = tb_fn(pb, cfg.geo.nthr);
    if (!fk || cfg.tiles < 1) return cudaErrorInvalidValue;
    StepArgs sa = a;
    TbGeom g = cfg.geo;
    TbExchange xx = x;
    void *args[5] = {&sa, &g, &xx, &n0, &count};
    return cudaLaunchCooperativeKernel((const void *)fk, dim3((unsigned)cfg.tiles), dim3((unsigned)g.nthr), args, cfg.smem, st);
}
}  // namespace dsh
