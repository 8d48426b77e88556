/*
 * dsh_tblock.cuh — small elastic grids: a whole pass in one launch, several
 * time steps between two exchanges of neighbouring tiles (temporal blocking
 * with overlapped tiles, FDORDER 2-8).
 *
 * On a grid of less than one wave of blocks the kernel pair's two launches
 * per step are all latency (4.0 us per step at 160 x 80, 4.4 at 500 x 200,
 * of which launches and dependent loads from L2 are 3.0).  Here the grid is
 * cut into one tile per SM and a thread block keeps its tile in shared memory
 * and registers for the whole pass.
 *
 * A block owns tw x th points and holds them grown by gx x gy points (gy =
 * k (FDORDER - 1), gx the same rounded up to 4).  Thread t owns one vector of
 * four x-consecutive points of that region for the whole pass: its vy, sxy,
 * syz, 1/rho, uip, ujp stay in registers; shared memory holds copies of vy,
 * sxy, syz for the neighbouring threads (H rows and one vector of zeros around
 * them) and the thread's four CPML memory vectors.  One step of the velocity
 * update reads stresses up to H = FDORDER/2 points away (H left, H-1 right),
 * one of the stress update velocities H-1 left and H right, so each step
 * spoils 2H - 1 = FDORDER - 1 points at the region's edge; after k steps the
 * own points are still exact (every block recomputes its halo).  Then each
 * block writes its own points to an exchange buffer, publishes its count of
 * completed rounds with a release store, polls those of the tiles its halo
 * reaches into (bounded: on expiry the block sets status bit 2 and leaves) and
 * reads its halo from their buffers.  Two buffers alternate: a tile that
 * writes round n+1 has seen round n of its neighbours, who have read round
 * n-1 by then.  All blocks are resident (cooperative launch).
 *
 * What bounds it: the two barriers of a step (217 to 238 instructions per warp
 * and step; of 15 to 19 cycles between two instructions of a warp 9 to 11 are
 * spent at a barrier) and per round one exchange of 4 to 5 us through L2.  The
 * launch shape (tw, th, k) minimises that cost (tb_config).  us per step,
 * pair and this pass: 160 x 80, FDORDER 4: 4.0 and 1.9; 500 x 200: 4.4 and 2.5.
 *
 * Modes: plain forward (TB_FWD; with the energy sum where the pass keeps
 * checkpoints), forward with storage of the acceleration and the strain rates
 * (TB_STORE), adjoint with the correlations (TB_ADJ; the stored fields and the
 * signals come through a ring of cp.async copies three steps ahead).
 *
 * Per point the arithmetic is that of v_body / s_body (dsh_kernels.cuh) for
 * L = 0, the same expressions in the same order, compiled with -fmad=false,
 * so results are bit-identical to the kernel pair (update_v_PML.c:51-198,
 * update_s_elastic_PML.c:51-455, seismo_ssg.c:17-27, denise.c:1589-1609,
 * eprecond.c:11).  A point lies in at most one CPML strip per axis (the host
 * requires NX, NY >= 2 FW).
 */
#pragma once

#include "dsh_kernels.cuh"

namespace dsh {

/* block sizes of the builds: 64, 80 (704 threads are 22 warps, six on one scheduler) and up to 128 registers per
 * thread; the first two spill (FDORDER 4: 100-140 and 44-60 bytes stored) */
constexpr int TB_MAX_THREADS = 1024, TB_MID_THREADS = 704, TB_FEW_THREADS = 512;
constexpr int TB_MAX_ENT = 1024; /* sources of a slot (receivers in the adjoint) */
constexpr int TB_MAX_MEM = 8;    /* sources at one point */
constexpr int TB_MAX_REC = 2048; /* receivers of a slot */
constexpr int TB_RING = 4;       /* steps of signals and stored fields in flight or in use */
constexpr int TB_XFIELDS = 7;    /* exchanged: vy sxy syz psi_vxx psi_vyy psi_sxx psi_syy */
enum TbMode { TB_FWD = 0, TB_STORE = 1, TB_ADJ = 2 };

struct TbGeom {
    int tw, th;                  /* own tile: tw x th grid points, tw a multiple of 4 */
    int k;                       /* steps per round */
    int gx, gy;                  /* halo per side */
    int nv, eh;                  /* region: nv vectors x eh rows */
    int ntx, nty;                /* tiles of a slot */
    int nthr;                    /* threads per block: nv*eh rounded up to warps */
    int nent, nrec;              /* list capacities */
};

/* dynamic shared memory of a block, offsets in 4-byte words */
struct TbSmem {
    int vy, sxy, syz, psi, coef, acc, ring, sig, ent, point, rec, cnt, total;
};
__host__ __device__ inline TbSmem tb_smem(const TbGeom &g, int H, int mode)
{
    TbSmem s;
    const int field = (g.eh + 2 * H) * (4 * g.nv + 8), nown = g.tw * g.th;
    int o = 0;
    s.vy = o; o += field;
    s.sxy = o; o += field;
    s.syz = o; o += field;
    s.psi = o; o += 4 * 4 * g.nthr;                      /* [field][thread] float4 */
    s.coef = o; o += 4 * 4 * g.nv;                       /* x strips: a, b, a_half, b_half per column */
    s.acc = o; o += (mode == TB_ADJ ? 3 : 1) * nown;     /* W, and in the adjoint g_u, g_rho */
    s.ring = o; o += mode == TB_ADJ ? TB_RING * 3 * nown : 0;
    s.sig = o; o += TB_RING * g.nent;
    s.ent = o; o += g.nent;
    s.point = o; o += 2 * g.nthr;                        /* per point: 0 or first entry + 1 | members << 12 */
    s.rec = o; o += 2 * g.nrec;
    s.cnt = o; o += 2;
    s.total = o;
    return s;
}

struct TbExchange {
    float *buf;                  /* [2][slot][TB_XFIELDS][dstride] */
    unsigned *done;              /* [slot][tile]: rounds completed, 0 at launch */
};

__device__ __forceinline__ float4 lds4v(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void sts4v(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ void tb_copy16(float *dst, const float *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void tb_copy4(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void tb_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tb_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

/* waits until *f >= need, at most `limit` polls; on expiry sets status bit 2 and returns 0 */
__device__ __forceinline__ int tb_poll(const unsigned *f, unsigned need, long long limit, int *status)
{
    for (long long it = 0; it < limit; it++) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
        if (v >= need) return 1;
    }
    atomicOr(status, 2);
    return 0;
}

/* CPML recursion of a thread's four x-strip points (bits of in) with the
 * memory psi and the coefficient columns in shared memory; K from global
 * memory where it is not 1 */
__device__ __forceinline__ void tb_cpml_x(float *d, float *psi, const float *ca, const float *cb, int in, const float *K, int h,
                                          int hr, bool k_one)
{
    const float4 p = lds4v(psi), a = lds4v(ca), b = lds4v(cb);
    float4 n = p;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (in >> k & 1) {
            const float t = get(b, k) * get(p, k) + get(a, k) * d[k];
            set(n, k, t);
            if (!k_one) {
                stay_in_branch();
                d[k] = d[k] / __ldg(K + (in >> (4 + k) & 1 ? hr : h) + k);
            }
            d[k] = d[k] + t;
        }
    sts4v(psi, n);
}
__device__ __forceinline__ void tb_cpml_y(float *d, float *psi, float a, float b, const float *K, bool k_one)
{
    const float4 p = lds4v(psi);
    const float4 n = make_float4(b * p.x + a * d[0], b * p.y + a * d[1], b * p.z + a * d[2], b * p.w + a * d[3]);
    sts4v(psi, n);
    if (!k_one) {
        stay_in_branch();
        const float kk = __ldg(K);
#pragma unroll
        for (int k = 0; k < 4; k++) d[k] = d[k] / kk;
    }
    d[0] = d[0] + n.x; d[1] = d[1] + n.y; d[2] = d[2] + n.z; d[3] = d[3] + n.w;
}

template <int FDO, bool P2, int MODE, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) tb_pass(StepArgs a, TbGeom g, TbExchange x, int n_first, int count)
{
    constexpr int H = FDO / 2, R = FDO - 1;
    extern __shared__ __align__(16) float tb_dyn[];
    const TbSmem sm = tb_smem(g, H, MODE);
    const int nx = a.nx, ny = a.ny, fw = a.fw, pitch = a.pitch;
    const int tiles = g.ntx * g.nty, slot = blockIdx.x / tiles, tile = blockIdx.x - slot * tiles;
    const int bx = tile % g.ntx, by = tile / g.ntx;
    const int ox = 1 + bx * g.tw, oy = 1 + by * g.th;
    const int t = threadIdx.x, row = t / g.nv, vec = t - row * g.nv;
    const int i0 = ox - g.gx + 4 * vec, j = oy - g.gy + row;
    const bool in = row < g.eh && i0 >= 1 && i0 <= nx && j >= 1 && j <= ny;
    const bool own = in && i0 >= ox && i0 < ox + g.tw && j >= oy && j < oy + g.th;
    const int nvalid = min(4, nx - i0 + 1);
    const int wp = 4 * g.nv + 8, at = (row + H) * wp + 4 + 4 * vec;     /* this vector in the shared fields */
    float *const vy_s = tb_dyn + sm.vy + at, *const sxy_s = tb_dyn + sm.sxy + at, *const syz_s = tb_dyn + sm.syz + at;
    float *const psi_s = tb_dyn + sm.psi + 4 * t;                       /* field f at + 4*nthr*f */
    float *const acc_s = tb_dyn + sm.acc + (own ? (j - oy) * g.tw + (i0 - ox) : 0);
    const int nown = g.tw * g.th;
    const long long so = (long long)slot * a.slot_stride;
    const long long drow = (long long)(j - 1) * pitch + (i0 - 1 + HX), hrow = drow + (long long)a.hy * pitch;
    const bool k_one = a.pml_k1 != 0;

    /* ---- strips: bits 0-3 points in an x strip, bits 4-7 those of the right one; hy the depth-strip index ---- */
    int xin = 0, hy = 0;
    const int hr = i0 - nx + 2 * fw;
    if (in && fw > 0) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i0 + k <= fw) xin |= 1 << k;
            else if (i0 + k >= nx - fw + 1 && i0 + k <= nx) xin |= 17 << k;
        }
        hy = (!a.free_surf && j <= fw) ? j : (j >= ny - fw + 1 ? j - ny + 2 * fw : 0);
    }
    float ya = 0.f, yb = 0.f, yah = 0.f, ybh = 0.f;
    if (hy) {
        ya = __ldg(a.pml.a_y + hy); yb = __ldg(a.pml.b_y + hy);
        yah = __ldg(a.pml.a_y_half + hy); ybh = __ldg(a.pml.b_y_half + hy);
    }

    /* ---- shared memory: zeros, coefficient columns ---- */
    for (int k = t; k < sm.psi; k += blockDim.x) tb_dyn[k] = 0.f;
    for (int k = t; k < 2 * g.nthr; k += blockDim.x) tb_dyn[sm.point + k] = 0.f;
    if (t < 2) reinterpret_cast<int *>(tb_dyn + sm.cnt)[t] = 0;
    if (fw > 0)
        for (int c = t; c < 4 * g.nv; c += blockDim.x) {
            const int i = ox - g.gx + c, h = i < 1 || i > nx ? 0 : i <= fw ? i : i >= nx - fw + 1 ? i - nx + 2 * fw : 0;
            float *q = tb_dyn + sm.coef + c;
            q[0] = h ? __ldg(a.pml.a_x + h) : 0.f;
            q[4 * g.nv] = h ? __ldg(a.pml.b_x + h) : 0.f;
            q[8 * g.nv] = h ? __ldg(a.pml.a_x_half + h) : 0.f;
            q[12 * g.nv] = h ? __ldg(a.pml.b_x_half + h) : 0.f;
        }
    __syncthreads();

    /* ---- model, state, CPML memory, sums ---- */
    float4 vy4 = make_float4(0.f, 0.f, 0.f, 0.f), sxy4 = vy4, syz4 = vy4, b4 = vy4, ui4 = vy4, uj4 = vy4;
    if (in) {
        b4 = ldg4(a.brho + drow); ui4 = ldg4(a.uip + drow); uj4 = ldg4(a.ujp + drow);
        vy4 = ld4(a.vy + so + hrow); sxy4 = ld4(a.sxy + so + hrow); syz4 = ld4(a.syz + so + hrow);
        sts4v(vy_s, vy4); sts4v(sxy_s, sxy4); sts4v(syz_s, syz4);
        float4 px = make_float4(0.f, 0.f, 0.f, 0.f), ps = px, py = px, pz = px;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (xin >> k & 1) {
                const long long o = so + (long long)(j - 1) * 2 * fw + ((xin >> (4 + k) & 1 ? hr : i0) + k - 1);
                set(px, k, a.psi_vxx[o]);
                set(ps, k, a.psi_sxx[o]);
            }
        if (hy) {
            const long long o = so + (long long)(hy - 1) * pitch + (i0 - 1 + HX);
            py = ld4(a.psi_vyy_v + o);
            pz = ld4(a.psi_syy + o);
        }
        sts4v(psi_s, px); sts4v(psi_s + 4 * g.nthr, py); sts4v(psi_s + 8 * g.nthr, ps); sts4v(psi_s + 12 * g.nthr, pz);
    }
    if (own) {
        if (a.ws) sts4v(acc_s, ld4(a.ws + so + drow));
        if (MODE == TB_ADJ) {
            sts4v(acc_s + nown, ld4(a.gu + so + drow));
            sts4v(acc_s + 2 * nown, ld4(a.grho + so + drow));
        }
    }

    /* ---- sources in the region (every block that recomputes a point adds its signals), own receivers ---- */
    int *cnt = reinterpret_cast<int *>(tb_dyn + sm.cnt), *ent = reinterpret_cast<int *>(tb_dyn + sm.ent);
    unsigned short *point = reinterpret_cast<unsigned short *>(tb_dyn + sm.point);
    int *rl = reinterpret_cast<int *>(tb_dyn + sm.rec);
    {
        const int T = a.tl.ntiles;
        const int *go = a.tl.goff + (long long)slot * (T + 1);
        for (int q = __ldg(go) + t, g1 = __ldg(go + T); q < g1; q += blockDim.x) {
            const unsigned pk = (unsigned)__ldg(a.tl.gpt + q);
            const int c = (int)(pk & 0xffff) - (ox - g.gx), r = (int)(pk >> 16) - (oy - g.gy);
            if (c < 0 || c >= 4 * g.nv || r < 0 || r >= g.eh) continue;
            const int e0 = __ldg(a.tl.gbeg + q), nm = __ldg(a.tl.gbeg + q + 1) - e0, e = atomicAdd(cnt, nm);
            if (e + nm > g.nent) continue;               /* the host sized nent for the slot's sources */
            point[4 * (r * g.nv + c / 4) + (c & 3)] = (unsigned short)((e + 1) | nm << 12);
            for (int m = 0; m < nm; m++) ent[e + m] = __ldg(a.tl.src_id + e0 + m);
        }
        if (MODE != TB_ADJ && a.tl.sample) {
            const int *ro = a.tl.roff + (long long)slot * (T + 1);
            for (int q = __ldg(ro) + t, r1 = __ldg(ro + T); q < r1; q += blockDim.x) {
                const unsigned pk = (unsigned)__ldg(a.tl.rpt + q);
                const int c = (int)(pk & 0xffff) - ox, r = (int)(pk >> 16) - oy;
                if (c < 0 || c >= g.tw || r < 0 || r >= g.th) continue;
                const int e = atomicAdd(cnt + 1, 1);
                if (e >= g.nrec) continue;
                rl[e] = (r + g.gy + H) * wp + 4 + g.gx + c;
                rl[g.nrec + e] = __ldg(a.tl.rid + q);
            }
        }
    }
    __syncthreads();
    const int nent = min(cnt[0], g.nent), nrec = min(cnt[1], g.nrec);
    const ushort4 inj = reinterpret_cast<const ushort4 *>(point)[min(t, g.nthr - 1)];
    const bool has_inj = in && (inj.x | inj.y | inj.z | inj.w);
    const float *const sig = nent > 0 ? a.tl.sig + a.tl.sig_off[slot] : nullptr;
    const int ntr = nrec > 0 ? a.tl.rec_off[slot + 1] - a.tl.rec_off[slot] : 0;
    float *const seis = nrec > 0 ? a.tl.seis + a.tl.seis_off[slot] : nullptr;

    /* signals and stored fields of step q (0-based in the pass) into ring place q % TB_RING */
    auto fetch = [&](int q) {
        if (q < count) {
            const int nt = n_first + q, place = q % TB_RING;
            for (int e = t; e < nent; e += blockDim.x)
                tb_copy4(tb_dyn + sm.sig + place * g.nent + e,
                         sig + (long long)(nt - 1) * a.tl.sig_ts + (long long)ent[e] * a.tl.sig_ss);
            if (MODE == TB_ADJ && own) {
                const float *f = a.fwd + (long long)slot * a.fwd_slot_stride +
                                 store_idx(a.nt_total - nt, a.fwd_mod) * a.fwd_step_stride + drow;
                float *d = tb_dyn + sm.ring + place * 3 * nown + ((j - oy) * g.tw + (i0 - ox));
                tb_copy16(d, f);
                tb_copy16(d + nown, f + a.dstride);
                tb_copy16(d + 2 * nown, f + 2 * a.dstride);
            }
        }
        tb_commit();
    };
    const bool ring = MODE == TB_ADJ || nent > 0;      /* the same in all threads */
    if (ring) {
        fetch(0);
        fetch(1);
        fetch(2);
        tb_wait<2>();
    }
    __syncthreads();

    const int oy1 = min(oy + g.th - 1, ny);
    /* one thread per tile that the halo reaches into polls its count (every
       halo thread polling for itself: 500 x 200 24 % slower per round) */
    const int nbx = 2 * ((g.gx + g.tw - 1) / g.tw) + 1, nby = 2 * ((g.gy + g.th - 1) / g.th) + 1;
    auto wait_round = [&](unsigned need) {
        int ok = 1;
        for (int e = t; e < nbx * nby; e += blockDim.x) {
            const int cx = bx + e % nbx - nbx / 2, cy = by + e / nbx - nby / 2;
            if (cx >= 0 && cx < g.ntx && cy >= 0 && cy < g.nty && (cx != bx || cy != by))
                ok &= tb_poll(x.done + slot * tiles + cy * g.ntx + cx, need, a.wait_polls, a.status);
        }
        return ok;
    };
    int bad = 0, round = 0;
    for (int q = 0; q < count;) {
        const int ks = min(g.k, count - q);
        if (round > 0) {
            /* ---- neighbours' points of the previous round ---- */
            if (!__syncthreads_and(wait_round((unsigned)round))) { tb_wait<0>(); return; }
            if (in && !own) {
                const float *e = x.buf + ((long long)(round & 1) * a.nslots + slot) * TB_XFIELDS * a.dstride + drow;
                vy4 = __ldcg(reinterpret_cast<const float4 *>(e));
                sxy4 = __ldcg(reinterpret_cast<const float4 *>(e + a.dstride));
                syz4 = __ldcg(reinterpret_cast<const float4 *>(e + 2 * a.dstride));
                sts4v(vy_s, vy4); sts4v(sxy_s, sxy4); sts4v(syz_s, syz4);
                if (xin) {
                    sts4v(psi_s, __ldcg(reinterpret_cast<const float4 *>(e + 3 * a.dstride)));
                    sts4v(psi_s + 8 * g.nthr, __ldcg(reinterpret_cast<const float4 *>(e + 5 * a.dstride)));
                }
                if (hy) {
                    sts4v(psi_s + 4 * g.nthr, __ldcg(reinterpret_cast<const float4 *>(e + 4 * a.dstride)));
                    sts4v(psi_s + 12 * g.nthr, __ldcg(reinterpret_cast<const float4 *>(e + 6 * a.dstride)));
                }
            }
            __syncthreads();
        }
        for (int s = 0; s < ks; s++, q++) {
            const int nt = n_first + q, e = (ks - 1 - s) * R, place = q % TB_RING;
            if (ring) fetch(q + TB_RING - 1);

            /* ---- velocity half-step (v_body) on the rows that later steps read ---- */
            if (in && j >= oy - e - (H - 1) && j <= oy1 + e + H) {
                const float4 l = lds4v(sxy_s - 4), r = lds4v(sxy_s + 4);
                const float xs[12] = {l.x, l.y, l.z, l.w, sxy4.x, sxy4.y, sxy4.z, sxy4.w, r.x, r.y, r.z, r.w};
                float dx[4], dy[4];
#pragma unroll
                for (int m = 1; m <= H; m++) {
                    const float4 u = m == 1 ? syz4 : lds4v(syz_s + (m - 1) * wp), d = lds4v(syz_s - m * wp);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float tx = a.hc[m] * (xs[4 + k + m - 1] - xs[4 + k - m]);
                        const float ty = a.hc[m] * (get(u, k) - get(d, k));
                        if (m == 1) { dx[k] = tx; dy[k] = ty; }
                        else { dx[k] = dx[k] + tx; dy[k] = dy[k] + ty; }
                    }
                }
                if (xin)
                    tb_cpml_x(dx, psi_s, tb_dyn + sm.coef + 4 * vec, tb_dyn + sm.coef + 4 * g.nv + 4 * vec, xin, a.pml.K_x, i0,
                              hr, k_one);
                if (hy) tb_cpml_y(dy, psi_s + 4 * g.nthr, ya, yb, a.pml.K_y + hy, k_one);
                const float4 old4 = vy4;
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; k++) v[k] = get(b4, k) * a.dt * (dx[k] + dy[k]);
                div4_dh<P2>(v, a);
#pragma unroll
                for (int k = 0; k < 4; k++) set(vy4, k, get(vy4, k) + v[k]);
                if (MODE == TB_STORE && own) {
                    float c[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) c[k] = get(b4, k) * (dx[k] + dy[k]);
                    div4_dh<P2>(c, a);
                    st4ms(a.fwd + (long long)slot * a.fwd_slot_stride + store_idx(nt - 1, a.fwd_mod) * a.fwd_step_stride + drow,
                          make_float4(c[0], c[1], c[2], c[3]), nvalid);
                }
                if (MODE == TB_ADJ && own) {             /* g_rho += old vy * stored acceleration */
                    const float4 f = lds4v(tb_dyn + sm.ring + place * 3 * nown + ((j - oy) * g.tw + (i0 - ox)));
                    float4 c = lds4v(acc_s + 2 * nown);
                    c.x = c.x + (old4.x * f.x); c.y = c.y + (old4.y * f.y);
                    c.z = c.z + (old4.z * f.z); c.w = c.w + (old4.w * f.w);
                    sts4v(acc_s + 2 * nown, c);
                }
                if (has_inj) {                           /* sources of a point in the reference's order */
                    const float *sg = tb_dyn + sm.sig + place * g.nent;
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const unsigned p = k == 0 ? inj.x : k == 1 ? inj.y : k == 2 ? inj.z : inj.w;
                        if (!p) continue;
                        float w = get(vy4, k);
                        for (unsigned m = 0; m < p >> 12; m++) w = w + sg[(p & 0xfff) - 1 + m];
                        set(vy4, k, w);
                    }
                }
                sts4v(vy_s, vy4);
            }
            __syncthreads();

            /* ---- receiver samples (own points; vy after the injection) ---- */
            if (MODE != TB_ADJ)
                for (int r = t; r < nrec; r += blockDim.x)
                    seis[(long long)(nt - 1) * ntr + rl[g.nrec + r]] = tb_dyn[sm.vy + rl[r]];

            /* ---- stress half-step (s_body, L = 0) ---- */
            if (in && j >= oy - e && j <= oy1 + e) {
                const float4 l = lds4v(vy_s - 4), r = lds4v(vy_s + 4);
                const float xs[12] = {l.x, l.y, l.z, l.w, vy4.x, vy4.y, vy4.z, vy4.w, r.x, r.y, r.z, r.w};
                float dx[4], dy[4];
#pragma unroll
                for (int m = 1; m <= H; m++) {
                    const float4 u = lds4v(vy_s + m * wp), d = m == 1 ? vy4 : lds4v(vy_s - (m - 1) * wp);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float tx = a.hc[m] * (xs[4 + k + m] - xs[4 + k - m + 1]);
                        const float ty = a.hc[m] * (get(u, k) - get(d, k));
                        if (m == 1) { dx[k] = tx; dy[k] = ty; }
                        else { dx[k] = dx[k] + tx; dy[k] = dy[k] + ty; }
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k++) { dx[k] = dx[k] * a.dhi_el; dy[k] = dy[k] * a.dhi_el; }
                if (xin)
                    tb_cpml_x(dx, psi_s + 8 * g.nthr, tb_dyn + sm.coef + 8 * g.nv + 4 * vec,
                              tb_dyn + sm.coef + 12 * g.nv + 4 * vec, xin, a.pml.K_x_half, i0, hr, k_one);
                if (hy) tb_cpml_y(dy, psi_s + 12 * g.nthr, yah, ybh, a.pml.K_y_half + hy, k_one);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    set(sxy4, k, get(sxy4, k) + get(ui4, k) * dx[k]);
                    set(syz4, k, get(syz4, k) + get(uj4, k) * dy[k]);
                }
                sts4v(sxy_s, sxy4);
                sts4v(syz_s, syz4);
                if (own) {
                    /* finite check (a non-finite value never turns finite again) */
                    if (((nt & a.chk_mask) == 0 || nt >= a.nt_last) &&
                        !(isfinite(sxy4.x) && isfinite(sxy4.y) && isfinite(sxy4.z) && isfinite(sxy4.w) && isfinite(syz4.x) &&
                          isfinite(syz4.y) && isfinite(syz4.z) && isfinite(syz4.w) && isfinite(vy4.x)))
                        bad = 1;
                    if (MODE == TB_STORE) {              /* uy, uyx beside the acceleration */
                        float *f = a.fwd + (long long)slot * a.fwd_slot_stride +
                                   store_idx(nt - 1, a.fwd_mod) * a.fwd_step_stride + drow;
                        st4ms(f + a.dstride, make_float4(dy[0], dy[1], dy[2], dy[3]), nvalid);
                        st4ms(f + 2 * a.dstride, make_float4(dx[0], dx[1], dx[2], dx[3]), nvalid);
                    }
                    if (a.ws) {                          /* W += vy^2 */
                        float4 w = lds4v(acc_s);
#pragma unroll
                        for (int k = 0; k < 4; k++) set(w, k, get(w, k) + get(vy4, k) * get(vy4, k));
                        sts4v(acc_s, w);
                    }
                    if (MODE == TB_ADJ) {                /* g_u += uyx_fwd*sxy + uy_fwd*syz */
                        const float *f = tb_dyn + sm.ring + place * 3 * nown + ((j - oy) * g.tw + (i0 - ox));
                        const float4 fy = lds4v(f + nown), fu = lds4v(f + 2 * nown);
                        float4 c = lds4v(acc_s + nown);
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            set(c, k, get(c, k) + ((get(fu, k) * get(sxy4, k)) + (get(fy, k) * get(syz4, k))));
                        sts4v(acc_s + nown, c);
                    }
                }
            }
            if (ring) tb_wait<TB_RING - 2>();            /* the next step's signals have arrived */
            __syncthreads();
        }
        round++;
        const bool last = q >= count;
        if (!last || round == 1) {
            /* ---- own points to the exchange buffer of this round, then the flag ---- */
            if (own && !last) {
                float *e = x.buf + ((long long)(round & 1) * a.nslots + slot) * TB_XFIELDS * a.dstride + drow;
                __stcg(reinterpret_cast<float4 *>(e), vy4);
                __stcg(reinterpret_cast<float4 *>(e + a.dstride), sxy4);
                __stcg(reinterpret_cast<float4 *>(e + 2 * a.dstride), syz4);
                if (xin) {
                    __stcg(reinterpret_cast<float4 *>(e + 3 * a.dstride), lds4v(psi_s));
                    __stcg(reinterpret_cast<float4 *>(e + 5 * a.dstride), lds4v(psi_s + 8 * g.nthr));
                }
                if (hy) {
                    __stcg(reinterpret_cast<float4 *>(e + 4 * a.dstride), lds4v(psi_s + 4 * g.nthr));
                    __stcg(reinterpret_cast<float4 *>(e + 6 * a.dstride), lds4v(psi_s + 12 * g.nthr));
                }
            }
            __syncthreads();
            if (t == 0)                                  /* the barrier orders the block's stores before this release */
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(x.done + slot * tiles + tile), "r"((unsigned)round)
                             : "memory");
        }
    }
    if (round == 1) {
        /* a pass of one round: the neighbours have read the initial state before it is overwritten */
        if (!__syncthreads_and(wait_round(1u))) { tb_wait<0>(); return; }
    }
    tb_wait<0>();

    /* ---- own points, CPML memory and sums back to the slot ---- */
    if (own) {
        st4m(a.vy + so + hrow, vy4, nvalid);
        st4m(a.sxy + so + hrow, sxy4, nvalid);
        st4m(a.syz + so + hrow, syz4, nvalid);
        const float4 px = lds4v(psi_s), ps = lds4v(psi_s + 8 * g.nthr);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (xin >> k & 1) {
                const long long o = so + (long long)(j - 1) * 2 * fw + ((xin >> (4 + k) & 1 ? hr : i0) + k - 1);
                a.psi_vxx[o] = get(px, k);
                a.psi_sxx[o] = get(ps, k);
            }
        if (hy) {
            const long long o = so + (long long)(hy - 1) * pitch + (i0 - 1 + HX);
            st4m(a.psi_vyy_v + o, lds4v(psi_s + 4 * g.nthr), nvalid);
            st4m(a.psi_syy + o, lds4v(psi_s + 12 * g.nthr), nvalid);
        }
        if (a.ws) st4m(a.ws + so + drow, lds4v(acc_s), nvalid);
        if (MODE == TB_ADJ) {
            st4m(a.gu + so + drow, lds4v(acc_s + nown), nvalid);
            st4m(a.grho + so + drow, lds4v(acc_s + 2 * nown), nvalid);
        }
    }
    if (__syncthreads_or(bad) && t == 0) atomicOr(a.status, 1);
}

}  // namespace dsh
