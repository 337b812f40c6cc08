/*
 * Mixed-precision FIRE for one large network over the whole GPU, in spatial
 * tiles, with ONE grid barrier per FIRE step and every tile's read-only data
 * streamed into shared memory by TMA bulk copies.
 *
 * The cooperative grid kernel of fire_mixed.cu runs a step as four passes
 * separated by grid barriers (drift, item pass writing every bond's and
 * triple's FP32 force change to global memory, gather reading them back,
 * reduction by the last CTA); it is bound by the latency of those passes and
 * barriers.  Here one CTA per SM takes whole tiles (NetTile, nr_device.cuh)
 * and does a tile's whole step on chip:
 *   0. the tile's record (item references, anchor records, incidence,
 *      fcodes, halo list: one contiguous block) and its own nodes' state
 *      (contiguous in tile order) arrive in shared memory by cp.async.bulk,
 *      issued while the previous tile computes, the first tile's during the
 *      grid barrier (two stage buffers, an mbarrier each); a CTA with a
 *      single tile keeps it in shared memory between anchors;
 *   1. u, v, F of the halo (cp.async during the previous tile's gather);
 *   2. pass A (mixing, drift, half kick) for own AND halo nodes: the halo's
 *      drift is recomputed from the same inputs with the same operations as
 *      its owner's, so it has the same bits and needs no barrier;
 *   3. the item pass: every bond's and triple's FP32 force change into
 *      shared memory (boundary items are evaluated by each tile they touch);
 *   4. the gather of the own nodes in the canonical incidence order, half
 *      kick, the next step's u, v, F written, the step's partial sums.
 * Then one grid barrier; every CTA combines the CTAs' partials in CTA order
 * itself and advances an identical copy of the FIRE scalars.  The
 * arithmetic (double-float u, bond_dforce, tri_dforce, FP32 FIRE step, FP64
 * anchors and certification) is mixed_common.cuh's; per node the force is
 * the same sum in the same order as in the other mixed kernels.  Anchors
 * (rare) take two more barriers: X += u, then the FP64 force and the tile
 * records' anchor data.
 *
 * What bounds a step (65 536 nodes, one tile per SM, 6.3 us): items 1.2 us,
 * gather 1.3, pass A and halo 0.8, totals and scalars 1.2, barrier 1.7; the
 * step took 8.3 us when every step loaded the record and the own state again,
 * the totals' loads came in five dependent rounds, each triple entry of the
 * gather selected its share, and the item loops ended in nearly empty rounds.
 * 16 384 nodes 6.7 -> 4.8, 262 144 nodes 19.1 -> 15.6, 1 048 576 nodes 58.2 ->
 * 50.8 us: there 14 tiles a step pass through the SM, whose warps issue on
 * 45 % of the cycles (360 000 nodes: 42 %) and wait for shared memory and at
 * the barriers between the phases.  Of the last 5.8 us, 2.4 came from the
 * gather's entries in quads (four 2-byte loads of scattered addresses before),
 * 3.4 from pass A following the previous tile's gather without a barrier.  Two
 * groups of 512 threads with a tile each were slower (62 us): with one buffer
 * a group the loads are exposed, and the phases share the same pipes.
 *
 * Every wait is bounded: the grid barrier by a %globaltimer budget, the
 * mbarrier waits by the same budget; a wait that runs out sets the
 * network's abort flag (NR_ERR_TIMEOUT on the host), waits (bounded) for the
 * CTA's copy in flight, and returns.
 *
 * Compiled with --fmad=false; FP32 expressions use explicit fmaf().
 */
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fire_launch.h"
#include "mixed_common.cuh"
#include "nr_internal.h"

namespace nr {

/* ----- grid barrier: a monotonic counter, every CTA waits for all ----- */

/* Thread 0: arrives at the grid barrier, with release semantics, for a CTA
 * that has synchronised. */
__device__ __forceinline__ void tile_arrive(const NetTile &tl) {
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(tl.bar) : "memory");
}
/* Waits until all G CTAs have arrived at barrier number `epoch` (1, 2, ...)
 * of the launch; false when the wait exceeded budget_ns or another CTA gave
 * up (st->abort_flag); every thread of the CTA sees the same result. */
__device__ __forceinline__ bool tile_wait(const NetTile &tl, FireState *st, unsigned G, unsigned long long epoch,
                                          unsigned long long budget_ns, unsigned site, int *s_ok) {
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned long long target = epoch * (unsigned long long)G;
        unsigned long long t0 = 0, c;
        unsigned spins = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(tl.bar) : "memory");
            if (c >= target) break;
            if ((++spins & 63u) != 0) continue;
            if (*(volatile unsigned *)&st->abort_flag) {
                ok = 0;
                break;
            }
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 > budget_ns) {
                atomicExch(&st->abort_flag, 1u);
                atomicExch(&st->timeout_site, site);
                ok = 0;
                break;
            }
        }
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

/* The CTA's own barrier, then the grid's. */
__device__ __forceinline__ bool tile_barrier(const NetTile &tl, FireState *st, unsigned G, unsigned long long epoch,
                                             unsigned long long budget_ns, unsigned site, int *s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) tile_arrive(tl);
    return tile_wait(tl, st, G, epoch, budget_ns, site, s_ok);
}

/* ----- TMA bulk copy into shared memory, completion on an mbarrier ----- */

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)));
}

/* One thread: announce `bytes` of copies on the mbarrier's current phase. */
__device__ __forceinline__ void mbar_expect(unsigned long long *mbar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(bytes)
                 : "memory");
}
/* One thread: copy `bytes` (announced) from global src to shared dst (both
 * 16-byte aligned, bytes a multiple of 16: the host checks the layout). */
__device__ __forceinline__ void tma_copy(void *dst, const void *src, unsigned bytes, unsigned long long *mbar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(mbar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *mbar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(mbar)), "r"(parity)
        : "memory");
    return ok != 0;
}

/* Waits (every thread) until the mbarrier's phase `parity` completed, at
 * most budget_ns; false when it ran out. */
__device__ inline bool mbar_wait(unsigned long long *mbar, unsigned parity, unsigned long long budget_ns) {
    if (mbar_try_wait(mbar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (unsigned spins = 0;; ++spins) {
        if (mbar_try_wait(mbar, parity)) return true;
        if ((spins & 15u) == 15u && global_ns() - t0 > budget_ns) return false;
    }
}

/* ----- per-thread asynchronous copies into shared memory (cp.async) ----- */

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

/* ----- per-tile pieces ----- */

/* A tile's node state in shared memory: u, v, F of its own nodes (local 0
 * .. no - 1) and halo nodes (no .. no + nh - 1), the own nodes' anchor
 * force.  Two of them: the next tile's state is copied in while the current
 * tile computes. */
struct TileState {
    float4 *u;  /* double-float u {hi.x, hi.y, lo.x, lo.y} */
    float4 *vf; /* {v.x, v.y, F.x, F.y} */
    float4 *fa; /* own nodes: double-float anchor force {hi.x, hi.y, lo.x, lo.y} */
};
__host__ __device__ inline size_t tile_state_bytes(int max_nodes, int max_own) {
    return 32 * (size_t)max_nodes + 16 * (size_t)max_own;
}
__device__ inline TileState tile_state_at(unsigned char *base, int max_nodes, int max_own) {
    TileState t;
    t.u = reinterpret_cast<float4 *>(base);
    t.vf = t.u + max_nodes;
    t.fa = t.vf + max_nodes;
    return t;
}

/* One thread: starts the bulk copies of tile td's record and own state
 * (state copy `cur`) into a stage buffer and a state buffer.  Own state is
 * contiguous in tile order; own_pos is a multiple of 16, a node 16 bytes. */
__device__ __forceinline__ void load_tile(const NetTile &tl, const TileDesc &td, int cur, unsigned char *rec,
                                          const TileState &ts, unsigned long long *mbar) {
    const unsigned total = tile_segs(td).total, own = 16u * (unsigned)td.no;
    mbar_expect(mbar, total + 3u * own);
    tma_copy(rec, tl.ro + td.ro_off, total, mbar);
    tma_copy(ts.u, tl.u[cur] + td.own_pos, own, mbar);
    tma_copy(ts.vf, tl.vf[cur] + td.own_pos, own, mbar);
    tma_copy(ts.fa, tl.fa + td.own_pos, own, mbar);
}
/* Starts the copies of tile td's halo state (its record already in shared
 * memory). */
__device__ __forceinline__ void issue_halo(const NetTile &tl, const TileDesc &td, const unsigned char *rec, int cur,
                                           const TileState &ts) {
    const int *halo = reinterpret_cast<const int *>(rec + tile_segs(td).halo);
    for (int h = threadIdx.x; h < td.nh; h += blockDim.x) {
        const int pp = halo[h];
        cp_async16(ts.u + td.no + h, tl.u[cur] + pp);
        cp_async16(ts.vf + td.no + h, tl.vf[cur] + pp);
    }
}

/* Pass A of one node (mixed_pass_a's operations). */
__device__ __forceinline__ void tile_pass_a(const Coef &c, float4 &w, float2 &v, const float2 F) {
    if (c.mix_pending) {
        v.x = fmaf(c.na, v.x, v.x);
        v.y = fmaf(c.na, v.y, v.y);
        v.x = fmaf(c.a, F.x, v.x);
        v.y = fmaf(c.a, F.y, v.y);
        if (c.zero_v) v = make_float2(0.f, 0.f);
    }
    if (!c.done) {
        df_add(w.x, w.z, fmaf(c.dt, v.x, c.dtsq * F.x));
        df_add(w.y, w.w, fmaf(c.dt, v.y, c.dtsq * F.y));
        v.x = fmaf(c.dtm, F.x, v.x);
        v.y = fmaf(c.dtm, F.y, v.y);
    }
}

/* Pass A of local nodes first, first + NT, ... < end of a state buffer, in
 * place. */
template <int NT>
__device__ __forceinline__ void tile_pass_range(const Coef &c, const TileState &ts, int first, int end) {
    for (int k = first; k < end; k += NT) {
        float4 w = ts.u[k];
        const float4 q = ts.vf[k];
        float2 v = make_float2(q.x, q.y);
        tile_pass_a(c, w, v, make_float2(q.z, q.w));
        ts.u[k] = w;
        ts.vf[k] = make_float4(v.x, v.y, q.z, q.w);
    }
}

/* FP64 anchor evaluation: X += u was done; every node's canonical FP64
 * force (d.f), its double-float copy fa and F = fa_hi in the current state
 * copy (tile order); the anchor data of the CTA's tiles' records.  Returns
 * the CTA partials of |F|^2 (sum) and max |F|^2 in thread 0. */
static __device__ __noinline__ void tile_anchor_eval(const NetDev &d, const NetTile &tl, int cur, double *dslots,
                                                     double &tF2, double &tM2) {
    const double W = d.width;
    double F2 = 0.0, M2 = 0.0;
    const int G = gridDim.x;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < tl.n_pos; p += G * blockDim.x) {
        const int i = tl.node_of_pos[p];
        if (i < 0) continue;
        double fx, fy;
        node_force_fp64_own(d, i, fx, fy);
        d.f[i] = make_double2(fx, fy);
        const float hx = (float)fx, hy = (float)fy;
        tl.fa[p] = make_float4(hx, hy, (float)(fx - (double)hx), (float)(fy - (double)hy));
        float4 q = tl.vf[cur][p]; /* v stays, F = the anchor force */
        q.z = hx;
        q.w = hy;
        tl.vf[cur][p] = q;
        const double t = dot2(fx, fy, fx, fy);
        F2 += t;
        M2 = fmax(M2, t);
    }
    for (int t = blockIdx.x; t < tl.n_tiles; t += G) {
        const TileDesc td = tl.desc[t];
        const TileSegs g = tile_segs(td);
        unsigned char *rec = tl.ro + td.ro_off;
        float4 *mb = reinterpret_cast<float4 *>(rec + g.mb);
        float2 *sk = reinterpret_cast<float2 *>(rec + g.sk);
        float4 *arms = reinterpret_cast<float4 *>(rec + g.arms);
        float2 *pk = reinterpret_cast<float2 *>(rec + g.pk);
        if (d.use_bonds)
            for (int k = threadIdx.x; k < td.nb; k += blockDim.x) {
                const int b = tl.bid[td.bond_off + k];
                const int4 r = d.bond[b];
                const double2 p1 = d.x[r.x], p2 = d.x[r.y];
                const double rx = (p2.x + wrap_shift(r.z, W)) - p1.x, ry = p2.y - p1.y;
                const double kk = d.bond_k ? d.bond_k[b] : d.ks;
                const float hx = (float)rx, hy = (float)ry;
                mb[k] = make_float4(hx, hy, (float)(rx - (double)hx), (float)(ry - (double)hy));
                sk[k] = make_float2((float)(sqrt_ieee(fma(rx, rx, ry * ry)) - d.bond_l0[b]), (float)kk);
            }
        if (d.use_triples)
            for (int k = threadIdx.x; k < td.nt; k += blockDim.x) {
                const int tt = tl.tid[td.tri_off + k];
                const int4 r = d.tri[tt];
                const double2 ph = d.x[r.x], pj = d.x[r.y], pkk = d.x[r.z];
                const int wj = (signed char)(r.w & 0xff), wk = (signed char)((r.w >> 8) & 0xff);
                const double ax = wrap_add(pj.x, wj, W) - ph.x, ay = pj.y - ph.y;
                const double bx = wrap_add(pkk.x, wk, W) - ph.x, by = pkk.y - ph.y;
                const double kb = d.tri_kb ? d.tri_kb[tt] : d.kb;
                const double phi0 = d.tri_phi0 ? d.tri_phi0[tt] : 0.0;
                arms[k] = make_float4((float)ax, (float)ay, (float)bx, (float)by);
                pk[k] = make_float2((float)bend_dtheta(ax, ay, bx, by, phi0), (float)kb);
            }
    }
    /* the records are read later by bulk copies (the async proxy) */
    asm volatile("fence.proxy.async.global;" ::: "memory");
    anchor_reduce(F2, M2, dslots, tF2, tM2);
}

/* Totals of the CTAs' FP64 anchor partials, in CTA order (thread 0). */
static __device__ __noinline__ void tile_anchor_totals(const NetTile &tl, int G, double &F2, double &M2) {
    double s = 0.0, m = 0.0;
    for (int c = 0; c < G; ++c) {
        s = s + __ldcg(tl.dpart + 2 * c);
        m = fmax(m, __ldcg(tl.dpart + 2 * c + 1));
    }
    F2 = s;
    M2 = m;
}

/* Instantiated for 512 or 768 threads per CTA with one CTA per SM (768: more
 * warps to hide latency, fewer registers per thread), and for 256 threads
 * with two CTAs per SM (smaller tiles; one CTA's barriers overlap the
 * other's work). */

/* Shared memory by which the tile size is chosen: records with the entries not
 * in quads, and item results with arrays of their own (16 B a triple, 8 B a
 * bond; they now overwrite the record), so that the tiles, and with them the
 * order of the sums, stay what they were. */
size_t tile_plan_smem(const TileHost &th) {
    return 2 * (size_t)th.max_plain + 2 * tile_state_bytes(th.max_nodes, th.max_own) + 16 * (size_t)th.max_tris +
           8 * (size_t)th.max_bonds;
}

constexpr int kDescCache = 32;

/* A wait that ran out: record the timeout, let every copy in flight land
 * (bounded waits; n0, n1: loads issued into each buffer that were not waited
 * for).  Kept out of line: captured by reference, the counters and with them
 * the buffers' addresses would live in local memory. */
static __device__ __noinline__ void tile_abort(FireState *st, unsigned long long *mbar, bool n0, unsigned par0, bool n1,
                                               unsigned par1, unsigned long long budget_ns) {
    if (threadIdx.x == 0) {
        atomicExch(&st->abort_flag, 1u);
        atomicExch(&st->timeout_site, 25u);
    }
    cp_async_wait_all();
    if (n0) mbar_wait(&mbar[0], par0, budget_ns);
    if (n1) mbar_wait(&mbar[1], par1, budget_ns);
}

/* resident: one tile per CTA at most.  Its record and own state stay in shared
 * memory between anchors, a step reads only the halo; the item results then go
 * to the second stage buffer (a streamed record is overwritten in place).
 * quads: the layout of the incidence entries (NetTile). */
template <int NT, int MINB, bool resident, bool quads>
__global__ void __launch_bounds__(NT, MINB)
    k_fire_tile_mixed(NetDev d, NetTile tl, FireParamsDev p, unsigned long long budget_ns) {
    extern __shared__ float4 s_dyn[];
    __shared__ MixShared sh;
    __shared__ __align__(8) unsigned long long s_mbar[2];
    __shared__ int s_fail, s_ok;
    /* FIRE scalars, advanced by thread 0 of every CTA (identical copies) */
    __shared__ MixScal s;
    __shared__ MixParams q;
    /* the descriptors of the CTA's first kDescCache tiles, loaded once: a
     * tile's first instructions then wait on shared memory, not on L2 */
    __shared__ TileDesc s_desc[kDescCache];
    unsigned char *dyn = reinterpret_cast<unsigned char *>(s_dyn);
    unsigned char *const stage0 = dyn, *const stage1 = dyn + tl.max_ro;
    const size_t sbytes = tile_state_bytes(tl.max_nodes, tl.max_own);
    const TileState ts0 = tile_state_at(dyn + 2 * (size_t)tl.max_ro, tl.max_nodes, tl.max_own);
    const TileState ts1 = tile_state_at(dyn + 2 * (size_t)tl.max_ro + sbytes, tl.max_nodes, tl.max_own);
    const unsigned G = gridDim.x;
    FireState *st = d.st;
    unsigned long long epoch = 0;
    unsigned uses0 = 0u, uses1 = 0u; /* completed phases of each stage buffer's mbarrier */
    unsigned iss0 = 0u, iss1 = 0u;   /* loads issued into each stage buffer */
    if (threadIdx.x == 0) {
        q = mix_params(p, d.sqrt_dof);
        mbar_init(&s_mbar[0]);
        mbar_init(&s_mbar[1]);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_fail = 0;
    }
    __syncthreads();
    int cur = 0;
    for (int i = blockIdx.x * NT + threadIdx.x; i < tl.n_pos; i += G * NT) {
        tl.u[0][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        tl.vf[0][i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    double tF2, tM2;
    tile_anchor_eval(d, tl, cur, sh.dslots, tF2, tM2);
    if (threadIdx.x == 0) {
        tl.dpart[2 * blockIdx.x] = tF2;
        tl.dpart[2 * blockIdx.x + 1] = tM2;
    }
    if (!tile_barrier(tl, st, G, ++epoch, budget_ns, 21, &s_ok)) return;
    if (threadIdx.x == 0) {
        double F2, M2;
        tile_anchor_totals(tl, G, F2, M2);
        mix_init(s, q);
        mix_certify(s, p, d.sqrt_dof, F2, M2);
        sh.coef = coef_of(s, 0);
    }
    __syncthreads();
    const int n_mine = (int)blockIdx.x < tl.n_tiles ? (tl.n_tiles - 1 - (int)blockIdx.x) / (int)G + 1 : 0;
    for (int k = threadIdx.x; k < min(n_mine, kDescCache); k += NT) s_desc[k] = tl.desc[blockIdx.x + k * G];
    __syncthreads();
    /* the gather's threads: the order of the sums does not depend on NT */
    constexpr int NG = NT < 512 ? NT : 512;
    auto desc = [&](int k) -> TileDesc { return k < kDescCache ? s_desc[k] : tl.desc[blockIdx.x + k * G]; };
    bool loaded = false; /* tile 0 is in buffer 0, or its load in flight */
    if (resident && quads && n_mine > 0 && threadIdx.x < 4) /* ordered by the barriers before the first gather */
        reinterpret_cast<float *>(stage1 + tile_segs(s_desc[0]).zero)[threadIdx.x] = 0.f;
    for (;;) {
        const Coef &c = sh.coef;
        if (c.done) {
            /* the last pass A: mixing of v only (u is 0 after the certifying
             * anchor); the FP64 velocities out */
            for (int pp = blockIdx.x * NT + threadIdx.x; pp < tl.n_pos; pp += G * NT) {
                const int i = tl.node_of_pos[pp];
                if (i < 0) continue;
                float4 w = tl.u[cur][pp];
                const float4 q = tl.vf[cur][pp];
                float2 v = make_float2(q.x, q.y);
                tile_pass_a(c, w, v, make_float2(q.z, q.w));
                d.v[i] = make_double2((double)v.x, (double)v.y);
            }
            break;
        }
        const int nxt = cur ^ 1;
        float P = 0.f, V2 = 0.f, Fs = 0.f, M2f = 0.f, A = 0.f;
        /* the pipeline, two barriers a streamed tile: the record and own state (TMA)
         * of tile k + 1 are in flight while tile k's items and gather run, its
         * halo state (cp.async) during the gather, and its pass A follows the
         * gather directly: a thread waits only for what it reads, the bulk
         * copies (own nodes) and its own halo copies (the same thread's
         * nodes), so that the threads without a node to gather start it while
         * the others sum */
        if (n_mine > 0) {
            const TileDesc td0 = desc(0);
            if (!loaded) {
                if (threadIdx.x == 0) {
                    /* what other CTAs wrote at the anchor and its barrier
                     * made visible, before bulk copies read it */
                    asm volatile("fence.proxy.async;" ::: "memory");
                    load_tile(tl, td0, cur, stage0, ts0, &s_mbar[0]);
                }
                ++iss0;
                loaded = true;
            }
            bool in = true;
            if (iss0 > uses0) {
                in = mbar_wait(&s_mbar[0], uses0 & 1u, budget_ns);
                if (in) ++uses0;
                else s_fail = 1;
            }
            if (in) issue_halo(tl, td0, stage0, cur, ts0); /* only from a record that arrived */
            if (resident) {
                /* nothing else to do meanwhile: own and halo nodes in one
                 * sequence over the threads (5.0 us a step against 5.3 at
                 * 22 500 nodes) */
                cp_async_wait_all();
                __syncthreads();
                if (in) tile_pass_range<NT>(c, ts0, threadIdx.x, td0.no + td0.nh);
            } else if (in) {
                tile_pass_range<NT>(c, ts0, threadIdx.x, td0.no);
                cp_async_wait_all();
                tile_pass_range<NT>(c, ts0, td0.no + threadIdx.x, td0.no + td0.nh);
            }
            if (!resident) loaded = false;
        }
        for (int k = 0; k < n_mine; ++k) {
            const int b = k & 1;
            const TileDesc td = desc(k);
            const bool more = k + 1 < n_mine;
            const TileDesc tn = more ? desc(k + 1) : td;
            float4 *const sc_u = b ? ts1.u : ts0.u, *const sc_vf = b ? ts1.vf : ts0.vf, *const sc_fa = b ? ts1.fa : ts0.fa;
            const TileState sn{b ? ts0.u : ts1.u, b ? ts0.vf : ts1.vf, b ? ts0.fa : ts1.fa};
            unsigned char *const rec_n = b ? stage0 : stage1;
            __syncthreads(); /* this tile's pass A; the previous tile's gather is done with the other buffers */
            if (s_fail) {
                tile_abort(st, s_mbar, iss0 > uses0, uses0 & 1u, iss1 > uses1, uses1 & 1u, budget_ns);
                return;
            }
            /* the next tile: its halo list straight from memory (no anchor
             * changes it), before its record is here */
            const int *const halo_n = reinterpret_cast<const int *>(tl.ro + tn.ro_off + tile_segs(tn).halo);
            int hp = 0;
            if (more) {
                if (threadIdx.x == 0) load_tile(tl, tn, cur, rec_n, sn, &s_mbar[b ^ 1]);
                if (b) ++iss0;
                else ++iss1;
                if ((int)threadIdx.x < tn.nh) hp = __ldg(halo_n + threadIdx.x);
            }
            const TileSegs g = tile_segs(td);
            const int no = td.no, op = td.own_pos;
            unsigned char *const rec = b ? stage1 : stage0;
            unsigned char *const out = resident ? stage1 : rec;
            /* item pass: groups of 32 triples, then of 32 bonds, dealt to the
             * warps in one sequence, so that no warp idles in a last round of
             * either.  A result replaces the anchor data it came from:
             *   bond    sk    force change on node i
             *   triple  arms  {dF_j, dF_k};  pk  the hinge's -(dF_j + dF_k);
             *           tref  the hinge's sum of |components| (first word)
             * so that the gather adds what it loads, without a select per
             * role (30 instructions an entry before). */
            {
                const int lane = threadIdx.x & 31, ntg = d.use_triples ? (td.nt + 31) >> 5 : 0,
                          nbg = d.use_bonds ? (td.nb + 31) >> 5 : 0;
                const unsigned *bref = reinterpret_cast<const unsigned *>(rec + g.bref);
                const float4 *mb = reinterpret_cast<const float4 *>(rec + g.mb);
                const float2 *sk = reinterpret_cast<const float2 *>(rec + g.sk);
                const uint2 *tref = reinterpret_cast<const uint2 *>(rec + g.tref);
                const float4 *arms = reinterpret_cast<const float4 *>(rec + g.arms);
                const float2 *pk = reinterpret_cast<const float2 *>(rec + g.pk);
                float2 *o_b = reinterpret_cast<float2 *>(out + g.sk);
                float4 *o_t = reinterpret_cast<float4 *>(out + g.arms);
                float2 *o_h = reinterpret_cast<float2 *>(out + g.pk);
                float2 *o_m = reinterpret_cast<float2 *>(out + g.tref);
                for (int w = threadIdx.x >> 5; w < ntg + nbg; w += NT / 32) {
                    if (w < ntg) {
                        const int kk = 32 * w + lane;
                        if (kk >= td.nt) continue;
                        const uint2 r = tref[kk];
                        const float4 uh = sc_u[r.x & 0xffffu], uj = sc_u[r.x >> 16], uk = sc_u[r.y];
                        const float2 hh = make_float2(uh.x, uh.y), hl = make_float2(uh.z, uh.w);
                        float2 dFj, dFk;
                        tri_dforce(arms[kk], pk[kk], u_diff(make_float2(uj.x, uj.y), make_float2(uj.z, uj.w), hh, hl),
                                   u_diff(make_float2(uk.x, uk.y), make_float2(uk.z, uk.w), hh, hl), dFj, dFk);
                        o_t[kk] = make_float4(dFj.x, dFj.y, dFk.x, dFk.y);
                        o_h[kk] = make_float2(-(dFj.x + dFk.x), -(dFj.y + dFk.y));
                        o_m[kk].x = ((fabsf(dFj.x) + fabsf(dFj.y)) + fabsf(dFk.x)) + fabsf(dFk.y);
                    } else {
                        const int kk = 32 * (w - ntg) + lane;
                        if (kk >= td.nb) continue;
                        const unsigned r = bref[kk];
                        const float4 ui = sc_u[r & 0xffffu], uj = sc_u[r >> 16];
                        float2 dh, dlo;
                        u_diff2(make_float2(uj.x, uj.y), make_float2(uj.z, uj.w), make_float2(ui.x, ui.y),
                                make_float2(ui.z, ui.w), dh, dlo);
                        o_b[kk] = bond_dforce(mb[kk], sk[kk], dh, dlo);
                    }
                }
            }
            if (more)
                for (int h = threadIdx.x; h < tn.nh; h += NT) {
                    const int pp = h == (int)threadIdx.x ? hp : __ldg(halo_n + h);
                    cp_async16(sn.u + tn.no + h, tl.u[cur] + pp);
                    cp_async16(sn.vf + tn.no + h, tl.vf[cur] + pp);
                }
            __syncthreads();
            /* gather of the own nodes, half kick, the next step's state */
            const unsigned short *iptr = reinterpret_cast<const unsigned short *>(rec + g.iptr);
            const unsigned short *ibe = reinterpret_cast<const unsigned short *>(rec + g.ibe);
            const unsigned short *inc = reinterpret_cast<const unsigned short *>(rec + g.inc);
            const ushort2 *cnt = reinterpret_cast<const ushort2 *>(rec + g.cnt);
            const unsigned *gq = reinterpret_cast<const unsigned *>(rec + g.gq);
            const unsigned char *fcode = rec + g.fcode;
            const int to_mag = (int)g.tref - (int)g.pk;
            for (int kk = threadIdx.x; (int)threadIdx.x < NG && kk < no; kk += NG) {
                const unsigned fc = fcode[kk];
                const float4 fa = sc_fa[kk];
                const float2 ah = make_float2(fa.x, fa.y), al = make_float2(fa.z, fa.w);
                float2 F = make_float2(0.f, 0.f);
                if (fc != 0) {
                    /* the node's bond entries, then its triple entries (the
                     * canonical order), four loads at a time; own nodes are
                     * ordered by list lengths */
                    float2 dF = make_float2(0.f, 0.f);
                    float mag = 0.f;
                    if (quads) {
                        const ushort2 n = cnt[kk];
                        const uint2 *qp = reinterpret_cast<const uint2 *>(inc) + gq[kk >> 5] + (kk & 31);
                        const int nbe = n.x, nen = n.y;
                        for (int e = 0; e < nen; e += 4, qp += 32) {
                            const uint2 w = *qp;
                            const unsigned code[4] = {w.x & 0xffffu, w.x >> 16, w.y & 0xffffu, w.y >> 16};
                            float2 df[4];
                            float mg[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const unsigned char *at = out + 8u * (code[j] & 0x7fffu);
                                const bool flag = (code[j] >> 15) != 0, bond = e + j < nbe;
                                df[j] = neg_if(*reinterpret_cast<const float2 *>(at), flag && bond ? 1u : 0u);
                                mg[j] = fabsf(df[j].x) + fabsf(df[j].y);
                                if (flag && !bond) mg[j] = *reinterpret_cast<const float *>(at + to_mag);
                            }
                            /* the zeros that fill up the last quad change
                             * nothing: no sum here is ever -0 */
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                dF.x += df[j].x;
                                dF.y += df[j].y;
                                mag += mg[j];
                            }
                        }
                    } else {
                        const int e0 = iptr[kk], eb = ibe[kk], e1 = iptr[kk + 1];
                        for (int e = e0; e < eb; e += 4) {
                            float2 df[4];
                            unsigned code[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) code[j] = inc[min(e + j, eb - 1)];
#pragma unroll
                            for (int j = 0; j < 4; ++j) df[j] = *reinterpret_cast<const float2 *>(out + 8u * (code[j] & 0x7fffu));
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (e + j < eb) {
                                    df[j] = neg_if(df[j], code[j] >> 15);
                                    dF.x += df[j].x;
                                    dF.y += df[j].y;
                                    mag += fabsf(df[j].x) + fabsf(df[j].y);
                                }
                        }
                        for (int e = eb; e < e1; e += 4) {
                            float2 df[4];
                            float mg[4];
                            unsigned code[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) code[j] = inc[min(e + j, e1 - 1)];
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const unsigned char *at = out + 8u * (code[j] & 0x7fffu);
                                df[j] = *reinterpret_cast<const float2 *>(at);
                                mg[j] = fabsf(df[j].x) + fabsf(df[j].y);
                                if (code[j] >> 15) mg[j] = *reinterpret_cast<const float *>(at + to_mag);
                            }
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (e + j < e1) {
                                    dF.x += df[j].x;
                                    dF.y += df[j].y;
                                    mag += mg[j];
                                }
                        }
                    }
                    A = fmaxf(A, mag);
                    F.x = ah.x + (al.x + dF.x);
                    F.y = ah.y + (al.y + dF.y);
                    if (!(fc & 1)) F.x = 0.f;
                    if (!(fc & 2)) F.y = 0.f;
                }
                const float4 q = sc_vf[kk];
                float2 v = make_float2(q.x, q.y);
                v.x = fmaf(c.dtm, F.x, v.x);
                v.y = fmaf(c.dtm, F.y, v.y);
                const float4 vf = make_float4(v.x, v.y, F.x, F.y);
                tl.u[nxt][op + kk] = sc_u[kk];
                tl.vf[nxt][op + kk] = vf;
                if (resident) sc_vf[kk] = vf;
                P += fmaf(v.x, F.x, v.y * F.y);
                V2 += fmaf(v.x, v.x, v.y * v.y);
                const float f2 = fmaf(F.x, F.x, F.y * F.y);
                Fs += f2;
                M2f = fmaxf(M2f, f2);
            }
            /* the shared memory written here, before bulk copies (the async
             * proxy) overwrite it; the next tile's barrier orders the rest */
            if (!resident) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (more) {
                if (mbar_wait(&s_mbar[b ^ 1], (b ? uses0 : uses1) & 1u, budget_ns)) {
                    if (b) ++uses0;
                    else ++uses1;
                    tile_pass_range<NT>(c, sn, threadIdx.x, tn.no);
                    cp_async_wait_all();
                    tile_pass_range<NT>(c, sn, tn.no + threadIdx.x, tn.no + tn.nh);
                } else {
                    s_fail = 1;
                }
            }
        }
        /* the next state just written, before bulk copies read it */
        if (!resident) asm volatile("fence.proxy.async.global;" ::: "memory");
        warp_part(Part{P, V2, Fs, M2f, A}, sh.slots);
        __syncthreads();
        if (threadIdx.x < 32) {
            const Part t = block_totals(sh.slots);
            if (threadIdx.x < 5) {
                /* two copies by step parity: a CTA that runs ahead into the
                 * next step writes the other copy while the rest still read
                 * this one */
                float v = t.P;
                if (threadIdx.x == 1) v = t.V2;
                if (threadIdx.x == 2) v = t.F2;
                if (threadIdx.x == 3) v = t.M2;
                if (threadIdx.x == 4) v = t.A;
                tl.cpart[(5 * (size_t)cur + threadIdx.x) * G + blockIdx.x] = v;
            }
        }
        /* the first tile's record and own state (written by this CTA) of the
         * next step travel during the barrier and the totals */
        const bool ahead = !resident && n_mine > 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            tile_arrive(tl);
            if (ahead) load_tile(tl, s_desc[0], nxt, stage0, ts0, &s_mbar[0]);
        }
        if (!tile_wait(tl, st, G, ++epoch, budget_ns, 22, &s_ok)) {
            if (ahead) mbar_wait(&s_mbar[0], uses0 & 1u, budget_ns);
            return;
        }
        if (ahead) {
            ++iss0;
            loaded = true;
        }
        if (threadIdx.x < 32) {
            /* lane l accumulates CTAs l, l + 32, ... in order, then the
             * butterfly: the same totals in every CTA.  160 CTAs' loads are
             * in flight at once (a loop paid an L2 round trip per 32) */
            Part t{0.f, 0.f, 0.f, 0.f, 0.f};
            const float *cp = tl.cpart + 5 * (size_t)cur * G;
            for (int k0 = threadIdx.x; k0 < (int)G; k0 += 160) {
                float v[5][5];
#pragma unroll
                for (int r = 0; r < 5; ++r)
#pragma unroll
                    for (int w = 0; w < 5; ++w) v[r][w] = __ldcg(cp + w * G + min(k0 + 32 * r, (int)G - 1));
#pragma unroll
                for (int r = 0; r < 5; ++r)
                    if (k0 + 32 * r < (int)G) {
                        t.P += v[r][0];
                        t.V2 += v[r][1];
                        t.F2 += v[r][2];
                        t.M2 = fmaxf(t.M2, v[r][3]);
                        t.A = fmaxf(t.A, v[r][4]);
                    }
            }
            t = warp_reduce(t);
            if (threadIdx.x == 0) {
                mix_step(s, q, t);
                sh.coef = coef_of(s, need_anchor(s, q, t));
            }
        }
        __syncthreads();
        cur = nxt;
        if (sh.coef.anchor) {
            /* the load under way, or the resident tile, will be stale */
            if (iss0 > uses0) {
                if (!mbar_wait(&s_mbar[0], uses0 & 1u, budget_ns)) {
                    tile_abort(st, s_mbar, iss0 > uses0, uses0 & 1u, iss1 > uses1, uses1 & 1u, budget_ns);
                    return;
                }
                ++uses0;
            }
            loaded = false;
            asm volatile("fence.proxy.async;" ::: "memory"); /* the buffers are loaded again */
            /* X += u (FP64), u = 0, then the FP64 anchor */
            for (int pp = blockIdx.x * NT + threadIdx.x; pp < tl.n_pos; pp += G * NT) {
                const int i = tl.node_of_pos[pp];
                if (i < 0) continue;
                const float4 w = tl.u[cur][pp];
                double2 x = d.x[i];
                x.x = x.x + ((double)w.x + (double)w.z);
                x.y = x.y + ((double)w.y + (double)w.w);
                d.x[i] = x;
                tl.u[cur][pp] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (!tile_barrier(tl, st, G, ++epoch, budget_ns, 23, &s_ok)) return;
            tile_anchor_eval(d, tl, cur, sh.dslots, tF2, tM2);
            if (threadIdx.x == 0) {
                tl.dpart[2 * blockIdx.x] = tF2;
                tl.dpart[2 * blockIdx.x + 1] = tM2;
            }
            if (!tile_barrier(tl, st, G, ++epoch, budget_ns, 24, &s_ok)) return;
            if (threadIdx.x == 0) {
                double F2, M2;
                tile_anchor_totals(tl, G, F2, M2);
                mix_certify(s, p, d.sqrt_dof, F2, M2);
                sh.coef = coef_of(s, 0);
            }
            __syncthreads();
            /* every CTA reads dpart before any CTA's next anchor rewrites
             * it: at least one step barrier lies between two anchors */
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) mix_report(st, s);
}

/* ------------------------------------------------------------------ */
/* Host side: layout and launch                                         */
/* ------------------------------------------------------------------ */

/* Dynamic shared memory of a CTA: two record buffers and two node-state
 * buffers. */
size_t tile_smem(const NetTile &tl) {
    return 2 * (size_t)tl.max_ro + 2 * tile_state_bytes(tl.max_nodes, tl.max_own);
}

/* The kernel instantiation for `threads` per CTA (512, 768 or 256). */
template <bool resident, bool quads>
static const void *tile_kernel_of(int threads) {
    if (threads == 256) return (const void *)k_fire_tile_mixed<256, 2, resident, quads>;
    if (threads == 768) return (const void *)k_fire_tile_mixed<768, 1, resident, quads>;
    return (const void *)k_fire_tile_mixed<512, 1, resident, quads>;
}
static const void *tile_kernel(int threads, bool resident, bool quads) {
    if (quads) return resident ? tile_kernel_of<true, true>(threads) : tile_kernel_of<false, true>(threads);
    return resident ? tile_kernel_of<true, false>(threads) : tile_kernel_of<false, false>(threads);
}

/* CTAs of the cooperative launch: co-resident CTAs per SM times SMs (0 when
 * the kernel cannot launch with this shared memory). */
int tile_grid_ctas(const NetTile &tl, int threads) {
    const size_t smem = tile_smem(tl);
    int dev = 0, sms = 0, least = 1 << 30;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    for (const bool resident : {false, true}) {
        const void *k = tile_kernel(threads, resident, tl.quads != 0);
        int per_sm = 0;
        if (allow_dynamic_smem(k, smem) != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem) != cudaSuccess) return 0;
        least = std::min(least, per_sm);
    }
    return least * sms;
}

cudaError_t launch_mixed_tile(const NetDev &d, const NetTile &tl, const FireParamsDev &p, int ctas, int threads,
                              unsigned long long budget_ns, cudaStream_t stream) {
    const void *k = tile_kernel(threads, tl.n_tiles <= ctas, tl.quads != 0);
    cudaError_t e = allow_dynamic_smem(k, tile_smem(tl));
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(tl.bar, 0, sizeof(unsigned long long), stream)) != cudaSuccess) return e;
    NetDev dd = d;
    NetTile tt = tl;
    FireParamsDev pp = p;
    unsigned long long bb = budget_ns;
    void *args[] = {&dd, &tt, &pp, &bb};
    return launch_cooperative(k, ctas, threads, args, tile_smem(tl), stream);
}

/* Spatial tiles of one network (see NetTile): at most about target_nodes
 * nodes per tile, the tile count a multiple of `ctas`, equal-count cells in
 * strips of the box [0, width) x [miny, maxy] with the box's aspect ratio.
 * Returns NR_OK with the layout in `out` (host arrays), or NR_ERR_CAPACITY
 * when a tile exceeds the 16-bit local encoding. */
int build_tile_layout(const nr_host_network &h, const Incidence &inc, const unsigned char *fcodes, bool use_bonds,
                      bool use_triples, int ctas, int target_nodes, bool quads, TileHost &out) {
    const int n = h.n_points, ne = h.n_edges(), nt = h.n_triples();
    const double W = h.offset, H = std::max(h.maxy - h.miny, 1e-300);
    if (n <= 0 || !(W > 0) || ctas < 1) return NR_ERR_INVALID;
    const long per = (long)ctas * target_nodes;
    const long want = (long)ctas * std::max(1L, (n + per - 1) / per);
    const int ny = (int)std::min(want, std::max(1L, std::lround(std::sqrt((double)want * H / W))));
    /* equal-count cells: ny strips of consecutive y, strip s cut into the
     * cells [want s / ny, want (s + 1) / ny) of consecutive x (periodic x
     * folded into [0, W)), each strip holding nodes in proportion to its
     * cells: exactly `want` cells (a multiple of ctas), each owning n / want
     * nodes however unevenly the nodes are spread (fibre networks), so no
     * tile's record is much larger than the mean and every CTA takes the
     * same number of tiles */
    const long ncells = want;
    std::vector<int> cell(n), count((size_t)ncells, 0), idx(n);
    std::vector<double> xs(n);
    for (int i = 0; i < n; ++i) {
        idx[i] = i;
        xs[i] = h.points[2 * i] - W * std::floor(h.points[2 * i] / W);
    }
    std::sort(idx.begin(), idx.end(), [&](int a, int b) {
        const double ya = h.points[2 * a + 1], yb = h.points[2 * b + 1];
        return ya < yb || (ya == yb && a < b);
    });
    for (int sy = 0; sy < ny; ++sy) {
        const long c0 = ncells * sy / ny, c1 = ncells * (sy + 1) / ny;
        const long lo = (long)n * c0 / ncells, hi = (long)n * c1 / ncells;
        std::sort(idx.begin() + lo, idx.begin() + hi,
                  [&](int a, int b) { return xs[a] < xs[b] || (xs[a] == xs[b] && a < b); });
        for (long k = lo; k < hi; ++k) {
            const long c = c0 + (k - lo) * (c1 - c0) / std::max(1L, hi - lo);
            cell[idx[k]] = (int)c;
            count[c]++;
        }
    }
    std::vector<int> tile_of_cell((size_t)ncells, -1);
    int T = 0;
    for (long c = 0; c < ncells; ++c)
        if (count[c] > 0) tile_of_cell[c] = T++;
    std::vector<std::vector<int>> own(T);
    for (int i = 0; i < n; ++i) own[tile_of_cell[cell[i]]].push_back(i); /* ascending */
    /* within a tile, own nodes by their numbers of triple and bond entries:
     * the lanes of a warp gather (nearly) equally long incidence lists */
    auto entries = [&](int i, bool tri) {
        if (tri) return use_triples ? inc.tptr[i + 1] - inc.tptr[i] : 0;
        return use_bonds ? inc.bptr[i + 1] - inc.bptr[i] : 0;
    };
    for (std::vector<int> &o : own)
        std::stable_sort(o.begin(), o.end(), [&](int a, int b) {
            const int ta = entries(a, true), tb = entries(b, true);
            return ta != tb ? ta > tb : entries(a, false) > entries(b, false);
        });
    out = TileHost();
    out.n_tiles = T;
    /* tile-order positions: each tile's own range starts on a multiple of 16 */
    std::vector<int> pos_of(n), own_pos(T);
    int P = 0;
    for (int t = 0; t < T; ++t) {
        own_pos[t] = P;
        for (size_t k = 0; k < own[t].size(); ++k) pos_of[own[t][k]] = P + (int)k;
        P += (int)((own[t].size() + 15) / 16 * 16);
    }
    out.n_pos = P;
    out.node_of_pos.assign(P, -1);
    for (int i = 0; i < n; ++i) out.node_of_pos[pos_of[i]] = i;
    std::vector<int> loc(n, -1), bslot(use_bonds ? ne : 0, -1), tslot(use_triples ? nt : 0, -1);
    std::vector<int> bl, tlist, halo;
    std::vector<unsigned short> iptr, ibe, incv;
    for (int t = 0; t < T; ++t) {
        const std::vector<int> &o = own[t];
        for (size_t k = 0; k < o.size(); ++k) loc[o[k]] = (int)k;
        bl.clear();
        tlist.clear();
        halo.clear();
        for (int i : o) {
            if (use_bonds)
                for (int e = inc.bptr[i]; e < inc.bptr[i + 1]; ++e) bl.push_back(inc.bent[e] >> 1);
            if (use_triples)
                for (int e = inc.tptr[i]; e < inc.tptr[i + 1]; ++e) tlist.push_back(inc.tent[e] >> 2);
        }
        std::sort(bl.begin(), bl.end());
        bl.erase(std::unique(bl.begin(), bl.end()), bl.end());
        std::sort(tlist.begin(), tlist.end());
        tlist.erase(std::unique(tlist.begin(), tlist.end()), tlist.end());
        auto touch = [&](int v) {
            if (loc[v] == -1) {
                loc[v] = -2; /* halo, numbered below */
                halo.push_back(v);
            }
        };
        for (int b : bl) {
            touch(h.edge_ij[2 * b]);
            touch(h.edge_ij[2 * b + 1]);
        }
        for (int qq : tlist)
            for (int r = 0; r < 3; ++r) touch(h.tri_hjk[3 * qq + r]);
        std::sort(halo.begin(), halo.end());
        for (size_t k = 0; k < halo.size(); ++k) loc[halo[k]] = (int)(o.size() + k);
        auto reset = [&]() {
            for (int v : o) loc[v] = -1;
            for (int v : halo) loc[v] = -1;
            for (int b : bl) bslot[b] = -1;
            for (int qq : tlist) tslot[qq] = -1;
        };
        const size_t nn = o.size() + halo.size();
        if (nn > 0xffff || bl.size() >= 0x4000 || tlist.size() >= 0x2000) {
            reset();
            return NR_ERR_CAPACITY;
        }
        for (size_t k = 0; k < bl.size(); ++k) bslot[bl[k]] = (int)k;
        for (size_t k = 0; k < tlist.size(); ++k) tslot[tlist[k]] = (int)k;
        /* incidence of the own nodes, canonical order: bonds, then triples;
         * an entry is where its result will lie in the record (these
         * segments' offsets do not depend on the incidence) */
        const TileSegs at = tile_segs((int)bl.size(), (int)tlist.size(), (int)o.size(), 0, 0, quads ? 0 : -1);
        iptr.clear();
        ibe.clear();
        incv.clear();
        for (int i : o) {
            iptr.push_back((unsigned short)incv.size());
            if (use_bonds)
                for (int e = inc.bptr[i]; e < inc.bptr[i + 1]; ++e)
                    incv.push_back((unsigned short)(((inc.bent[e] & 1) << 15) | (at.sk / 8 + bslot[inc.bent[e] >> 1])));
            ibe.push_back((unsigned short)incv.size());
            if (use_triples)
                for (int e = inc.tptr[i]; e < inc.tptr[i + 1]; ++e) {
                    const int sl = tslot[inc.tent[e] >> 2], role = inc.tent[e] & 3;
                    incv.push_back((unsigned short)(role == 0 ? 0x8000 | (at.pk / 8 + sl)
                                                              : at.arms / 8 + 2 * sl + (role == 2)));
                }
            if (incv.size() > 0xffff) {
                reset();
                return NR_ERR_CAPACITY;
            }
        }
        iptr.push_back((unsigned short)incv.size());
        TileDesc td;
        td.ro_off = (long long)out.ro.size();
        td.own_pos = own_pos[t];
        td.no = (int)o.size();
        td.nh = (int)halo.size();
        td.nb = (int)bl.size();
        td.nt = (int)tlist.size();
        td.ni = (int)incv.size();
        td.bond_off = (int)out.bid.size();
        td.tri_off = (int)out.tid.size();
        /* entries in quads: as many for each lane of a group of 32 nodes as
         * its longest list takes */
        const int no = td.no, groups = (no + 31) / 32;
        std::vector<unsigned> gq(groups);
        td.nq = quads ? 0 : -1;
        if (quads)
            for (int q = 0; q < groups; ++q) {
                gq[q] = (unsigned)td.nq;
                int most = 0;
                for (int k = 32 * q; k < std::min(no, 32 * q + 32); ++k)
                    most = std::max(most, (iptr[k + 1] - iptr[k] + 3) / 4);
                td.nq += 32 * most;
            }
        const TileSegs g = tile_segs(td);
        out.ro.resize(out.ro.size() + g.total, 0);
        unsigned char *rec = out.ro.data() + td.ro_off;
        for (size_t k = 0; k < bl.size(); ++k) {
            const int b = bl[k];
            const unsigned r = (unsigned)loc[h.edge_ij[2 * b]] | ((unsigned)loc[h.edge_ij[2 * b + 1]] << 16);
            memcpy(rec + g.bref + 4 * k, &r, 4);
            out.bid.push_back(b);
        }
        for (size_t k = 0; k < tlist.size(); ++k) {
            const int qq = tlist[k];
            const uint2 r = make_uint2((unsigned)loc[h.tri_hjk[3 * qq]] | ((unsigned)loc[h.tri_hjk[3 * qq + 1]] << 16),
                                       (unsigned)loc[h.tri_hjk[3 * qq + 2]]);
            memcpy(rec + g.tref + 8 * k, &r, 8);
            out.tid.push_back(qq);
        }
        if (quads) {
            const unsigned short none = (unsigned short)(g.zero / 8);
            unsigned short *q = reinterpret_cast<unsigned short *>(rec + g.inc);
            std::fill(q, q + 4 * (size_t)td.nq, none);
            if (groups) memcpy(rec + g.gq, gq.data(), 4 * gq.size());
            for (int k = 0; k < no; ++k) {
                const unsigned short c[2] = {(unsigned short)(ibe[k] - iptr[k]), (unsigned short)(iptr[k + 1] - iptr[k])};
                memcpy(rec + g.cnt + 4 * k, c, 4);
                for (int e = 0; e < c[1]; ++e)
                    q[4 * (gq[k >> 5] + 32 * (size_t)(e >> 2) + (k & 31)) + (e & 3)] = incv[iptr[k] + e];
            }
        } else {
            memcpy(rec + g.iptr, iptr.data(), 2 * iptr.size());
            if (!ibe.empty()) memcpy(rec + g.ibe, ibe.data(), 2 * ibe.size());
            if (!incv.empty()) memcpy(rec + g.inc, incv.data(), 2 * incv.size());
        }
        for (size_t k = 0; k < o.size(); ++k) rec[g.fcode + k] = fcodes[o[k]];
        for (size_t k = 0; k < halo.size(); ++k) {
            const int pp = pos_of[halo[k]];
            memcpy(rec + g.halo + 4 * k, &pp, 4);
        }
        out.desc.push_back(td);
        out.max_nodes = std::max(out.max_nodes, (int)nn);
        out.max_own = std::max(out.max_own, td.no);
        out.max_bonds = std::max(out.max_bonds, td.nb);
        out.max_tris = std::max(out.max_tris, td.nt);
        out.max_ro = std::max(out.max_ro, g.total);
        out.max_plain = std::max(out.max_plain, tile_segs(td.nb, td.nt, td.no, td.ni, td.nh, -1).total);
        reset();
    }
    out.max_nodes = std::max(out.max_nodes, 1);
    out.max_own = std::max(out.max_own, 1);
    out.max_bonds = std::max(out.max_bonds, 1);
    out.max_tris = std::max(out.max_tris, 1);
    out.max_ro = std::max(out.max_ro, 16u);
    out.max_plain = std::max(out.max_plain, 16u);
    return NR_OK;
}

/* Builds a layout and counts its violations (nr_tile_layout_check). */
static int check_tile_layout(const nr_host_network *h, const Incidence &inc, const std::vector<unsigned char> &fc, int ctas,
                             int target_nodes, bool quads, long long stats[6]) {
    const int n = h->n_points, ne = h->n_edges(), nt = h->n_triples();
    TileHost th;
    const int rc = build_tile_layout(*h, inc, fc.data(), true, true, ctas, target_nodes, quads, th);
    if (rc != NR_OK) return rc;
    long long bad = 0, halo_total = 0;
    std::vector<int> owned(n, 0);
    for (int t = 0; t < th.n_tiles; ++t) {
        const TileDesc &td = th.desc[t];
        const TileSegs g = tile_segs(td);
        if (td.ro_off % 16 || g.total % 16 || td.ro_off + (long long)g.total > (long long)th.ro.size() ||
            g.total > th.max_ro) {
            ++bad;
            continue;
        }
        if (td.own_pos % 16 || td.own_pos + td.no > th.n_pos || td.no + td.nh > th.max_nodes ||
            td.nb > th.max_bonds || td.nt > th.max_tris || td.no > th.max_own)
            ++bad;
        const unsigned char *rec = th.ro.data() + td.ro_off;
        const int nn = td.no + td.nh;
        for (int k = 0; k < td.no; ++k) {
            const int i = th.node_of_pos[td.own_pos + k];
            if (i < 0 || i >= n) {
                ++bad;
                continue;
            }
            owned[i]++;
            if (rec[g.fcode + k] != fc[i]) ++bad;
        }
        for (int k = 0; k < td.nb; ++k) {
            unsigned r;
            memcpy(&r, rec + g.bref + 4 * k, 4);
            if ((int)(r & 0xffffu) >= nn || (int)(r >> 16) >= nn) ++bad;
            const int b = th.bid[td.bond_off + k];
            if (b < 0 || b >= ne) ++bad;
        }
        for (int k = 0; k < td.nt; ++k) {
            unsigned r[2];
            memcpy(r, rec + g.tref + 8 * k, 8);
            if ((int)(r[0] & 0xffffu) >= nn || (int)(r[0] >> 16) >= nn || (int)r[1] >= nn) ++bad;
            const int q = th.tid[td.tri_off + k];
            if (q < 0 || q >= nt) ++bad;
        }
        for (int k = 0; k < td.nh; ++k) {
            int pp;
            memcpy(&pp, rec + g.halo + 4 * k, 4);
            if (pp < 0 || pp >= th.n_pos || th.node_of_pos[pp] < 0) ++bad;
        }
        for (int k = 0; k < td.no; ++k) {
            /* the node's entries: bonds up to b, all up to e (quads: those
             * that fill up, up to full) */
            unsigned short a = 0, b, e;
            unsigned q0 = 0, full = 0;
            if (quads) {
                const int groups = (td.no + 31) / 32;
                unsigned q1 = (unsigned)td.nq;
                memcpy(&q0, rec + g.gq + 4 * (k >> 5), 4);
                if ((k >> 5) + 1 < groups) memcpy(&q1, rec + g.gq + 4 * (k >> 5) + 4, 4);
                if (q0 > q1 || q1 > (unsigned)td.nq || (q1 - q0) % 32) {
                    ++bad;
                    continue;
                }
                full = (q1 - q0) / 32 * 4;
                memcpy(&b, rec + g.cnt + 4 * k, 2);
                memcpy(&e, rec + g.cnt + 4 * k + 2, 2);
                if (e > full) {
                    ++bad;
                    continue;
                }
            } else {
                memcpy(&a, rec + g.iptr + 2 * k, 2);
                memcpy(&e, rec + g.iptr + 2 * k + 2, 2);
                memcpy(&b, rec + g.ibe + 2 * k, 2);
                full = e;
            }
            if (!(a <= b && b <= e && (quads || e <= td.ni))) {
                ++bad;
                continue;
            }
            for (int x = a; x < (int)full; ++x) {
                unsigned short c;
                memcpy(&c, rec + g.inc + 2 * (quads ? 4 * (q0 + 32 * (size_t)(x >> 2) + (k & 31)) + (x & 3) : (size_t)x), 2);
                /* where the entry's result lies: sk, pk (hinges) or arms */
                const unsigned at = c & 0x7fffu, flag = c >> 15;
                const unsigned lo = x >= e ? g.zero / 8 : x < b ? g.sk / 8 : flag ? g.pk / 8 : g.arms / 8;
                const unsigned cnt = x >= e ? 1 : x < b ? td.nb : flag ? td.nt : 2 * td.nt;
                if (g.total > 8u * 0x8000u) continue; /* larger than any shared memory: never launched */
                if (at < lo || at >= lo + cnt || (x >= e && flag)) ++bad;
            }
        }
        halo_total += td.nh;
    }
    for (int i = 0; i < n; ++i)
        if (owned[i] != 1) ++bad;
    stats[0] = th.n_tiles;
    stats[1] = th.n_pos;
    stats[2] = th.max_nodes;
    stats[3] = th.max_plain;
    stats[4] = halo_total;
    stats[5] += bad;
    return NR_OK;
}

}  // namespace nr

extern "C" int nr_tile_layout_check(const nr_host_network *h, int ctas, int target_nodes, long long stats[6]) {
    using namespace nr;
    if (!h || !stats || ctas < 1 || target_nodes < 1) return NR_ERR_INVALID;
    for (int k = 0; k < 6; ++k) stats[k] = 0;
    Incidence inc;
    build_incidence(h->n_points, h->edge_ij.data(), h->n_edges(), h->tri_hjk.data(), h->n_triples(), true, true, inc);
    std::vector<unsigned char> fc(h->n_points);
    nr_host_network_fcodes(h, fc.data());
    const int rc = check_tile_layout(h, inc, fc, ctas, target_nodes, true, stats);
    return rc != NR_OK ? rc : check_tile_layout(h, inc, fc, ctas, target_nodes, false, stats);
}

