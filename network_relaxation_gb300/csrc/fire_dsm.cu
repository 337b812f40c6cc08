/*
 * Mixed-precision FIRE with the per-step state in distributed shared memory.
 *
 * One thread-block cluster of C CTAs relaxes one network at a time (a
 * persistent kernel over the batch's work queue).  Every value a FIRE step
 * writes and reads back lives in the cluster's shared memory:
 *   per node (owner CTA)   u (double-float, float4), FP32 v, FP32 F
 *   per item (owner CTA)   the FP32 force change of the current step
 * A CTA reads another CTA's u (item pass) or item results (gather) with
 * ld.shared::cluster on addresses from mapa, after the hardware cluster
 * barrier that ends the producing pass.  Only read-only data comes from
 * global memory during a step: topology (read-only cache), the anchor
 * records and the anchor force (rewritten only at anchors, by the CTA that
 * reads them).  In the global-memory cluster kernel (fire_mixed.cu) each
 * pass paid dependent L2 round trips; here a step costs three cluster
 * barriers and on-chip latencies.
 *
 * The arithmetic (bond_dforce, tri_dforce, double-float u, the FP32 FIRE
 * step and the FP64 anchors and certification) is mixed_common.cuh's,
 * unchanged.  Layout: NetDsm (nr_device.cuh).  Shared memory per CTA:
 * 32 B per owned node + 8 B per owned bond + 16 B per owned triple; the
 * host uses this kernel when the largest network of the batch fits.
 *
 * What bounds a step (8100 nodes on 4 CTAs, read-only data in global memory;
 * cycles): items 10 100, gather 10 000, pass A 2 200, three cluster barriers
 * with the wait for the slowest CTA 8 000, totals and scalars 4 500.  The gather
 * took 16 200 while it decoded every entry and loaded it from L2 as it went:
 * entries are addresses now, a warp's lie in quads side by side (one
 * conflict-free 16-byte load for four entries; lists behind one another cost
 * eight wavefronts for each 4-byte load), in shared memory where there is room,
 * and the next quad travels while one is added.  192-network batch of 600
 * steps without escalation 47.2 -> 36 ms (phases that may escalate run the
 * earlier kernel, fire_dsm_escalate.cu; this one takes up what yielded there),
 * one network on 4 resident CTAs, us per step: 304 nodes 4.5 -> 3.5, 2491 nodes
 * 7.5 -> 6.0.  Loads from other CTAs (94 clocks a warp against 5 to 9) are
 * hidden: copying the boundary once a step and evaluating its items on both
 * sides was 5 to 10 % slower.
 *
 * Compiled with --fmad=false; FP32 expressions use explicit fmaf().
 */
#include "mixed_common.cuh"
#include "nr_internal.h"

namespace nr {

/* Shared::cluster address of the u of node reference `ref` (sub-block << 16
 * | index in it) when each CTA owns spr = 2^lg sub-blocks of bsub nodes;
 * au[r] = address of CTA r's s_u. */
__device__ __forceinline__ unsigned u_addr(const unsigned *au, int ref, int lg, int bsub) {
    const int sb = (int)((unsigned)ref >> 16), r = sb >> lg;
    const int local = (sb & ((1 << lg) - 1)) * bsub + (ref & 0xffff);
    return au[r] + 16u * (unsigned)local;
}

/* Per-CTA dynamic shared memory: the step's state and, when `resident`,
 * copies of the CTA's read-only slices (item references and anchor
 * records, node pointers and incidence entries, anchor force).  Segments
 * of 16-byte elements first, then 8-byte, then 4-byte ones. */
struct DsmSizes {
    int bmax, emax, tmax;   /* nodes, bonds, triples per CTA */
    int ebmax, etmax;       /* bond / triple incidence entries per CTA */
    int resident;
    int extra; /* bytes behind the entries, for more of them (quads) */
};
struct DsmLayout {
    size_t u, tdf, mb, arms, tref, grec, v, f, bdf, fahi, falo, sk, pk, bref, bent, tent, total;
};
__host__ __device__ inline DsmLayout dsm_layout(const DsmSizes &z) {
    const size_t R = z.resident ? 1 : 0, bm = (size_t)z.bmax, em = (size_t)z.emax, tm = (size_t)z.tmax;
    DsmLayout L;
    size_t o = 0;
    L.u = o;    o += 16 * bm;
    L.tdf = o;  o += 16 * tm;
    L.mb = o;   o += R * 16 * em;
    L.arms = o; o += R * 16 * tm;
    L.tref = o; o += R * 16 * tm;
    L.grec = o; o += R * 16 * bm;
    L.v = o;    o += 8 * bm;
    L.f = o;    o += 8 * bm;
    L.bdf = o;  o += 8 * em;
    L.fahi = o; o += R * 8 * bm;
    L.falo = o; o += R * 8 * bm;
    L.sk = o;   o += R * 8 * em;
    L.pk = o;   o += R * 8 * tm;
    L.bref = o; o += R * 8 * em;
    L.bent = o; o += R * 4 * (size_t)z.ebmax;
    L.tent = o; o += R * 4 * (size_t)z.etmax;
    L.total = o + (size_t)z.extra;
    return L;
}

/* Shared-memory copies the anchor writes besides global memory (null when
 * the CTA is not resident). */
struct DsmRes {
    float4 *mb, *arms;
    float2 *sk, *pk, *fahi, *falo;
};

/* Anchor step 2 for the CTA's own items and nodes: FP32 anchor records by
 * slot, FP64 forces into f, the double-float anchor force, F = F(X) in
 * shared memory; CTA partials of |F|^2 and max|F|^2 in F2, M2. */
static __device__ __noinline__ void anchor_eval_dsm(const NetDev &d, const NetDsm &m, int n0, int nloc, int b0, int b1,
                                                    int t0, int t1, float2 *s_f, DsmRes res, double &F2, double &M2) {
    const double W = d.width;
    F2 = 0.0;
    M2 = 0.0;
    if (d.use_bonds)
        for (int sl = b0 + threadIdx.x; sl < b1; sl += blockDim.x) {
            const int b = __ldg(m.bidx + sl);
            const int4 r = __ldg(d.bond + b);
            const double2 p1 = d.x[r.x], p2 = d.x[r.y];
            const double rx = (p2.x + wrap_shift(r.z, W)) - p1.x, ry = p2.y - p1.y;
            const double k = d.bond_k ? d.bond_k[b] : d.ks;
            const float hx = (float)rx, hy = (float)ry;
            const float4 rec = make_float4(hx, hy, (float)(rx - (double)hx), (float)(ry - (double)hy));
            const float2 sk = make_float2((float)(sqrt_ieee(fma(rx, rx, ry * ry)) - d.bond_l0[b]), (float)k);
            d.mb_data[sl] = rec;
            d.mb_sk[sl] = sk;
            if (res.mb) {
                res.mb[sl - b0] = rec;
                res.sk[sl - b0] = sk;
            }
        }
    if (d.use_triples)
        for (int sl = t0 + threadIdx.x; sl < t1; sl += blockDim.x) {
            const int t = __ldg(m.tref + sl).w;
            const int4 r = __ldg(d.tri + t);
            const double2 ph = d.x[r.x], pj = d.x[r.y], pk = d.x[r.z];
            const int wj = (signed char)(r.w & 0xff), wk = (signed char)((r.w >> 8) & 0xff);
            const double ax = wrap_add(pj.x, wj, W) - ph.x, ay = pj.y - ph.y;
            const double bx = wrap_add(pk.x, wk, W) - ph.x, by = pk.y - ph.y;
            const double kb = d.tri_kb ? d.tri_kb[t] : d.kb;
            const double phi0 = d.tri_phi0 ? d.tri_phi0[t] : 0.0;
            const float4 arms = make_float4((float)ax, (float)ay, (float)bx, (float)by);
            const float2 pkv = make_float2((float)bend_dtheta(ax, ay, bx, by, phi0), (float)kb);
            d.mt_arms[sl] = arms;
            d.mt_pk[sl] = pkv;
            if (res.arms) {
                res.arms[sl - t0] = arms;
                res.pk[sl - t0] = pkv;
            }
        }
    for (int li = threadIdx.x; li < nloc; li += blockDim.x) {
        const int i = n0 + li;
        double fx, fy;
        node_force_fp64_own(d, i, fx, fy);
        d.f[i] = make_double2(fx, fy);
        const float hx = (float)fx, hy = (float)fy;
        const float2 fh = make_float2(hx, hy), fl = make_float2((float)(fx - (double)hx), (float)(fy - (double)hy));
        d.fa_hi[i] = fh;
        d.fa_lo[i] = fl;
        if (res.fahi) {
            res.fahi[li] = fh;
            res.falo[li] = fl;
        }
        s_f[li] = fh;
        const double t = dot2(fx, fy, fx, fy);
        F2 += t;
        M2 = fmax(M2, t);
    }
}

/* Read-only load: through the read-only cache from global memory, or a
 * plain load of a shared-memory copy. */
template <bool RES, class T>
__device__ __forceinline__ T ldro(const T *p) {
    if constexpr (RES) return *p;
    else return __ldg(p);
}

/* Four entries of a node's gather: addresses with flags (see the kernel),
 * their force changes, added in order.  tri_entry's values: dF_j or dF_k
 * (plus an exact 0), or -(dF_j + dF_k). */
struct GatherQuad {
    unsigned c[4];
    float2 a[4], b[4];
    __device__ __forceinline__ void load(uint4 code) {
        c[0] = code.x;
        c[1] = code.y;
        c[2] = code.z;
        c[3] = code.w;
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] = dsm_ld2(c[j] & ~3u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            b[j] = make_float2(0.f, 0.f);
            if (c[j] & 2u) b[j] = dsm_ld2((c[j] & ~3u) + 8u);
        }
    }
    /* The product with the sign is exact. */
    __device__ __forceinline__ void add(float2 &dF, float &mag) const {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float sg = (c[j] & 1u) ? -1.0f : 1.0f;
            dF.x = fmaf(sg, a[j].x + b[j].x, dF.x);
            dF.y = fmaf(sg, a[j].y + b[j].y, dF.y);
            mag += ((fabsf(a[j].x) + fabsf(a[j].y)) + fabsf(b[j].x)) + fabsf(b[j].y);
        }
    }
};

template <int NT, bool RES>
__global__ void __launch_bounds__(NT, 1)
    k_fire_dsm_mixed(const NetDev *nets, const NetDsm *dsms, int n_nets, const int *n_dev, FireParamsDev p,
                     int *queue, const int *order, DsmSizes z) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ float4 s_dyn[];
    unsigned char *dyn = reinterpret_cast<unsigned char *>(s_dyn);
    const DsmLayout L = dsm_layout(z);
    constexpr bool R = RES;
    float4 *s_u = reinterpret_cast<float4 *>(dyn + L.u); /* {hi.x, hi.y, lo.x, lo.y} */
    float4 *s_tdf = reinterpret_cast<float4 *>(dyn + L.tdf);
    float2 *s_v = reinterpret_cast<float2 *>(dyn + L.v);
    float2 *s_f = reinterpret_cast<float2 *>(dyn + L.f);
    float2 *s_bdf = reinterpret_cast<float2 *>(dyn + L.bdf);
    DsmRes res{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    if (R)
        res = DsmRes{reinterpret_cast<float4 *>(dyn + L.mb), reinterpret_cast<float4 *>(dyn + L.arms),
                     reinterpret_cast<float2 *>(dyn + L.sk), reinterpret_cast<float2 *>(dyn + L.pk),
                     reinterpret_cast<float2 *>(dyn + L.fahi), reinterpret_cast<float2 *>(dyn + L.falo)};
    int4 *s_tref = reinterpret_cast<int4 *>(dyn + L.tref);
    int2 *s_bref = reinterpret_cast<int2 *>(dyn + L.bref);
    int4 *s_grec = reinterpret_cast<int4 *>(dyn + L.grec); /* NetDsm.xrec */
    /* the entries' quads, from L.bent on, where they fit */
    uint4 *s_quad = reinterpret_cast<uint4 *>(dyn + (L.bent + 15) / 16 * 16);
    __shared__ MixShared sh;
    __shared__ NetDev s_d;
    __shared__ NetDsm s_m;
    __shared__ int s_slot;
    __shared__ float4 s_zero; /* what padding entries add */
    /* every CTA's step totals, pushed into every CTA of the cluster before
     * the barrier that ends the step: each CTA then reads them from its own
     * shared memory */
    __shared__ float s_parts[kDsmParts][5];
    __shared__ double s_ancs[kDsmParts][2]; /* every CTA's FP64 anchor totals (pushed) */
    __shared__ int s_resume; /* the network yielded in an earlier phase (fire_dsm_escalate.cu) */
    __shared__ unsigned s_au[kDsmParts], s_ab[kDsmParts], s_at[kDsmParts];
    const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
    const int spr = kDsmParts / C, lg = __ffs(spr) - 1; /* sub-blocks per CTA, log2 */
    if (threadIdx.x == 0) s_zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((int)threadIdx.x < C) {
        s_au[threadIdx.x] = dsm_addr(s_u, threadIdx.x);
        s_ab[threadIdx.x] = dsm_addr(s_bdf, threadIdx.x);
        s_at[threadIdx.x] = dsm_addr(s_tdf, threadIdx.x);
    }
    /* n_dev: the count of this launch's networks, written on the device by
     * an earlier kernel (device-side escalation) */
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            const int sl = atomicAdd(queue, 1);
            s_slot = n_dev && sl >= *(volatile const int *)n_dev ? n_nets : sl;
        }
        cl.sync();
        const int slot = *cl.map_shared_rank(&s_slot, 0);
        /* every CTA has read rank 0's slot before any CTA may exit (a CTA's
         * shared memory must not be read remotely after it exits) or rank 0
         * overwrites it for the next network */
        cl.sync();
        if (slot >= n_nets) return;
        if (threadIdx.x == 0) {
            const int idx = order ? order[slot] : slot;
            s_d = nets[idx];
            s_m = dsms[idx];
        }
        __syncthreads();
        const NetDev &d = s_d;
        const NetDsm &m = s_m;
        const int bsub = m.bsub;
        const int n0 = rank * spr * bsub, nloc = max(0, min(spr * bsub, d.n - n0));
        const int b0 = m.bo[rank * spr], b1 = m.bo[(rank + 1) * spr];
        const int t0 = m.to[rank * spr], t1 = m.to[(rank + 1) * spr];
        if (R) /* the CTA's read-only slices into shared memory */
            for (int k = threadIdx.x; k < nloc; k += NT) s_grec[k] = m.xrec[n0 + k];
        /* Node references and incidence entries resolved, once per network
         * and launch, to the shared::cluster addresses of this cluster size:
         * decoding owner, slot and role of every entry took two thirds of the
         * gather's instructions.  References go to the shared copies, or to
         * idle scratch (the force changes of the global-memory kernels: 8 B a
         * bond, 16 B a triple):
         *   bond item    addresses of u_i, u_j
         *   triple item  addresses of u_h, u_j, u_k
         * A node's entries, bonds then triples, lie in the quads of
         * NetDsm.xent (or a shared copy), padded with s_zero:
         *   bond    address of the force change | 1 on the second node
         *   triple  address of {dF_j, dF_k}, for k of its second half, for
         *           the hinge | 3: minus the sum of both halves */
        uint2 *const xb = R ? reinterpret_cast<uint2 *>(s_bref) : reinterpret_cast<uint2 *>(d.bdf) + b0;
        int4 *const xt = R ? s_tref : reinterpret_cast<int4 *>(d.tdf) + t0;
        auto bond_entry = [&](int e) -> unsigned {
            const unsigned code = (unsigned)__ldg(m.bent + e);
            const int r = (int)(code >> 28) >> lg, ls = (int)((code >> 1) & 0x7ffffffu) - m.bo[r * spr];
            return (s_ab[r] + 8u * (unsigned)ls) | (code & 1u);
        };
        auto triple_entry = [&](int e) -> unsigned {
            const unsigned code = (unsigned)__ldg(m.tent + e);
            const int r = (int)(code >> 28) >> lg, ls = (int)((code >> 2) & 0x3ffffffu) - m.to[r * spr];
            const unsigned role = code & 3u;
            return (s_at[r] + 16u * (unsigned)ls + (role == 2u ? 8u : 0u)) | (role == 0u ? 3u : 0u);
        };
        if (d.use_bonds)
            for (int k = threadIdx.x; k < b1 - b0; k += NT) {
                const int2 r = __ldg(m.bref + b0 + k);
                xb[k] = make_uint2(u_addr(s_au, r.x, lg, bsub), u_addr(s_au, r.y, lg, bsub));
            }
        if (d.use_triples)
            for (int k = threadIdx.x; k < t1 - t0; k += NT) {
                const int4 r = __ldg(m.tref + t0 + k);
                xt[k] = make_int4((int)u_addr(s_au, r.x, lg, bsub), (int)u_addr(s_au, r.y, lg, bsub),
                                  (int)u_addr(s_au, r.z, lg, bsub), r.w);
            }
        const unsigned zero_at = dsm_addr(&s_zero, (unsigned)rank);
        /* the CTA's quads: first .. last of its groups of 32 nodes */
        uint4 *quad = m.xent;
        if (nloc > 0) {
            const int4 x0 = __ldg(m.xrec + n0), x1 = __ldg(m.xrec + n0 + nloc - 1);
            if ((size_t)(x1.y + 32 * x1.z - x0.y) * sizeof(uint4) + (size_t)((unsigned char *)s_quad - dyn) <= L.total)
                quad = s_quad - x0.y;
        }
        for (int k = threadIdx.x; k < nloc; k += NT) {
            const int4 g = __ldg(m.grec + n0 + k);
            const int nb = d.use_bonds ? g.z & 0xffff : 0, nt = d.use_triples ? (int)((unsigned)g.z >> 16) : 0;
            const int4 x = __ldg(m.xrec + n0 + k);
            unsigned *const p = reinterpret_cast<unsigned *>(quad + x.y + (k & 31));
            for (int e = 0; e < 4 * x.z; ++e)
                p[128 * (e >> 2) + (e & 3)] =
                    e < nb ? bond_entry(g.y + e) : e < nb + nt ? triple_entry(g.w + e - nb) : zero_at;
        }
        /* item and node data for the step loops: shared copies or global */
        const uint2 *Bref = xb;
        const float4 *Mb = R ? res.mb : d.mb_data + b0;
        const float2 *Sk = R ? res.sk : d.mb_sk + b0;
        const int4 *Tref = xt;
        const float4 *Arms = R ? res.arms : d.mt_arms + t0;
        const float2 *Pk = R ? res.pk : d.mt_pk + t0;
        const int4 *Gr = R ? s_grec : m.xrec + n0;
        const float2 *FaH = R ? res.fahi : d.fa_hi + n0;
        const float2 *FaL = R ? res.falo : d.fa_lo + n0;
        if (threadIdx.x == 0) s_resume = ((volatile FireState *)d.st)->yielded;
        __syncthreads();
        /* the FIRE scalars, advanced by thread 0 of every CTA (identical
         * copies), in shared memory: registers stay free for the passes */
        __shared__ MixScal s_mix;
        __shared__ MixParams s_mq;
        MixScal &s = s_mix;
        MixParams &q = s_mq;
        double F2, M2, tF2, tM2;
        if (s_resume) {
            /* resume a network a smaller cluster left at an anchor: u = 0,
             * v and the FIRE scalars saved, F = F(X) and the anchor records
             * in global memory (slot-indexed: the layout does not depend on
             * the cluster size) */
            for (int li = threadIdx.x; li < nloc; li += NT) {
                s_u[li] = make_float4(0.f, 0.f, 0.f, 0.f);
                s_v[li] = d.vf[n0 + li];
                s_f[li] = d.fa_hi[n0 + li];
            }
            if (R) {
                if (d.use_bonds)
                    for (int k = threadIdx.x; k < b1 - b0; k += NT) {
                        res.mb[k] = d.mb_data[b0 + k];
                        res.sk[k] = d.mb_sk[b0 + k];
                    }
                if (d.use_triples)
                    for (int k = threadIdx.x; k < t1 - t0; k += NT) {
                        res.arms[k] = d.mt_arms[t0 + k];
                        res.pk[k] = d.mt_pk[t0 + k];
                    }
                for (int li = threadIdx.x; li < nloc; li += NT) {
                    res.fahi[li] = d.fa_hi[n0 + li];
                    res.falo[li] = d.fa_lo[n0 + li];
                }
            }
            if (threadIdx.x == 0) {
                s = mix_load(d.st);
                q = mix_params(p, d.sqrt_dof);
                sh.coef = coef_of(s, 0);
            }
            __syncthreads();
        } else {
            for (int li = threadIdx.x; li < nloc; li += NT) {
                s_u[li] = make_float4(0.f, 0.f, 0.f, 0.f);
                s_v[li] = make_float2(0.f, 0.f);
            }
            anchor_eval_dsm(d, m, n0, nloc, b0, b1, t0, t1, s_f, res, F2, M2);
            anchor_reduce(F2, M2, sh.dslots, tF2, tM2);
            if (threadIdx.x == 0) anchor_push(s_ancs, rank, C, tF2, tM2);
            cl.sync();
            if (threadIdx.x == 0) {
                double t[2];
                anchor_totals(s_ancs, C, t);
                q = mix_params(p, d.sqrt_dof);
                mix_init(s, q);
                mix_certify(s, p, d.sqrt_dof, t[0], t[1]);
                sh.coef = coef_of(s, 0);
            }
            __syncthreads();
        }
        for (;;) {
            const Coef c = sh.coef;
            /* pass A: mixing, drift, half kick of the owned nodes */
            for (int li = threadIdx.x; li < nloc; li += NT) {
                float2 v = s_v[li];
                const float2 F = s_f[li];
                if (c.mix_pending) {
                    v.x = fmaf(c.na, v.x, v.x);
                    v.y = fmaf(c.na, v.y, v.y);
                    v.x = fmaf(c.a, F.x, v.x);
                    v.y = fmaf(c.a, F.y, v.y);
                    if (c.zero_v) v = make_float2(0.f, 0.f);
                }
                if (!c.done) {
                    float4 u = s_u[li];
                    df_add(u.x, u.z, fmaf(c.dt, v.x, c.dtsq * F.x));
                    df_add(u.y, u.w, fmaf(c.dt, v.y, c.dtsq * F.y));
                    s_u[li] = u;
                    v.x = fmaf(c.dtm, F.x, v.x);
                    v.y = fmaf(c.dtm, F.y, v.y);
                }
                s_v[li] = v;
            }
            if (c.done) break;
            cl.sync();
            /* item pass: owned bonds and triples, u of any CTA.  Software
             * pipelined: the next item's reference and anchor record (read
             * only, mostly from L2) are loaded while the current one computes */
            if (d.use_bonds) {
                const int nb = b1 - b0;
                int sl = threadIdx.x;
                if (sl < nb) {
                    uint2 r = Bref[sl];
                    float4 ra = Mb[sl];
                    float2 sk = Sk[sl];
                    for (;;) {
                        const float4 ui = dsm_ld4(r.x), uj = dsm_ld4(r.y);
                        const int nx = sl + NT;
                        uint2 rn = r;
                        float4 ran = ra;
                        float2 skn = sk;
                        if (nx < nb) {
                            rn = Bref[nx];
                            ran = Mb[nx];
                            skn = Sk[nx];
                        }
                        float2 dh, dlo;
                        u_diff2(make_float2(uj.x, uj.y), make_float2(uj.z, uj.w), make_float2(ui.x, ui.y),
                                make_float2(ui.z, ui.w), dh, dlo);
                        s_bdf[sl] = bond_dforce(ra, sk, dh, dlo);
                        if (nx >= nb) break;
                        sl = nx;
                        r = rn;
                        ra = ran;
                        sk = skn;
                    }
                }
            }
            if (d.use_triples) {
                const int nt = t1 - t0;
                int sl = threadIdx.x;
                if (sl < nt) {
                    int4 r = Tref[sl];
                    float4 arms = Arms[sl];
                    float2 pk = Pk[sl];
                    for (;;) {
                        const float4 uh = dsm_ld4((unsigned)r.x), uj = dsm_ld4((unsigned)r.y),
                                     uk = dsm_ld4((unsigned)r.z);
                        const int nx = sl + NT;
                        int4 rn = r;
                        float4 armsn = arms;
                        float2 pkn = pk;
                        if (nx < nt) {
                            rn = Tref[nx];
                            armsn = Arms[nx];
                            pkn = Pk[nx];
                        }
                        const float2 hh = make_float2(uh.x, uh.y), hl = make_float2(uh.z, uh.w);
                        float2 dFj, dFk;
                        tri_dforce(arms, pk, u_diff(make_float2(uj.x, uj.y), make_float2(uj.z, uj.w), hh, hl),
                                   u_diff(make_float2(uk.x, uk.y), make_float2(uk.z, uk.w), hh, hl), dFj, dFk);
                        s_tdf[sl] = make_float4(dFj.x, dFj.y, dFk.x, dFk.y);
                        if (nx >= nt) break;
                        sl = nx;
                        r = rn;
                        arms = armsn;
                        pk = pkn;
                    }
                }
            }
            cl.sync();
            /* gather: F = F(X) + the node's entries in incidence order, half
             * kick; the nodes in gather-record order (lanes of a warp take
             * nodes with equally long entry lists) */
            float P = 0.f, V2 = 0.f, Fs = 0.f, M2f = 0.f, A = 0.f;
            for (int k = threadIdx.x; k < nloc; k += NT) {
                /* one record load gives the node, its fcode and its entries */
                const int4 g = ldro<RES>(Gr + k);
                const int li = (g.x & 0x0fffffff) - n0;
                const unsigned fc = (unsigned)g.x >> 28;
                const float2 ah = FaH[li], al = FaL[li];
                float2 F = make_float2(0.f, 0.f);
                float2 dF = make_float2(0.f, 0.f);
                float mag = 0.f;
                /* quads of the whole group, the next one's addresses on their
                 * way while this one is added; padding entries add 0 */
                const uint4 *const p = quad + g.y + (k & 31);
                uint4 code = g.z > 0 ? p[0] : make_uint4(zero_at, zero_at, zero_at, zero_at);
                for (int i = 0; i < g.z; ++i) {
                    const uint4 next = p[32 * min(i + 1, g.z - 1)];
                    GatherQuad q;
                    q.load(code);
                    q.add(dF, mag);
                    code = next;
                }
                if (fc != 0) {
                    A = fmaxf(A, mag);
                    F.x = ah.x + (al.x + dF.x);
                    F.y = ah.y + (al.y + dF.y);
                    if (!(fc & 1)) F.x = 0.f;
                    if (!(fc & 2)) F.y = 0.f;
                }
                float2 v = s_v[li];
                v.x = fmaf(c.dtm, F.x, v.x);
                v.y = fmaf(c.dtm, F.y, v.y);
                s_v[li] = v;
                s_f[li] = F;
                P += fmaf(v.x, F.x, v.y * F.y);
                V2 += fmaf(v.x, v.x, v.y * v.y);
                const float f2 = fmaf(F.x, F.x, F.y * F.y);
                Fs += f2;
                M2f = fmaxf(M2f, f2);
            }
            warp_part(Part{P, V2, Fs, M2f, A}, sh.slots);
            __syncthreads();
            if (threadIdx.x < 32) {
                const Part t = block_totals(sh.slots);
                /* lane r pushes this CTA's totals into CTA r (remote stores
                 * complete before the cluster barrier releases) */
                if ((int)threadIdx.x < C) {
                    const unsigned a = dsm_addr(&s_parts[rank][0], threadIdx.x);
                    dsm_st1(a, t.P);
                    dsm_st1(a + 4u, t.V2);
                    dsm_st1(a + 8u, t.F2);
                    dsm_st1(a + 12u, t.M2);
                    dsm_st1(a + 16u, t.A);
                }
            }
            cl.sync();
            if (threadIdx.x < 32) {
                /* lane r takes rank r's totals: the same butterfly in every CTA */
                Part t{0.f, 0.f, 0.f, 0.f, 0.f};
                if ((int)threadIdx.x < C)
                    t = Part{s_parts[threadIdx.x][0], s_parts[threadIdx.x][1], s_parts[threadIdx.x][2],
                             s_parts[threadIdx.x][3], s_parts[threadIdx.x][4]};
                t = warp_reduce(t);
                if (threadIdx.x == 0) {
                    mix_step(s, q, t);
                    sh.coef = coef_of(s, need_anchor(s, q, t));
                }
            }
            __syncthreads();
            if (sh.coef.anchor) {
                /* X += u (FP64, global), u = 0, then the FP64 anchor */
                for (int li = threadIdx.x; li < nloc; li += NT) {
                    const int i = n0 + li;
                    const float4 u = s_u[li];
                    double2 x = d.x[i];
                    x.x = x.x + ((double)u.x + (double)u.z);
                    x.y = x.y + ((double)u.y + (double)u.w);
                    d.x[i] = x;
                    s_u[li] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                cl.sync();
                anchor_eval_dsm(d, m, n0, nloc, b0, b1, t0, t1, s_f, res, F2, M2);
                anchor_reduce(F2, M2, sh.dslots, tF2, tM2);
                if (threadIdx.x == 0) anchor_push(s_ancs, rank, C, tF2, tM2);
                cl.sync();
                if (threadIdx.x == 0) {
                    double t[2];
                    anchor_totals(s_ancs, C, t);
                    mix_certify(s, p, d.sqrt_dof, t[0], t[1]);
                    sh.coef = coef_of(s, 0);
                }
                __syncthreads();
            }
        }
        for (int li = threadIdx.x; li < nloc; li += NT) {
            const float2 v = s_v[li];
            d.v[n0 + li] = make_double2((double)v.x, (double)v.y);
        }
        cl.sync();
        if (rank == 0) {
            mixed_energies(d, sh.dslots);
            if (threadIdx.x == 0) {
                mix_report(d.st, s);
                d.st->yielded = 0;
            }
        }
        cl.sync();
    }
}

/* Dynamic shared memory of k_fire_dsm_mixed for the given per-CTA maxima. */
size_t dsm_smem_bytes(int bmax, int emax, int tmax, int ebmax, int etmax, int resident) {
    return dsm_layout(DsmSizes{bmax, emax, tmax, ebmax, etmax, resident, 0}).total;
}

constexpr int kDsmStatic = 3024;
/* Largest dynamic shared memory the kernel may use on this device. */
size_t dsm_smem_limit() {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
    /* (at least kDsmStatic of it static: the plans, and with them the order
     * of the sums, do not move with the kernel's static arrays) */
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, (const void *)k_fire_dsm_mixed<512, true>) != cudaSuccess) return 0;
    const int fixed = std::max((int)fa.sharedSizeBytes, kDsmStatic);
    return optin > fixed ? (size_t)(optin - fixed) : 0;
}

/* Shared memory for the entries filled up to quads, up to twice their size
 * (4 bytes each; a resident CTA has the first half by its layout), as far as
 * there is room. */
static int dsm_extra(const DsmSizes &z) {
    const size_t total = dsm_layout(z).total, limit = dsm_smem_limit();
    if (limit <= total) return 0;
    return (int)std::min<size_t>(limit - total, (z.resident ? 4 : 8) * (size_t)(z.ebmax + z.etmax) + 4096);
}

template <int NT, bool RES>
static cudaError_t dsm_config(int cluster, const DsmSizes &z, cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr,
                              int *max_clusters) {
    cudaError_t e;
    int dev, sms;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const size_t smem = dsm_layout(z).total;
    if ((e = allow_dynamic_smem((const void *)k_fire_dsm_mixed<NT, RES>, smem)) != cudaSuccess) return e;
    if (cluster > 8 &&
        (e = cudaFuncSetAttribute(k_fire_dsm_mixed<NT, RES>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) !=
            cudaSuccess)
        return e;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg = cudaLaunchConfig_t{};
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((sms / cluster) * cluster);
    *max_clusters = 0;
    return cudaOccupancyMaxActiveClusters(max_clusters, (void *)k_fire_dsm_mixed<NT, RES>, &cfg);
}

template <int NT, bool RES>
static cudaError_t launch_dsm_nt(const NetDev *nets_dev, const NetDsm *dsm_dev, int n_nets, const int *n_dev,
                                 int cluster, const DsmSizes &z, int cap, const FireParamsDev &p, int *queue_dev,
                                 const int *order_dev, cudaStream_t stream) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    int max_clusters = 0;
    cudaError_t e = dsm_config<NT, RES>(cluster, z, cfg, attr, &max_clusters);
    if (e != cudaSuccess) return e;
    if (max_clusters < 1) return cudaErrorLaunchOutOfResources;
    int clusters = std::max(1, std::min(n_nets, max_clusters));
    if (cap > 0) clusters = std::min(clusters, cap);
    cfg.gridDim = dim3(clusters * cluster);
    cfg.stream = stream;
    if ((e = cudaMemsetAsync(queue_dev, 0, sizeof(int), stream)) != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, k_fire_dsm_mixed<NT, RES>, nets_dev, dsm_dev, n_nets, n_dev, p, queue_dev,
                              order_dev, z);
}

/* Threads per CTA: NR_MIX_THREADS (512 or 1024), else 1024 when the state
 * fills shared memory (many items per thread: more warps hide more
 * latency) and 512 when the CTA is resident (few items per thread: the
 * 128-register budget keeps the step free of spills). */
static int dsm_threads(bool resident) {
    const char *env = knob("NR_MIX_THREADS");
    if (env && (atoi(env) == 512 || atoi(env) == 1024)) return atoi(env);
    return resident ? 512 : 1024;
}

cudaError_t launch_mixed_dsm(const NetDev *nets_dev, const NetDsm *dsm_dev, int n_nets, int cluster, int bmax,
                             int emax, int tmax, int ebmax, int etmax, int resident, double escalate, int cap,
                             const FireParamsDev &p, int *queue_dev, const int *order_dev, cudaStream_t stream,
                             const int *n_dev) {
    if (cluster < 1 || cluster > kDsmParts || (kDsmParts % cluster) != 0) return cudaErrorInvalidValue;
    const bool wide = dsm_threads(resident != 0) == 1024;
    if (escalate > 0) /* when they yield is a matter of timing: fire_dsm_escalate.cu */
        return launch_mixed_dsm_escalate(nets_dev, dsm_dev, n_nets, cluster, bmax, emax, tmax, ebmax, etmax, resident,
                                         wide, escalate, cap, p, queue_dev, order_dev, stream, n_dev);
    DsmSizes z{bmax, emax, tmax, ebmax, etmax, resident, 0};
    z.extra = dsm_extra(z);
    auto launch = resident ? (wide ? launch_dsm_nt<1024, true> : launch_dsm_nt<512, true>)
                           : (wide ? launch_dsm_nt<1024, false> : launch_dsm_nt<512, false>);
    return launch(nets_dev, dsm_dev, n_nets, n_dev, cluster, z, cap, p, queue_dev, order_dev, stream);
}

/* Device-side escalation: the networks of a batch that left their last
 * launch at an anchor (FireState.yielded), in index order, into order_out,
 * and their count into *count_out.  One CTA; a block-wide scan per chunk of
 * blockDim networks. */
__global__ void k_compact_yielded(const FireState *st, int n, int *order_out, int *count_out) {
    __shared__ int s_warp[32];
    __shared__ int s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (int c0 = 0; c0 < n; c0 += blockDim.x) {
        const int i = c0 + threadIdx.x;
        const int flag = i < n && ((volatile const FireState *)st)[i].yielded ? 1 : 0;
        const unsigned bal = __ballot_sync(kFull, flag);
        const int in_warp = __popc(bal & ((1u << lane) - 1u));
        if (lane == 0) s_warp[warp] = __popc(bal);
        __syncthreads();
        int before = s_base;
        for (int w = 0; w < warp; ++w) before += s_warp[w];
        if (flag) order_out[before + in_warp] = i;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 0; w < nw; ++w) s_base += s_warp[w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *count_out = s_base;
}

cudaError_t launch_compact_yielded(const FireState *st, int n, int *order_out, int *count_out, cudaStream_t stream) {
    k_compact_yielded<<<1, 256, 0, stream>>>(st, n, order_out, count_out);
    return cudaGetLastError();
}

cudaError_t dsm_max_active(int cluster, int bmax, int emax, int tmax, int ebmax, int etmax, int resident, int *out) {
    DsmSizes z{bmax, emax, tmax, ebmax, etmax, resident, 0};
    z.extra = dsm_extra(z);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const bool wide = dsm_threads(resident != 0) == 1024;
    if (resident)
        return wide ? dsm_config<1024, true>(cluster, z, cfg, attr, out) : dsm_config<512, true>(cluster, z, cfg, attr, out);
    return wide ? dsm_config<1024, false>(cluster, z, cfg, attr, out) : dsm_config<512, false>(cluster, z, cfg, attr, out);
}

}  // namespace nr
