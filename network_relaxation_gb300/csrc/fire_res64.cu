/*
 * Plain FP64 FIRE (the run_fire_md arithmetic, bit-identical to the oracle)
 * of one network held on chip by the whole GPU, with ONE grid barrier per
 * FIRE step.
 *
 * What bounds an FP64 step.  The FP64 pipe issues 1.7 lanes per clock and SM
 * (a warp instruction every 19 clocks, 64 clocks apart on one scheduler), so
 * a step costs about 110 FP64 slots per node after ieee_int.h took the
 * divisions and roots off that pipe; the cooperative grid kernel
 * (fire_fp64.cu) adds three software grid barriers, a last CTA that reduces
 * and advances the scalars alone while the others wait, and L2 round trips
 * for every position, incidence entry and item force.  Here each CTA keeps a
 * spatial tile of the network in shared memory for the whole relaxation:
 *   - own nodes' x, v, F, the halo's x, every item (bond, triple, gel
 *     element) that touches an own node, its topology, its forces;
 *   - per step only the boundary nodes' {v, F} and the reduction partials
 *     cross CTAs (through L2);
 *   - pass A (mixing, drift, half kick) of the halo is recomputed from the
 *     owner's published v and F with the owner's operations: same bits, no
 *     barrier between drift and forces; items on a tile boundary are
 *     evaluated by each tile they touch (7 % more bonds, 13 % more triples on
 *     32 x 13 node tiles);
 *   - every CTA combines the partials itself, in the canonical order, and
 *     advances its own copy of the FIRE scalars: no second barrier.
 * Tiles are made of whole reduction units (`sub` chunks of 32 consecutive
 * nodes, 256-node tiles of the canonical sum cut in 8 / sub units), so the
 * chunk butterflies stay inside a warp.
 *
 * FP64 work per step and tile: the three sums of a chunk share one butterfly
 * (6 additions for 3 x 5: once xor 16 and 8 have left each sum in fewer
 * lanes, other sums use the free ones), maxima run on the integer pipe, a
 * triple's hinge force is formed once instead of at each of its three
 * entries, and the nodes are gathered in the order of their list lengths, one
 * thread per node and component.
 *
 * Measured per FIRE step (us): 1 024 nodes 22.5 (cluster of 16) -> 8.5; 9 991
 * nodes 40 (grid kernel) -> 10.1; 65 536 nodes 77 -> 22.9; gel of 27 648 nodes
 * 67 -> 25.7.  Of 23 us: items 10.7, passes over nodes and the gather 7.1,
 * barrier and imbalance 1.7, totals and scalars 3.9; the FP64 pipe is active for
 * 17 (62 % of a peak of a warp instruction in 16 clocks, of which FP64
 * instructions reach 84 %).  512 threads: 768 and 1024 measured 3 to 9 % slower;
 * smaller networks: the CTA shapes below.
 *
 * Tiles that do not fit whole (from about 125 000 nodes of a p = 0.65 lattice) are
 * still twice as fast as the grid kernel with their topology, v and F in L2
 * (res64_segs): 160 000 nodes 128 -> 57 us a step, a gel of 90 300 nodes 115 ->
 * 77, and with two forces a triple instead of three in shared memory Mikado of
 * 197 246 nodes 136 -> 77 (numbered by y bands: boundary items add 27 %; the
 * FP64 pipe's share of that tile is 58).  The streamed reads are in order, a
 * warp's line at a time, and hide behind the FP64 work of the other 15 warps.
 *
 * Compiled with --fmad=false: the same bits as the oracle.
 */
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <thread>
#include <type_traits>
#include <vector>

#include "fire_launch.h"
#include "fp64_step.cuh"
#include "nr_internal.h"

namespace nr {

/* Tile sum from its unit partials (tile_from_units with wide loads). */
__device__ __forceinline__ double res_tile_sum(const double *p, int sub) {
    if (sub == 8) return __ldcg(p);
    const double2 *q = reinterpret_cast<const double2 *>(p);
    const double2 a = __ldcg(q);
    if (sub == 4) return a.x + a.y;
    const double2 b = __ldcg(q + 1);
    if (sub == 2) return (a.x + a.y) + (b.x + b.y);
    const double2 c = __ldcg(q + 2), e = __ldcg(q + 3);
    return ((a.x + a.y) + (b.x + b.y)) + ((c.x + c.y) + (e.x + e.y));
}

/* CTA shapes for tiles that are held whole. A large network fills the SMs'
 * FP64 pipes; a step of a small one is a chain of latencies, and networks
 * relaxed from several threads have to share an SM or they run one after the
 * other (each takes 128 of the 152 SMs from 4 096 nodes on).
 *   kResSmall   256 threads, 80 registers, three on an SM: at most 8 groups of
 *               items a tile and 64 tiles in the sums
 *   kResShared  512 threads, 64 registers, two on an SM: fewer than 64 tiles in
 *               the sums (up to 16 128 nodes)
 *   kResAlone   512 threads, one on an SM
 * us per step and network, one thread | 16 threads, against one 512-thread CTA
 * on an SM for all sizes: 1 024 nodes 8.5 | 2.1 -> 8.45 | 1.25, 4 096 8.8 | 8.8
 * -> 8.85 | 4.0, 4 900 9.2 | 9.2 -> 9.3 | 5.7, 9 216 9.8 | 9.7 -> 9.9 | 6.4,
 * 12 544 12.3 | 12.1 -> 12.35 | 7.9; at 16 384, 11.2 | 11.3, one thread would
 * lose 2 %.  (By __maxnreg__: with a minimum of CTAs an SM the compiler goes
 * below the registers it may use, 4 % slower for one thread.) */
enum { kResSmall, kResShared, kResAlone };
constexpr int kResSmallGroups = 8, kResSmallTiles = 64, kResSharedTiles = 63;
__host__ __device__ constexpr int res_threads(int shape) { return shape == kResSmall ? 256 : 512; }

/* One tile of the network per CTA (Res64Desc / Res64Segs, nr_device.cuh).
 * kGel: the network carries a gel; its elements, their reference inverses
 * and the duplicate vertices join the tile.  kMode other than
 * kResWhole: tiles too large to be held whole; topology, v and F are read from
 * L2 in order, and what is reached at random (x, the items' forces) is in
 * shared memory. */
template <int kShape, bool kGel, int kMode>
__global__ void __launch_bounds__(res_threads(kShape))
    __maxnreg__(kShape == kResSmall ? 80 : kShape == kResShared ? 64 : 128)
    k_fire_res64(NetDev d, Res64Dev r, FireParamsDev p, unsigned long long budget_ns) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ Scal s_sc;
    __shared__ double s_tot[24];
    __shared__ unsigned long long s_max[res_threads(kShape) / 32];
    __shared__ unsigned long long s_m2;
    __shared__ int s_ok;
    const Res64Desc td = r.desc[blockIdx.x];
    const Res64Segs g = res64_segs(td, kMode);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr bool kStream = kMode != kResWhole, kPairs = kMode == kResPairs;
    constexpr int NT = res_threads(kShape), NW = NT / 32;
    constexpr int kSplit = kShape == kResSmall ? 2 : 4; /* lane groups whose sums take a warp each */
    const int sub = r.sub, un = kChunk * sub; /* nodes of a unit, a power of two */
    const int lg_un = 31 - __clz(un);
    const int no = td.nu * un;                /* own local indices (the last unit may be padded) */
    /* the tile's record, then the working arrays */
    const unsigned char *const rec = kStream ? r.ro + td.ro_off : s_raw;
    {
        const int4 *src = reinterpret_cast<const int4 *>(r.ro + td.ro_off);
        int4 *dst = reinterpret_cast<int4 *>(s_raw);
        const unsigned bytes = kStream ? tile_pad16(4u * td.nu) : g.rec; /* the unit numbers come first */
        for (unsigned k = tid; k < bytes / 16u; k += NT) dst[k] = __ldg(src + k);
    }
    const int *units = reinterpret_cast<const int *>(s_raw + g.units);
    const int *halo = reinterpret_cast<const int *>(rec + g.halo);
    const double *bl0 = reinterpret_cast<const double *>(rec + g.bl0);
    const double *bk = reinterpret_cast<const double *>(rec + g.bk);
    const unsigned *bref = reinterpret_cast<const unsigned *>(rec + g.bref);
    const signed char *bwrap = reinterpret_cast<const signed char *>(rec + g.bwrap);
    const uint2 *tref = reinterpret_cast<const uint2 *>(rec + g.tref);
    const double *tkb = reinterpret_cast<const double *>(rec + g.tkb);
    const double *tphi = reinterpret_cast<const double *>(rec + g.tphi);
    const uint2 *eref = reinterpret_cast<const uint2 *>(rec + g.eref);
    const int *eid = reinterpret_cast<const int *>(rec + g.eid);
    const uint2 *grec = reinterpret_cast<const uint2 *>(rec + g.grec);
    const unsigned short *inc = reinterpret_cast<const unsigned short *>(rec + g.inc);
    const unsigned short *part = reinterpret_cast<const unsigned short *>(rec + g.partner);
    const unsigned char *pub = rec + g.pub;
    const unsigned short *grp = reinterpret_cast<const unsigned short *>(rec + g.grp);
    double2 *s_x = reinterpret_cast<double2 *>(s_raw + g.x);
    double2 *s_v = reinterpret_cast<double2 *>(s_raw + g.v);
    double2 *s_f = reinterpret_cast<double2 *>(s_raw + g.f);   /* own force sums (gel: before the partner's) */
    double2 *s_ff = kGel ? reinterpret_cast<double2 *>(s_raw + g.ff) : s_f; /* forces */
    double2 *s_bf = reinterpret_cast<double2 *>(s_raw + g.bf);
    double2 *s_tf = reinterpret_cast<double2 *>(s_raw + g.tf); /* per triple: hinge, j, k */
    double *s_M = reinterpret_cast<double *>(s_raw + g.eM);    /* per element: 6 inverse entries, area, - */
    double *s_du = reinterpret_cast<double *>(s_raw + g.du);   /* per element: dU/dF11, F12, F21, F22 */
    __syncthreads();
    auto node_of = [&](int li) { return (units[li >> lg_un] << lg_un) + (li & (un - 1)); };
    for (int li = tid; li < no; li += NT) {
        const int i = node_of(li);
        s_x[li] = i < d.n ? d.x[i] : make_double2(0.0, 0.0);
        if (!kStream) {
            s_v[li] = make_double2(0.0, 0.0);
            s_ff[li] = make_double2(0.0, 0.0);
        }
    }
    for (int h = tid; h < td.nh; h += NT) s_x[no + h] = d.x[halo[h]];
    const int nel = kGel ? td.nel : 0;
    if (kGel && !kStream)
        for (int e = tid; e < nel; e += NT) {
            const double *M = d.gel->elem_inv + 6 * (size_t)eid[e];
            for (int c = 0; c < 6; ++c) s_M[8 * e + c] = M[c];
            s_M[8 * e + 6] = d.gel->elem_area[eid[e]];
        }
    const double W = d.width;
    const int nb = d.use_bonds ? td.nb : 0, nt = d.use_triples ? td.nt : 0;
    const int ngrp = (int)res64_groups(td);
    const int n_units = r.n_units, upt = 8 / sub;
    const int ng = min(8, (d.n_tiles + 31) / 32); /* lane groups of the canonical sum that hold a tile */
    unsigned long long epoch = 0;
    int par = 0;
    bool init = true;
    /* v and F of the thread's first halo node, loaded while the totals and
     * the scalars are computed */
    double2 hv = make_double2(0.0, 0.0), hf = hv;
    for (;;) {
        if (!init) {
            const Scal &s = s_sc;
            if (s.done) break;
            for (int li = tid; li < no; li += NT) {
                const int i = kStream ? node_of(li) : 0;
                if (kStream && i >= d.n) continue;
                double2 *const pv = kStream ? d.v + i : s_v + li;
                double2 x = s_x[li], v = *pv;
                const double2 f = kStream ? d.f[i] : s_ff[li];
                res_mix(s, v, f);
                res_drift(s, x, v, f);
                s_x[li] = x;
                v.x = fma(s.dtm, f.x, v.x);
                v.y = fma(s.dtm, f.y, v.y);
                *pv = v;
            }
            for (int h = tid; h < td.nh; h += NT) {
                if (h != tid) {
                    const double2 *q = r.vf[par ^ 1] + 2 * (size_t)halo[h];
                    hv = __ldcg(q);
                    hf = __ldcg(q + 1);
                }
                double2 x = s_x[no + h];
                res_mix(s, hv, hf);
                res_drift(s, x, hv, hf);
                s_x[no + h] = x;
            }
        }
        __syncthreads();
        /* items, 32 to a warp */
        for (int w = warp; w < ngrp; w += NW) {
            const int code = grp[w], kind = code >> 14, item = 32 * (code & 0x3fff) + lane;
            if (kGel && kind == 2) {
                const int e = item;
                if (e < nel) {
                    const uint2 q = eref[e];
                    const double2 p1 = s_x[q.x & 0xffffu], p2 = s_x[q.x >> 16], p3 = s_x[q.y];
                    const double *M = kStream ? d.gel->elem_inv + 6 * (size_t)eid[e] : s_M + 8 * e;
                    const double area = kStream ? d.gel->elem_area[eid[e]] : M[6];
                    const double f11 = p1.x * M[0] + p2.x * M[2] + p3.x * M[4];
                    const double f12 = p1.x * M[1] + p2.x * M[3] + p3.x * M[5];
                    const double f21 = p1.y * M[0] + p2.y * M[2] + p3.y * M[4];
                    const double f22 = p1.y * M[1] + p2.y * M[3] + p3.y * M[5];
                    double *du = s_du + 4 * e;
                    gel_du_of(*d.gel, area, f11, f12, f21, f22, du[0], du[1], du[2], du[3]);
                }
            } else if (kind == 1) {
                const int t = item;
                if (t < nt) {
                    const uint2 q = tref[t];
                    const double2 ph = s_x[q.x & 0xffffu], pj = s_x[q.x >> 16], pk = s_x[q.y & 0xffffu];
                    const int wj = (signed char)(q.y >> 16), wk = (signed char)(q.y >> 24);
                    const double ax = wrap_add(pj.x, wj, W) - ph.x, ay = pj.y - ph.y;
                    const double bx = wrap_add(pk.x, wk, W) - ph.x, by = pk.y - ph.y;
                    double fjx, fjy, fkx, fky;
                    bend_force(ax, ay, bx, by, td.has_kb ? tkb[t] : d.kb, td.has_phi ? tphi[t] : 0.0, fjx, fjy, fkx,
                               fky);
                    if (kPairs) {
                        s_tf[2 * t] = make_double2(fjx, fjy);
                        s_tf[2 * t + 1] = make_double2(fkx, fky);
                    } else {
                        /* the hinge's (-F_j) - F_k */
                        s_tf[3 * t] = make_double2(ii_flip(fjx, true) - fkx, ii_flip(fjy, true) - fky);
                        s_tf[3 * t + 1] = make_double2(fjx, fjy);
                        s_tf[3 * t + 2] = make_double2(fkx, fky);
                    }
                }
            } else if (kind == 0) {
                const int b = item;
                if (b < nb) {
                    const unsigned q = bref[b];
                    const double2 p1 = s_x[q & 0xffffu], p2 = s_x[q >> 16];
                    double fx, fy;
                    bond_force(p1.x, p1.y, p2.x, p2.y, wrap_shift(bwrap[b], W), bl0[b], td.has_k ? bk[b] : d.ks, fx,
                               fy);
                    s_bf[b] = make_double2(fx, fy);
                }
            }
        }
        __syncthreads();
        /* gather in canonical order, one thread per node and component, two
         * entries in flight (four take registers: 65 536 nodes 23.1 us a step
         * against 22.9, 9 216 nodes 9.95 against 9.88) */
        {
            const double *bfd = reinterpret_cast<const double *>(s_bf);
            const double *tfd = reinterpret_cast<const double *>(s_tf);
            double *fd = reinterpret_cast<double *>(kStream && !kGel ? d.f : s_f);
            for (int k = tid; k < 2 * td.ngather; k += NT) {
                const uint2 q = grec[k >> 1];
                const int c = k & 1;
                const unsigned short *e = inc + (q.y & 0xffffu);
                double f = 0.0;
                if ((q.y >> (24 + c)) & 1u) {
                    if (d.use_bonds) {
                        const int m = (int)((q.x >> 16) & 0xffu);
#pragma unroll 2
                        for (int a = 0; a < m; ++a) {
                            const unsigned code = e[a];
                            f = f + ii_flip(bfd[(code & ~1u) + c], (code & 1u) != 0);
                        }
                        e += m;
                    }
                    if (d.use_triples) {
                        const int m = (int)(q.x >> 24);
#pragma unroll 2
                        for (int a = 0; a < m; ++a) {
                            if (kPairs) {
                                const unsigned code = e[a], t = code / 3u, role = code - 3u * t;
                                const double u = tfd[4 * t + (role == 2u ? 2u : 0u) + c];
                                f = f + (role == 0u ? ii_flip(u, true) - tfd[4 * t + 2u + c] : u);
                            } else {
                                f = f + tfd[2 * e[a] + c];
                            }
                        }
                        e += m;
                    }
                    if (kGel) {
                        const int m = (int)((q.y >> 16) & 0xffu);
                        for (int a = 0; a < m; ++a) {
                            const int el = e[a] / 3, v = e[a] - 3 * el;
                            const double *M =
                                (kStream ? d.gel->elem_inv + 6 * (size_t)eid[el] : s_M + 8 * el) + 2 * v;
                            f = f + s_du[4 * el + 2 * c] * M[0];
                            f = f + s_du[4 * el + 2 * c + 1] * M[1];
                        }
                    }
                }
                const int li = (int)(q.x & 0xffffu);
                if (!kStream || kGel) fd[2 * li + c] = f;
                else if (li < no) fd[2 * (size_t)node_of(li) + c] = f; /* a gel that is not set: no use for other tiles' duplicates */
            }
        }
        __syncthreads();
        /* half kick, publication, the chunks' partial sums in node order */
        const double dtm = init ? 0.0 : s_sc.dtm;
        unsigned long long mx = 0ULL;
        double2 *vf = r.vf[par];
        double *pt = r.part[par];
        for (int u = warp; u < td.nu; u += NW) {
            const int unit = units[u];
            double acc = 0.0, acc2 = 0.0, acc4 = 0.0;
            for (int c = 0; c < sub; ++c) {
                const int li = u * un + c * kChunk + lane, i = unit * un + c * kChunk + lane;
                double tP = 0.0, tV = 0.0, tF = 0.0;
                if (i < d.n) {
                    double2 f = kStream && !kGel ? d.f[i] : s_f[li];
                    if (kGel) {
                        const unsigned q = part[li];
                        if (q != 0xffffu) {
                            const double2 o = s_f[q];
                            f.x = f.x + o.x;
                            f.y = f.y + o.y;
                        }
                        if (kStream) d.f[i] = f;
                        else s_ff[li] = f;
                    }
                    double2 v = make_double2(0.0, 0.0);
                    if (!init) {
                        v = kStream ? d.v[i] : s_v[li];
                        v.x = fma(dtm, f.x, v.x);
                        v.y = fma(dtm, f.y, v.y);
                    }
                    if (kStream) d.v[i] = v;
                    else if (!init) s_v[li] = v;
                    if (pub[li]) {
                        vf[2 * (size_t)i] = v;
                        vf[2 * (size_t)i + 1] = f;
                    }
                    tP = dot2(v.x, v.y, f.x, f.y);
                    tV = dot2(v.x, v.y, v.x, v.y);
                    tF = dot2(f.x, f.y, f.x, f.y);
                }
                mx = max(mx, max_bits(tF));
                const double cs = warp_sum3(tP, tV, tF, lane);
                /* the lower levels of tree8 over the unit's chunks */
                if (sub == 1) {
                    acc4 = cs;
                } else if ((c & 1) == 0) {
                    acc = cs;
                } else {
                    const double p2 = acc + cs;
                    if (sub == 2) acc4 = p2;
                    else if ((c & 2) == 0) acc2 = p2;
                    else {
                        const double p4 = acc2 + p2;
                        if (sub == 4) acc4 = p4;
                        else if ((c & 4) == 0) acc4 = p4;
                        else acc4 = acc4 + p4;
                    }
                }
            }
            if ((lane & 7) == 0 && lane != 24) pt[(size_t)(lane == 0 ? 0 : lane == 16 ? 1 : 2) * n_units + unit] = acc4;
        }
        mx = warp_max_bits(mx);
        if (lane == 0) s_max[warp] = mx;
        __syncthreads();
        if (warp == 0) {
            const unsigned long long m = warp_max_bits(lane < NW ? s_max[lane] : 0ULL);
            if (lane == 0) r.maxp[par][blockIdx.x] = m;
        }
        ++epoch;
        if (!epoch_barrier(r.bar, d.st, epoch * (unsigned long long)gridDim.x, budget_ns, 31, &s_ok)) return;
        if (tid < td.nh) {
            const double2 *q = vf + 2 * (size_t)halo[tid];
            hv = __ldcg(q);
            hf = __ldcg(q + 1);
        }
        /* the canonical totals.  Up to kSplit lane groups: a warp each for
         * every sum (the shortest chain); more (not kResSmall): warp k sums the
         * tiles of lane group k for all three (the fewest FP64 slots) */
        if (kShape == kResSmall || ng <= kSplit) {
            if (warp < 3 * ng) {
                const int q = warp / ng, grp = warp - q * ng, t = 32 * grp + lane;
                double a = t < d.n_tiles ? res_tile_sum(pt + (size_t)q * n_units + (size_t)t * upt, sub) : 0.0;
                a = warp_sum(a);
                if (lane == 0) s_tot[8 * q + grp] = a;
            } else if (warp == 3 * kSplit) {
                if (lane < 24 && (lane & 7) >= ng) s_tot[lane] = 0.0;
            } else if (warp == 3 * kSplit + 1) {
                unsigned long long m = 0ULL;
                for (unsigned b = lane; b < gridDim.x; b += 32) m = max(m, __ldcg(r.maxp[par] + b));
                m = warp_max_bits(m);
                if (lane == 0) s_m2 = m;
            }
        } else if (warp < ng) {
            const int k = 32 * warp + lane;
            double a[3] = {0.0, 0.0, 0.0};
            if (k < d.n_tiles) {
#pragma unroll
                for (int q = 0; q < 3; ++q) a[q] = res_tile_sum(pt + (size_t)q * n_units + (size_t)k * upt, sub);
                for (int t = k + kTile; t < d.n_tiles; t += kTile)
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        a[q] = a[q] + res_tile_sum(pt + (size_t)q * n_units + (size_t)t * upt, sub);
            }
            const double c = warp_sum3(a[0], a[1], a[2], lane);
            if ((lane & 7) == 0 && lane != 24) s_tot[8 * (lane == 0 ? 0 : lane == 16 ? 1 : 2) + warp] = c;
        } else if (warp < 8) {
            if (lane < 3) s_tot[8 * lane + warp] = 0.0;
        } else if (warp == 8) {
            unsigned long long m = 0ULL;
            for (unsigned b = lane; b < gridDim.x; b += 32) m = max(m, __ldcg(r.maxp[par] + b));
            m = warp_max_bits(m);
            if (lane == 0) s_m2 = m;
        }
        __syncthreads();
        if (warp == 0) scal_warp(s_sc, p, s_tot, ng, s_m2, d.sqrt_dof, init);
        __syncthreads();
        init = false;
        par ^= 1;
    }
    /* the last pass A only mixes v */
    for (int li = tid; li < no; li += NT) {
        const int i = node_of(li);
        if (i >= d.n) continue;
        double2 v = kStream ? d.v[i] : s_v[li];
        const double2 f = kStream ? d.f[i] : s_ff[li];
        res_mix(s_sc, v, f);
        d.x[i] = s_x[li];
        d.v[i] = v;
        if (!kStream) d.f[i] = f;
    }
    if (blockIdx.x == 0 && tid == 0) scal_store(d.st, s_sc);
}

template <int kShape, int kMode>
static const void *res_kernel_of(bool gel) {
    return gel ? (const void *)k_fire_res64<kShape, true, kMode> : (const void *)k_fire_res64<kShape, false, kMode>;
}
static const void *res_kernel(int shape, bool gel, int mode) {
    if (mode == kResPairs) return res_kernel_of<kResAlone, kResPairs>(gel);
    if (mode == kResStream) return res_kernel_of<kResAlone, kResStream>(gel);
    if (shape == kResSmall) return res_kernel_of<kResSmall, kResWhole>(gel);
    if (shape == kResShared) return res_kernel_of<kResShared, kResWhole>(gel);
    return res_kernel_of<kResAlone, kResWhole>(gel);
}

/* Largest dynamic shared memory of the kernel on this device (NR_RES64_SMEM:
 * bytes to stay below). */
size_t res64_smem_limit() {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, res_kernel(kResAlone, true, kResStream)) != cudaSuccess) return 0;
    const size_t most = optin > (int)fa.sharedSizeBytes ? (size_t)(optin - (int)fa.sharedSizeBytes) : 0;
    const char *env = getenv("NR_RES64_SMEM");
    return env ? std::min(most, (size_t)std::max(0, atoi(env))) : most;
}

/* Whether `ctas` CTAs of the kernel are co-resident. */
bool res64_fits(int ctas, int shape, bool gel, int mode, size_t smem) {
    int dev = 0, sms = 0, per_sm = 0;
    const void *k = res_kernel(shape, gel, mode);
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        allow_dynamic_smem(k, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, res_threads(shape), smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return ctas <= per_sm * sms;
}

cudaError_t launch_fp64_res(const NetDev &d, const Res64Dev &r, const FireParamsDev &p, size_t smem,
                            unsigned long long budget_ns, cudaStream_t stream) {
    const void *k = res_kernel(r.shape, d.use_gel != 0, r.mode);
    cudaError_t e = allow_dynamic_smem(k, smem);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(r.bar, 0, sizeof(unsigned long long), stream)) != cudaSuccess) return e;
    NetDev dd = d;
    Res64Dev rr = r;
    FireParamsDev pp = p;
    unsigned long long bb = budget_ns;
    void *args[] = {&dd, &rr, &pp, &bb};
    return launch_cooperative(k, r.n_ctas, res_threads(r.shape), args, smem, stream);
}

/* ------------------------------------------------------------------ */
/* Host side: the layout                                                */
/* ------------------------------------------------------------------ */

namespace {

/* Runs f(k, scratch) for k < n, on a few host threads when `items` items of
 * work repay their start; every thread has its own Scratch. */
template <class Scratch, class F>
void parallel_for(int n, long items, F f) {
    const int nt = std::max(1, std::min({n, (int)std::thread::hardware_concurrency(), 16, (int)(items / 3000)}));
    std::atomic<int> next{0};
    run_threads(nt, [&](int) {
        Scratch s;
        for (int k; (k = next.fetch_add(1)) < n;) f(k, s);
    });
}

struct NoScratch {};
/* Halo index of every node in the tile at hand (-1). */
struct TileScratch {
    std::vector<int> loc;
};

/* The items of every tile in index order (item[off[t] .. off[t + 1])) and the
 * slot of each in the tile of each of its k nodes (slot[k q + r]). */
struct TileItems {
    std::vector<int> off, item, slot;
};

}  // namespace

/* Tiles of whole reduction units (Res64Host).  A network of no more chunks than
 * there are CTAs gets a chunk a tile.  Else units are dealt to tiles in strips
 * of y and columns of x; of several unit sizes and column counts the one whose
 * largest tile takes the fewest FP64 slots is taken: row-ordered lattices get
 * blocks (256 x 256: 152 tiles of 32 x 13 or 14 nodes that evaluate 12 % more
 * items than the network has), networks numbered by y bands.  NR_ERR_CAPACITY
 * when a tile exceeds the 16-bit local encoding or smem_limit, or when boundary
 * items make the largest tile's work more than 2.5 times an even share (the
 * numbering then has no locality, and the kernels that evaluate every item once
 * are faster). May throw.
 *
 * Every network's creation pays for it, so the tiles' item lists come from one
 * walk over the items in index order, without sorting and without a search for
 * slots, and the records go to the image tile by tile.  Creating a network (us,
 * without a layout | with): 1 024 nodes 183 | 420, 2 500 333 | 810, 10 000
 * 1 309 | 3 030 (600, 1 350 and 3 400 when each tile gathered, sorted and
 * numbered its items itself).  A host thread takes 25 to 40 us to start there:
 * fewer than 3 000 items do not repay it. */
static int build_layout(const nr_host_network &h, const Incidence &inc, const unsigned char *fcodes, bool use_bonds,
                        bool use_triples, const std::vector<int> &eptr, const std::vector<int> &eent,
                        const std::vector<int> &partner, int max_ctas, size_t smem_limit, Res64Host &out) {
    const int n = h.n_points, ne = use_bonds ? h.n_edges() : 0, nt = use_triples ? h.n_triples() : 0;
    const int nel = h.n_facets();
    if (n <= 0 || max_ctas < 1) return NR_ERR_INVALID;
    /* duplicate vertices without elements: the other kernels */
    if (nel == 0 && h.n_mesh_pairs() > 0) return NR_ERR_CAPACITY;
    /* shared memory at the least: x, the bonds' and triples' forces */
    if (16.0 * n + 16.0 * ne + 32.0 * nt + 32.0 * nel > (double)max_ctas * smem_limit) return NR_ERR_CAPACITY;
    /* candidates: units of `sub` chunks dealt to S strips of y, each cut in
     * c columns of x.  Cuts move by up to a tenth of a strip (column) to the
     * widest gap nearby, so that strips end between rows and columns between
     * the chunks of a row. */
    struct Cand {
        int sub, c, T;
        std::vector<int> tile; /* of every unit */
        double cost;
    };
    auto snap = [](auto at, int target, int win, int lo, int hi) {
        int best = target;
        double gap = -1.0;
        for (int k = 0; k <= 2 * win; ++k) {
            const int i = target + (k & 1 ? (k + 1) / 2 : -(k / 2));
            if (i <= lo || i >= hi) continue;
            const double g = at(i) - at(i - 1);
            if (g > 1.5 * gap + 1e-12) {
                gap = g;
                best = i;
            }
        }
        return std::min(std::max(best, lo), hi);
    };
    const double W = std::max(h.offset, 1e-300), H = std::max(h.maxy - h.miny, 1e-300);
    auto units_of = [&](int sub) { return (n + kChunk * sub - 1) / (kChunk * sub); };
    auto deal = [&](Cand &q, const std::vector<double> &ux, const std::vector<double> &uy, const std::vector<int> &by_y) {
        const int U = (int)by_y.size(), S = std::max(1, std::min(U, max_ctas / q.c));
        std::vector<int> idx(by_y);
        q.tile.assign(U, 0);
        q.T = 0;
        for (int st = 0, lo = 0; st < S; ++st) {
            const int hi = st == S - 1 ? U
                                       : snap([&](int i) { return uy[idx[i]]; }, (int)((long)U * (st + 1) / S),
                                              std::max(1, U / S / 10), lo, U);
            if (q.c > 1)
                std::stable_sort(idx.begin() + lo, idx.begin() + hi, [&](int a, int b) { return ux[a] < ux[b]; });
            const int m = hi - lo;
            for (int k = 0, l = 0; k < q.c; ++k) {
                const int r = k == q.c - 1 ? m
                                           : snap([&](int i) { return ux[idx[lo + i]]; }, (int)((long)m * (k + 1) / q.c),
                                                  std::max(1, m / q.c / 10), l, m);
                if (r > l) {
                    for (int i = l; i < r; ++i) q.tile[idx[lo + i]] = q.T;
                    q.T++;
                }
                l = r;
            }
            lo = hi;
        }
    };
    /* FP64 slots of the largest tile's step (per warp of items: bonds 8,
     * triples 33, elements 45; nodes 45 a chunk; 12 for the halo, about a node
     * a cut bond) and of the totals that every CTA takes from the unit
     * partials */
    auto cost = [&](Cand &q) {
        const int sh = __builtin_ctz((unsigned)(kChunk * q.sub)); /* a power of two */
        std::vector<int> nb(q.T, 0), nt3(q.T, 0), ne3(q.T, 0), nu(q.T, 0), cut(q.T, 0);
        auto of = [&](int i) { return q.tile[i >> sh]; };
        for (int b = 0; b < ne; ++b) {
            const int x = of(h.edge_ij[2 * b]), y = of(h.edge_ij[2 * b + 1]);
            nb[x]++;
            if (y != x) {
                nb[y]++;
                cut[x]++;
                cut[y]++;
            }
        }
        auto three = [&](const int *v, std::vector<int> &cnt) {
            const int x = of(v[0]), y = of(v[1]), z = of(v[2]);
            cnt[x]++;
            if (y != x) cnt[y]++;
            if (z != x && z != y) cnt[z]++;
        };
        for (int t = 0; t < nt; ++t) three(&h.tri_hjk[3 * t], nt3);
        for (int e = 0; e < nel; ++e) three(&h.facets[3 * e], ne3);
        for (int t : q.tile) nu[t]++;
        double worst = 0.0;
        for (int t = 0; t < q.T; ++t)
            worst = std::max(worst, 8 * std::ceil(nb[t] / 32.0) + 33 * std::ceil(nt3[t] / 32.0) +
                                        45 * std::ceil(ne3[t] / 32.0) + 45.0 * nu[t] * q.sub + 12 * std::ceil(cut[t] / 32.0));
        q.cost = worst + 3.0 * (8 / q.sub - 1) * ((n + kTile - 1) / kTile) / 32.0;
    };
    const long items = (long)ne + nt + nel;
    std::vector<Cand> cand;
    std::vector<std::vector<double>> uxs(9), uys(9);
    std::vector<std::vector<int>> order(9);
    const char *env = getenv("NR_RES64_SUB"); /* units of so many chunks alone (tests) */
    const int only = env ? atoi(env) : 0;
    if (units_of(1) <= max_ctas && !only) { /* a chunk a tile: nothing to choose */
        cand.push_back(Cand{1, 1, units_of(1), std::vector<int>(units_of(1)), 0.0});
        std::iota(cand[0].tile.begin(), cand[0].tile.end(), 0);
        cost(cand[0]);
    } else {
        for (int sub : {1, 2, 4, 8}) {
            const int U = units_of(sub), un = kChunk * sub;
            if (only && sub != only) continue;
            if (!only && sub > 1 && (U < max_ctas || n < 16 * kTile)) break; /* fewer partials only matter when there are many */
            std::vector<double> &ux = uxs[sub], &uy = uys[sub];
            ux.assign(U, 0.0);
            uy.assign(U, 0.0);
            for (int u = 0; u < U; ++u) {
                /* x from the unit's first node on, the shorter way around the
                 * period: a unit that runs over a row's end lies at the seam
                 * (taken in the middle of the row it tore tiles apart: 181 x
                 * 181 nodes 77 % more items than the network has instead of
                 * 42, 19.2 us a step instead of 17.4) */
                const int i0 = u * un, i1 = std::min(n, i0 + un);
                const double x0 = h.points[2 * i0];
                for (int i = i0; i < i1; ++i) {
                    const double dx = h.points[2 * i] - x0;
                    ux[u] += std::fabs(dx) < 0.499 * W ? dx : dx - W * std::round(dx / W);
                    uy[u] += h.points[2 * i + 1];
                }
                ux[u] = x0 + ux[u] / (i1 - i0);
                ux[u] -= W * std::floor(ux[u] / W);
                uy[u] /= i1 - i0;
            }
            std::vector<int> &o = order[sub];
            o.resize(U);
            for (int u = 0; u < U; ++u) o[u] = u;
            std::stable_sort(o.begin(), o.end(), [&](int a, int b) { return uy[a] < uy[b]; });
            /* columns: bands (c = 1), and around square tiles */
            const int G = std::min(U, max_ctas), sq = std::max(1, (int)std::lround(std::sqrt(G * W / H)));
            std::vector<int> cs{1};
            for (int c : {sq / 3, sq / 2, 2 * sq / 3, 3 * sq / 4, sq}) cs.push_back(std::max(1, std::min(G, c)));
            std::sort(cs.begin(), cs.end());
            cs.erase(std::unique(cs.begin(), cs.end()), cs.end());
            for (int c : cs) cand.push_back(Cand{sub, c, 0, {}, 1e300});
        }
        parallel_for<NoScratch>((int)cand.size(), items, [&](int k, NoScratch &) {
            deal(cand[k], uxs[cand[k].sub], uys[cand[k].sub], order[cand[k].sub]);
            cost(cand[k]);
        });
    }
    if (cand.empty()) return NR_ERR_INVALID;
    const Cand &best = *std::min_element(cand.begin(), cand.end(),
                                         [](const Cand &a, const Cand &b) { return a.cost < b.cost; });
    const int sub = best.sub, un = kChunk * sub, U = units_of(sub), T = best.T;
    const std::vector<int> &tile = best.tile;
    out = Res64Host();
    out.sub = sub;
    out.n_ctas = T;
    out.n_units = (n + kTile - 1) / kTile * (8 / sub);
    /* every item once, shared by all SMs, against the largest tile (small
     * networks are bound by latency and may do more) */
    if (best.cost > 2.5 * (8.0 * ne + 33.0 * nt + 45.0 * nel + 45.0 * n) / 32.0 / max_ctas + 2000.0)
        return NR_ERR_CAPACITY;
    const int lg_un = __builtin_ctz((unsigned)un); /* a power of two */
    std::vector<std::vector<int>> tu(T);
    std::vector<int> uslot(U);
    for (int u = 0; u < U; ++u) {
        uslot[u] = (int)tu[tile[u]].size();
        tu[tile[u]].push_back(u);
    }
    auto tile_of = [&](int i) { return tile[i >> lg_un]; };
    /* the tile besides its own that gathers a node, its duplicate's (-1) */
    std::vector<int> other;
    if (nel > 0) {
        other.assign(n, -1);
        for (int i = 0; i < n; ++i)
            if (partner[i] >= 0 && tile_of(partner[i]) != tile_of(i)) other[i] = tile_of(partner[i]);
    }
    /* the items that touch a node gathered by a tile: bonds, triples, elements */
    TileItems its[3];
    auto list = [&](auto nodes, int count, const int *v, TileItems &L) {
        constexpr int k = decltype(nodes)::value;
        L.off.assign(T + 1, 0);
        L.slot.resize((size_t)k * count);
        /* f(tile) for each of an item's tiles once */
        auto tiles = [&](const int *w, auto f) {
            int ts[2 * k], m = 0;
            auto add = [&](int t) {
                for (int r = 0; r < m; ++r)
                    if (ts[r] == t) return;
                ts[m++] = t;
                f(t);
            };
            for (int r = 0; r < k; ++r) add(tile_of(w[r]));
            if (!other.empty())
                for (int r = 0; r < k; ++r)
                    if (other[w[r]] >= 0) add(other[w[r]]);
        };
        for (int q = 0; q < count; ++q) tiles(v + (size_t)k * q, [&](int t) { L.off[t + 1]++; });
        for (int t = 0; t < T; ++t) L.off[t + 1] += L.off[t];
        L.item.resize(L.off[T]);
        std::vector<int> fill(L.off.begin(), L.off.end() - 1);
        for (int q = 0; q < count; ++q) {
            const int *const w = v + (size_t)k * q;
            tiles(w, [&](int t) { L.item[fill[t]++] = q; });
            for (int r = 0; r < k; ++r) L.slot[(size_t)k * q + r] = fill[tile_of(w[r])] - 1 - L.off[tile_of(w[r])];
        }
    };
    parallel_for<NoScratch>(3, items, [&](int kind, NoScratch &) {
        if (kind == 0) list(std::integral_constant<int, 3>(), nt, h.tri_hjk.data(), its[1]);
        if (kind == 1) list(std::integral_constant<int, 2>(), ne, h.edge_ij.data(), its[0]);
        if (kind == 2) list(std::integral_constant<int, 3>(), nel, h.facets.data(), its[2]);
    });
    out.desc.assign(T, Res64Desc{});
    out.rec.resize(T);
    std::vector<std::vector<int>> halos(T);
    std::vector<char> failed(T, 0);
    const bool has_k = !h.bond_k.empty(), has_kb = !h.tri_kb.empty(), has_phi = !h.tri_phi0.empty();
    parallel_for<TileScratch>(T, items, [&](int t, TileScratch &sc) {
        if (sc.loc.empty()) sc.loc.assign(n, -1);
        const std::vector<int> &un_of = tu[t];
        const int no = (int)un_of.size() * un;
        struct Span {
            const int *b, *e;
            const int *begin() const { return b; }
            const int *end() const { return e; }
            size_t size() const { return (size_t)(e - b); }
        };
        auto span = [&](int kind) {
            return Span{its[kind].item.data() + its[kind].off[t], its[kind].item.data() + its[kind].off[t + 1]};
        };
        const Span bl = span(0), tl = span(1), el = span(2);
        /* nodes gathered here: the own ones and other tiles' duplicate
         * partners of own ones; the longest lists first, so that the lanes of a
         * warp gather equally many */
        auto nbe = [&](int i) { return use_bonds ? inc.bptr[i + 1] - inc.bptr[i] : 0; };
        auto nte = [&](int i) { return use_triples ? inc.tptr[i + 1] - inc.tptr[i] : 0; };
        auto nee = [&](int i) { return eptr[i + 1] - eptr[i]; };
        std::vector<std::pair<unsigned, int>> gn; /* (descending lists, place), later (.., node) */
        std::vector<int> gather, ghosts, hal;
        gather.reserve(no);
        for (int u : un_of)
            for (int i = u * un; i < std::min(n, (u + 1) * un); ++i) {
                gather.push_back(i);
                if (!other.empty() && other[i] >= 0) ghosts.push_back(partner[i]);
            }
        std::sort(ghosts.begin(), ghosts.end());
        ghosts.erase(std::unique(ghosts.begin(), ghosts.end()), ghosts.end());
        gather.insert(gather.end(), ghosts.begin(), ghosts.end());
        gn.reserve(gather.size());
        size_t ni = 0;
        for (size_t k = 0; k < gather.size(); ++k) {
            const int i = gather[k], a = nbe(i), b = nte(i), c = nee(i);
            if (a > 255 || b > 255 || c > 255) {
                failed[t] = 1;
                return;
            }
            gn.push_back({0xffffffu - ((unsigned)c << 16 | (unsigned)b << 8 | (unsigned)a), (int)k});
            ni += (size_t)a + b + c;
        }
        std::sort(gn.begin(), gn.end());
        for (auto &g : gn) g.second = gather[g.second];
        hal.reserve(4 * (size_t)kChunk * un_of.size());
        auto touch = [&](int i) {
            if (tile_of(i) != t && sc.loc[i] < 0) {
                sc.loc[i] = 0;
                hal.push_back(i);
            }
        };
        for (int i : ghosts) touch(i);
        for (int b : bl) {
            touch(h.edge_ij[2 * b]);
            touch(h.edge_ij[2 * b + 1]);
        }
        for (int q : tl)
            for (int r = 0; r < 3; ++r) touch(h.tri_hjk[3 * q + r]);
        for (int q : el)
            for (int r = 0; r < 3; ++r) touch(h.facets[3 * q + r]);
        std::sort(hal.begin(), hal.end());
        for (size_t k = 0; k < hal.size(); ++k) sc.loc[hal[k]] = no + (int)k;
        struct Reset {
            TileScratch &sc;
            const std::vector<int> &hal;
            ~Reset() {
                for (int i : hal) sc.loc[i] = -1;
            }
        } reset{sc, hal};
        auto local = [&](int i) {
            const int u = i >> lg_un;
            return tile[u] == t ? (uslot[u] << lg_un) + (i & (un - 1)) : sc.loc[i];
        };
        if (no + hal.size() > 0xffff || bl.size() > 0x7fff || 3 * tl.size() > 0xffff || 3 * el.size() > 0xffff) {
            failed[t] = 1;
            return;
        }
        Res64Desc &td = out.desc[t];
        td.nu = (int)un_of.size();
        td.no = no;
        td.nh = (int)hal.size();
        td.nb = (int)bl.size();
        td.nt = (int)tl.size();
        td.nel = (int)el.size();
        td.ngather = (int)gn.size();
        td.ni = (int)ni;
        td.has_k = has_k;
        td.has_kb = has_kb;
        td.has_phi = has_phi;
        td.has_gel = nel > 0;
        const Res64Segs g = res64_segs(td, kResWhole);
        if (res64_segs(td, kResPairs).total > smem_limit) {
            failed[t] = 1;
            return;
        }
        std::vector<unsigned char> &o = out.rec[t];
        o.assign(g.rec, 0);
        unsigned char *const rec = o.data();
        auto put = [&](unsigned off, const void *src, size_t bytes) {
            if (bytes) memcpy(rec + off, src, bytes);
        };
        put(g.units, un_of.data(), 4 * un_of.size());
        put(g.halo, hal.data(), 4 * hal.size());
        for (size_t k = 0; k < bl.size(); ++k) {
            const int b = bl.b[k];
            const unsigned q = (unsigned)local(h.edge_ij[2 * b]) | (unsigned)local(h.edge_ij[2 * b + 1]) << 16;
            memcpy(rec + g.bref + 4 * k, &q, 4);
            memcpy(rec + g.bl0 + 8 * k, &h.edge_l0[b], 8);
            if (has_k) memcpy(rec + g.bk + 8 * k, &h.bond_k[b], 8);
            rec[g.bwrap + k] = (unsigned char)h.edge_wrap[b];
        }
        for (size_t k = 0; k < tl.size(); ++k) {
            const int q = tl.b[k];
            const uint2 w = make_uint2((unsigned)local(h.tri_hjk[3 * q]) | (unsigned)local(h.tri_hjk[3 * q + 1]) << 16,
                                       (unsigned)local(h.tri_hjk[3 * q + 2]) |
                                           (unsigned)(unsigned char)h.tri_wrap[2 * q] << 16 |
                                           (unsigned)(unsigned char)h.tri_wrap[2 * q + 1] << 24);
            memcpy(rec + g.tref + 8 * k, &w, 8);
            if (has_kb) memcpy(rec + g.tkb + 8 * k, &h.tri_kb[q], 8);
            if (has_phi) memcpy(rec + g.tphi + 8 * k, &h.tri_phi0[q], 8);
        }
        for (size_t k = 0; k < el.size(); ++k) {
            const int *f = &h.facets[3 * (size_t)el.b[k]];
            const uint2 w = make_uint2((unsigned)local(f[0]) | (unsigned)local(f[1]) << 16, (unsigned)local(f[2]));
            memcpy(rec + g.eref + 8 * k, &w, 8);
            memcpy(rec + g.eid + 4 * k, &el.b[k], 4);
        }
        /* gather records and entries; a ghost's items by their place in the
         * tile's lists */
        auto slot = [&](int kind, int k, int q, int r, bool ghost) -> int {
            if (!ghost) return its[kind].slot[(size_t)k * q + r];
            const Span l = kind == 0 ? bl : kind == 1 ? tl : el;
            return (int)(std::lower_bound(l.b, l.e, q) - l.b);
        };
        size_t at = 0;
        for (size_t k = 0; k < gn.size(); ++k) {
            const int i = gn[k].second;
            const bool ghost = tile_of(i) != t;
            if (at > 0xffff) {
                failed[t] = 1;
                return;
            }
            const uint2 w = make_uint2((unsigned)local(i) | (unsigned)nbe(i) << 16 | (unsigned)nte(i) << 24,
                                       (unsigned)at | (unsigned)nee(i) << 16 | (unsigned)(fcodes[i] & 3u) << 24);
            memcpy(rec + g.grec + 8 * k, &w, 8);
            auto entry = [&](int v) {
                const unsigned short c = (unsigned short)v;
                memcpy(rec + g.inc + 2 * at++, &c, 2);
            };
            if (use_bonds)
                for (int e = inc.bptr[i]; e < inc.bptr[i + 1]; ++e)
                    entry(slot(0, 2, inc.bent[e] >> 1, inc.bent[e] & 1, ghost) << 1 | (inc.bent[e] & 1));
            if (use_triples)
                for (int e = inc.tptr[i]; e < inc.tptr[i + 1]; ++e)
                    entry(3 * slot(1, 3, inc.tent[e] >> 2, inc.tent[e] & 3, ghost) + (inc.tent[e] & 3));
            for (int e = eptr[i]; e < eptr[i + 1]; ++e) entry(3 * slot(2, 3, eent[e] / 3, eent[e] % 3, ghost) + eent[e] % 3);
        }
        /* groups of 32 items in the order the warps take them: four of one
         * kind (one for each scheduler), then four of the other, so that a
         * scheduler's warps are not all in their FP64 or all in their integer
         * part at once; what is left over last, the short bonds */
        std::vector<unsigned short> heavy, light, grp;
        for (int k = 0; k < (td.nel + 31) / 32; ++k) heavy.push_back((unsigned short)(2 << 14 | k));
        for (int k = 0; k < (td.nt + 31) / 32; ++k) heavy.push_back((unsigned short)(1 << 14 | k));
        for (int k = 0; k < (td.nb + 31) / 32; ++k) light.push_back((unsigned short)k);
        for (size_t a = 0, b = 0; a < heavy.size() || b < light.size();) {
            for (int k = 0; k < 4 && a < heavy.size(); ++k) grp.push_back(heavy[a++]);
            for (int k = 0; k < 4 && b < light.size(); ++k) grp.push_back(light[b++]);
        }
        put(g.grp, grp.data(), 2 * grp.size());
        if (td.has_gel)
            for (int u = 0; u < td.nu; ++u)
                for (int k = 0; k < un; ++k) {
                    const int i = un_of[u] * un + k;
                    const unsigned short q = i < n && partner[i] >= 0 ? (unsigned short)local(partner[i]) : 0xffff;
                    put(g.partner + 2 * (unsigned)(u * un + k), &q, 2);
                }
        halos[t] = hal;
    });
    for (char f : failed)
        if (f) return NR_ERR_CAPACITY;
    /* own nodes in other tiles' halos are published every step */
    std::vector<unsigned char> wanted(n, 0);
    for (const auto &hal : halos)
        for (int i : hal) wanted[i] = 1;
    for (int t = 0; t < T; ++t) {
        const Res64Segs g = res64_segs(out.desc[t], kResWhole);
        for (int u = 0; u < out.desc[t].nu; ++u)
            for (int k = 0; k < un; ++k) {
                const int i = tu[t][u] * un + k;
                out.rec[t][g.pub + (unsigned)(u * un + k)] = i < n ? wanted[i] : 0;
            }
        out.desc[t].ro_off = out.ro_bytes; /* a multiple of 16 */
        out.ro_bytes += (long long)out.rec[t].size();
    }
    for (out.mode = kResWhole;; ++out.mode) {
        out.max_smem = 0;
        for (const Res64Desc &td : out.desc) out.max_smem = std::max(out.max_smem, (size_t)res64_segs(td, out.mode).total);
        if (out.max_smem <= smem_limit) break; /* at kResPairs at the latest (above) */
    }
    unsigned groups = 0;
    for (const Res64Desc &td : out.desc) groups = std::max(groups, res64_groups(td));
    const int n_tiles = (n + kTile - 1) / kTile;
    out.shape = kResAlone;
    if (out.mode == kResWhole && n_tiles <= kResSharedTiles) out.shape = kResShared;
    if (out.mode == kResWhole && n_tiles <= kResSmallTiles && groups <= kResSmallGroups) out.shape = kResSmall;
    return NR_OK;
}

int build_res64_layout(const nr_host_network &h, const Incidence &inc, const unsigned char *fcodes, bool use_bonds,
                       bool use_triples, const std::vector<int> &eptr, const std::vector<int> &eent,
                       const std::vector<int> &partner, int max_ctas, size_t smem_limit, Res64Host &out) {
    try {
        return build_layout(h, inc, fcodes, use_bonds, use_triples, eptr, eent, partner, max_ctas, smem_limit, out);
    } catch (...) { /* no memory: the network runs on the other kernels */
        out = Res64Host();
        return NR_ERR_OOM;
    }
}

/* nr_res64_layout_check; may throw. */
static int check_res64_layout(const nr_host_network *h, int ctas, long long smem_limit, long long stats[6]) {
    const int n = h->n_points;
    Incidence inc;
    build_incidence(n, h->edge_ij.data(), h->n_edges(), h->tri_hjk.data(), h->n_triples(), true, true, inc);
    std::vector<int> eptr, eent, partner;
    element_incidence(*h, eptr, eent, partner);
    std::vector<unsigned char> fc(n);
    nr_host_network_fcodes(h, fc.data());
    Res64Host L;
    const int rc = build_res64_layout(*h, inc, fc.data(), true, true, eptr, eent, partner, ctas, (size_t)smem_limit, L);
    if (rc != NR_OK) return rc;
    const int un = kChunk * L.sub;
    long long bad = 0, items = 0, halo = 0;
    std::vector<int> owned(n, 0), wanted(n, 0), published(n, 0);
    if (L.n_ctas > ctas || (int)L.desc.size() != L.n_ctas) ++bad;
    long long ro_end = 0;
    for (const Res64Desc &td : L.desc) {
        const Res64Segs g = res64_segs(td, L.mode);
        const std::vector<unsigned char> &record = L.rec[&td - L.desc.data()];
        const bool placed = td.ro_off % 16 == 0 && td.ro_off == ro_end && record.size() == res64_segs(td, kResWhole).rec;
        ro_end = td.ro_off + (long long)record.size();
        if (!placed || ro_end > L.ro_bytes || g.total > (unsigned)smem_limit ||
            g.total > L.max_smem || td.no != td.nu * un) {
            ++bad;
            continue;
        }
        const unsigned char *rec = record.data();
        auto at = [&](unsigned off, auto &v) { memcpy(&v, rec + off, sizeof v); };
        /* node id of a local index, -1 when it is none */
        auto node = [&](unsigned l) -> int {
            int id = -1;
            if (l < (unsigned)td.no) {
                at(g.units + 4 * (l / un), id);
                id = id * un + (int)(l % un);
                return id < n ? id : -1;
            }
            if (l < (unsigned)(td.no + td.nh)) at(g.halo + 4 * (l - td.no), id);
            return id >= 0 && id < n ? id : -1;
        };
        for (int l = 0; l < td.no; ++l) {
            const int i = node(l);
            if (i < 0) continue;
            owned[i]++;
            published[i] = rec[g.pub + l];
            if (td.has_gel) {
                unsigned short q;
                at(g.partner + 2 * l, q);
                if ((q == 0xffff) != (partner[i] < 0) || (q != 0xffff && node(q) != partner[i])) ++bad;
            }
        }
        for (int k = 0; k < td.nh; ++k) {
            const int i = node(td.no + k);
            if (i < 0) ++bad;
            else wanted[i] = 1;
        }
        std::vector<int> bid(td.nb, -1), tid(td.nt, -1), els(td.nel, -1);
        std::vector<unsigned short> codes(res64_groups(td));
        for (size_t k = 0; k < codes.size(); ++k) at(g.grp + 2 * (unsigned)k, codes[k]);
        std::sort(codes.begin(), codes.end());
        for (size_t k = 0; k < codes.size(); ++k) {
            const size_t gb = (size_t)(td.nb + 31) / 32, gt = (size_t)(td.nt + 31) / 32;
            const size_t want = k < gb ? k : k < gb + gt ? (1u << 14 | (k - gb)) : (2u << 14 | (k - gb - gt));
            bad += codes[k] != want;
        }
        for (int k = 0; k < td.nel; ++k) {
            uint2 w;
            at(g.eid + 4 * k, els[k]);
            at(g.eref + 8 * k, w);
            const int *f = els[k] >= 0 && els[k] < h->n_facets() ? &h->facets[3 * (size_t)els[k]] : nullptr;
            if (!f || node(w.x & 0xffff) != f[0] || node(w.x >> 16) != f[1] || node(w.y) != f[2]) ++bad;
        }
        int gathered = 0;
        for (int k = 0; k < td.ngather; ++k) {
            uint2 w;
            at(g.grec + 8 * k, w);
            const int i = node(w.x & 0xffff);
            const int nbn = (w.x >> 16) & 255, ntn = w.x >> 24, nen = (w.y >> 16) & 255, e0 = w.y & 0xffff;
            if (i < 0 || (w.y >> 24) != (fc[i] & 3u) || e0 + nbn + ntn + nen > td.ni || nbn != inc.bptr[i + 1] - inc.bptr[i] ||
                ntn != inc.tptr[i + 1] - inc.tptr[i] || nen != eptr[i + 1] - eptr[i]) {
                ++bad;
                continue;
            }
            gathered += (w.x & 0xffff) < (unsigned)td.no;
            for (int a = 0; a < nbn + ntn + nen; ++a) {
                unsigned short c;
                at(g.inc + 2 * (e0 + a), c);
                if (a < nbn) {
                    const int b = inc.bent[inc.bptr[i] + a] >> 1;
                    unsigned q;
                    double l0;
                    if ((c >> 1) >= td.nb || (c & 1) != (inc.bent[inc.bptr[i] + a] & 1)) {
                        ++bad;
                        continue;
                    }
                    at(g.bref + 4 * (c >> 1), q);
                    at(g.bl0 + 8 * (c >> 1), l0);
                    if (node(q & 0xffff) != h->edge_ij[2 * b] || node(q >> 16) != h->edge_ij[2 * b + 1] ||
                        l0 != h->edge_l0[b] || (signed char)rec[g.bwrap + (c >> 1)] != h->edge_wrap[b])
                        ++bad;
                    if (bid[c >> 1] >= 0 && bid[c >> 1] != b) ++bad;
                    bid[c >> 1] = b;
                } else if (a < nbn + ntn) {
                    const int e = inc.tent[inc.tptr[i] + a - nbn], t = e >> 2;
                    uint2 q;
                    if (c / 3 >= td.nt || c % 3 != (e & 3)) {
                        ++bad;
                        continue;
                    }
                    at(g.tref + 8 * (c / 3), q);
                    if (node(q.x & 0xffff) != h->tri_hjk[3 * t] || node(q.x >> 16) != h->tri_hjk[3 * t + 1] ||
                        node(q.y & 0xffff) != h->tri_hjk[3 * t + 2] ||
                        (signed char)(q.y >> 16) != h->tri_wrap[2 * t] || (signed char)(q.y >> 24) != h->tri_wrap[2 * t + 1])
                        ++bad;
                    if (tid[c / 3] >= 0 && tid[c / 3] != t) ++bad;
                    tid[c / 3] = t;
                } else {
                    const int e = eent[eptr[i] + a - nbn - ntn];
                    if (c / 3 >= td.nel || els[c / 3] != e / 3 || c % 3 != e % 3) ++bad;
                }
            }
        }
        int own_nodes = 0;
        for (int l = 0; l < td.no; ++l) own_nodes += node(l) >= 0;
        if (gathered != own_nodes) ++bad;
        for (int b : bid) bad += b < 0;
        for (int t : tid) bad += t < 0;
        items += td.nb + td.nt + td.nel;
        halo += td.nh;
    }
    for (int i = 0; i < n; ++i) bad += owned[i] != 1 || wanted[i] != published[i];
    stats[0] = L.n_ctas;
    stats[1] = L.sub;
    stats[2] = (long long)L.max_smem;
    stats[3] = items;
    stats[4] = halo;
    stats[5] = bad;
    return NR_OK;
}

}  // namespace nr

extern "C" int nr_res64_layout_check(const nr_host_network *h, int ctas, long long smem_limit, long long stats[6]) {
    if (!h || !stats || ctas < 1 || smem_limit < 1) return NR_ERR_INVALID;
    for (int k = 0; k < 6; ++k) stats[k] = 0;
    try {
        return nr::check_res64_layout(h, ctas, smem_limit, stats);
    } catch (...) {
        return NR_ERR_OOM;
    }
}
