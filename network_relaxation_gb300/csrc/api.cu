/*
 * C ABI implementation: device images of networks and batches, relaxation
 * entry points, the strain sweep and the run_fire_md drop-in.
 *
 * Every network (or batch of networks) lives in ONE device allocation built
 * from a host staging image: node state first (x, v, f of all networks
 * contiguous, so a batch's positions are one array), then the FIRE states,
 * then per network its topology, incidence lists and reduction scratch; what
 * starts as zeros lies behind the uploaded part, in the same order.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "fire_launch.h"
#include "nr_device.cuh"
#include "nr_internal.h"

namespace nr {

#define NR_CUDA_TRY(call)                                                                        \
    do {                                                                                         \
        cudaError_t e_ = (call);                                                                 \
        if (e_ != cudaSuccess)                                                                   \
            return fail(NR_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));        \
    } while (0)

/* Wait budget of every grid barrier: NR_BARRIER_BUDGET_MS (default 2000). */
static unsigned long long barrier_budget_ns() {
    const char *env = getenv("NR_BARRIER_BUDGET_MS");
    double ms = env ? atof(env) : 2000.0;
    if (!(ms > 0)) ms = 2000.0;
    return (unsigned long long)(ms * 1e6);
}

/* Failure injection on the host for the wait-budget test:
 * NR_TEST_STALL_BARRIER=k makes the FP64 grid kernel's barriers wait for k
 * CTAs that were never launched, so the first wait runs out of its budget
 * and the relaxation ends with NR_ERR_TIMEOUT (no fault; the context stays
 * usable).  Unset or 0 in normal use. */
static unsigned barrier_stall() {
    const char *env = getenv("NR_TEST_STALL_BARRIER");
    const int k = env ? atoi(env) : 0;
    return k > 0 && k < 1024 ? (unsigned)k : 0u;
}

struct NetOff {
    size_t mb_data, mb_sk, bdf, mt_arms, mt_pk, tdf, bfrc, tfrc;
    size_t dsm_bref, dsm_bidx, dsm_tref, dsm_bent, dsm_tent, dsm_grec, dsm_xrec, dsm_xent;
    size_t fcode, bond, bond_l0, bond_k, tri, tri_kb, tri_phi0, bptr, bent, tptr, tent, part, epart;
    size_t elem, elem_inv, elem_area, efrc, eptr, eent, partner;
    bool has_bond_k, has_tri_kb, has_tri_phi0, has_dsm_quads;
};

/* Device image of n networks (n = 1 for nr_network). */
struct DeviceSet {
    int n_nets = 0;
    long total_nodes = 0;
    std::vector<long> node_off;
    std::vector<NetDev> dev;
    std::vector<double> miny, maxy, minx;
    /* gel coupling possible: every node is in at most one duplicate pair */
    std::vector<char> gel_ok;
    std::vector<NetGel> gel; /* host copies of the device array gel_array */
    NetGel *gel_array = nullptr;
    char *arena = nullptr;
    size_t arena_bytes = 0;
    NetDev *dev_array = nullptr;
    FireState *st = nullptr;
    int *queue = nullptr;
    double4 *affine_prm = nullptr;
    double2 *x_all = nullptr, *v_all = nullptr, *f_all = nullptr;
    float4 *u_all = nullptr;
    float2 *vf_all = nullptr, *ff_all = nullptr;
    float2 *fa_hi_all = nullptr, *fa_lo_all = nullptr;
    int max_nodes = 0;
    int *order = nullptr; /* networks by decreasing size (largest start first) */
    int *order2 = nullptr; /* networks of a later escalation phase */
    /* sub-block layouts for the distributed-shared-memory kernel (host copy
     * for sizing, device array for the kernel); dsm_ok: every network has one */
    std::vector<NetDsm> dsm;
    NetDsm *dsm_array = nullptr;
    bool dsm_ok = true;
    int launches = 0; /* kernel launches of the last batch relaxation */
    std::vector<int> order_host;
    /* second stream and events for the concurrent single-CTA launch */
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    /* tiled layout of a single large network (fire_tile.cu); tile_ctas = 0:
     * none */
    NetTile tile{};
    char *tile_mem = nullptr;
    int tile_ctas = 0;
    int tile_threads = 512;
    /* resident FP64 layout of a single network (fire_res64.cu); n_ctas = 0:
     * none */
    Res64Dev res{};
    size_t res_smem = 0;
    ~DeviceSet() {
        if (tile_mem) cudaFree(tile_mem);
        if (arena) cudaFree(arena);
        if (side) cudaStreamDestroy(side);
        if (ev_fork) cudaEventDestroy(ev_fork);
        if (ev_join) cudaEventDestroy(ev_join);
    }
};

/* Sub-block layout of one network for the distributed-shared-memory kernels
 * (NetDsm, nr_device.cuh): item slots grouped by the sub-block of the
 * bond's node i / the triple's hinge, in index order within a group; node
 * references and resolved incidence entries; per node, in gather order,
 * its gather record.  m.bsub = 0 when the network is too large for the
 * encoding (more than 2^20 nodes).  The mixed kernel's quads (xrec, xent) are
 * left out where 32 B a node of 16 CTAs, the least it keeps in shared memory,
 * exceed an SM's: a node of many entries has 31 others' lists filled up to its
 * own. */
constexpr int kDsmMaxSubBlock = 227 * 1024 / 32;
static void build_dsm_layout(const nr_host_network &h, const Incidence &inc, const unsigned char *fcodes, Image &img,
                             NetOff &o, NetDsm &m) {
    const int n = h.n_points, ne = h.n_edges(), nt = h.n_triples();
    memset(&m, 0, sizeof(m));
    /* sub-blocks of a whole number of 32-node chunks: a CTA's nodes then
     * start on a chunk boundary, which the FP64 cluster kernel's canonical
     * reduction (32-node units) needs */
    const int bsub = kChunk * ((n + kDsmParts * kChunk - 1) / (kDsmParts * kChunk));
    const bool fits = n <= (1 << 20) && bsub <= 0xffff;
    auto part = [&](int v) { return v / bsub; };
    auto ref = [&](int v) { return (part(v) << 16) | (v % bsub); };
    std::vector<int2> bref(fits ? ne : 0);
    std::vector<int> bidx(fits ? ne : 0), bslot(fits ? ne : 0), dbent(fits ? inc.bent.size() : 0);
    const bool has_quads = fits && bsub <= kDsmMaxSubBlock;
    std::vector<int4> tref(fits ? nt : 0), grec(fits ? n : 0), xrec(has_quads ? n : 0);
    size_t quads = 0;
    std::vector<int> tslot(fits ? nt : 0), dtent(fits ? inc.tent.size() : 0);
    if (fits) {
        int cnt[kDsmParts + 1] = {0};
        for (int b = 0; b < ne; ++b) cnt[part(h.edge_ij[2 * b]) + 1]++;
        for (int g = 0; g < kDsmParts; ++g) cnt[g + 1] += cnt[g];
        for (int g = 0; g <= kDsmParts; ++g) m.bo[g] = cnt[g];
        for (int b = 0; b < ne; ++b) {
            const int i = h.edge_ij[2 * b], j = h.edge_ij[2 * b + 1];
            const int sl = cnt[part(i)]++;
            bslot[b] = sl;
            bref[sl] = make_int2(ref(i), ref(j));
            bidx[sl] = b;
        }
        int tc[kDsmParts + 1] = {0};
        for (int t = 0; t < nt; ++t) tc[part(h.tri_hjk[3 * t]) + 1]++;
        for (int g = 0; g < kDsmParts; ++g) tc[g + 1] += tc[g];
        for (int g = 0; g <= kDsmParts; ++g) m.to[g] = tc[g];
        for (int t = 0; t < nt; ++t) {
            const int hh = h.tri_hjk[3 * t], jj = h.tri_hjk[3 * t + 1], kk = h.tri_hjk[3 * t + 2];
            const int sl = tc[part(hh)]++;
            tslot[t] = sl;
            tref[sl] = make_int4(ref(hh), ref(jj), ref(kk), t);
        }
        for (size_t e = 0; e < inc.bent.size(); ++e) {
            const int b = inc.bent[e] >> 1, role = inc.bent[e] & 1;
            const unsigned g = (unsigned)part(h.edge_ij[2 * b]);
            dbent[e] = (int)((g << 28) | ((unsigned)bslot[b] << 1) | (unsigned)role);
        }
        for (size_t e = 0; e < inc.tent.size(); ++e) {
            const int t = inc.tent[e] >> 2, role = inc.tent[e] & 3;
            const unsigned g = (unsigned)part(h.tri_hjk[3 * t]);
            dtent[e] = (int)((g << 28) | ((unsigned)tslot[t] << 2) | (unsigned)role);
        }
        for (int g = 0; g <= kDsmParts; ++g) {
            const int v = std::min(n, g * bsub);
            m.be[g] = inc.bptr[v];
            m.te[g] = inc.tptr[v];
        }
        /* gather records: within each sub-block the nodes ordered by their
         * numbers of triple and bond entries, so the lanes of a warp walk
         * (nearly) equally long lists */
        std::vector<int> ord;
        for (int g = 0; g * bsub < n; ++g) {
            const int v0 = g * bsub, v1 = std::min(n, v0 + bsub);
            ord.resize(v1 - v0);
            for (int v = v0; v < v1; ++v) ord[v - v0] = v;
            auto nbe = [&](int v) { return inc.bptr[v + 1] - inc.bptr[v]; };
            auto nte = [&](int v) { return inc.tptr[v + 1] - inc.tptr[v]; };
            std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) {
                return nte(a) != nte(b) ? nte(a) > nte(b) : nbe(a) > nbe(b);
            });
            for (int k = 0; k < v1 - v0; ++k) {
                const int v = ord[k];
                grec[v0 + k] = make_int4(v | ((int)(fcodes[v] & 3u) << 28), inc.bptr[v], nbe(v) | (nte(v) << 16),
                                         inc.tptr[v]);
            }
            /* bsub is a multiple of 32: the groups of a sub-block are the
             * groups a warp gathers */
            for (int k0 = 0; has_quads && k0 < v1 - v0; k0 += 32) {
                const int k1 = std::min(v1 - v0, k0 + 32);
                int nq = 0;
                for (int k = k0; k < k1; ++k) nq = std::max(nq, (nbe(ord[k]) + nte(ord[k]) + 3) / 4);
                for (int k = k0; k < k1; ++k) xrec[v0 + k] = make_int4(grec[v0 + k].x, (int)quads, nq, 0);
                quads += (size_t)32 * nq;
            }
        }
        m.bsub = bsub;
    }
    o.dsm_bref = img.put(bref.data(), bref.size());
    o.dsm_bidx = img.put(bidx.data(), bidx.size());
    o.dsm_tref = img.put(tref.data(), tref.size());
    o.dsm_bent = img.put(dbent.data(), dbent.size());
    o.dsm_tent = img.put(dtent.data(), dtent.size());
    o.dsm_grec = img.put(grec.data(), grec.size());
    o.has_dsm_quads = has_quads;
    o.dsm_xrec = img.put(xrec.data(), xrec.size());
    o.dsm_xent = img.zeros(sizeof(uint4) * quads); /* written by the kernel */
}

/* Networks of at least NR_TILE_MIN_NODES nodes (default 131072) relaxed
 * alone in mixed precision use the tiled kernel, tiles of about
 * NR_TILE_NODES nodes (default 512). */
static int tile_min_nodes() {
    const char *env = knob("NR_TILE_MIN_NODES");
    return env ? std::max(1, atoi(env)) : 131072;
}
static int tile_target_nodes() {
    const char *env = knob("NR_TILE_NODES");
    const int v = env ? atoi(env) : 512;
    return v >= 64 && v <= 8192 ? v : 512;
}
/* Threads per CTA of the tiled kernel (NR_TILE_THREADS): 512 (default) or
 * 768, one CTA per SM, or 256, two CTAs per SM. */
static int tile_threads() {
    const char *env = knob("NR_TILE_THREADS");
    const int v = env ? atoi(env) : 512;
    return v == 256 || v == 768 ? v : 512;
}

/* Builds and uploads the tiled layout of network 0 of S (one allocation);
 * leaves S.tile_ctas = 0 when the network does not fit its encoding or the
 * kernel cannot launch.  One or two CTAs per SM (NR_TILE_THREADS); the
 * tile size is the largest of NR_TILE_NODES, 4/5 of it, 16/25 ... whose two
 * stage buffers and working arrays fit the CTA's shared memory. */
static int build_tile_set(const nr_host_network &h, const Incidence &inc, const unsigned char *fcodes, DeviceSet &S,
                          cudaStream_t stream) {
    int dev = 0, sms = 0, optin = 0;
    NR_CUDA_TRY(cudaGetDevice(&dev));
    NR_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    NR_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    int per_sm_smem = 0;
    NR_CUDA_TRY(cudaDeviceGetAttribute(&per_sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    const int threads = tile_threads(), per_sm = threads == 256 ? 2 : 1;
    /* dynamic shared memory a CTA may take: the opt-in maximum less a
     * margin, or, when two CTAs share the SM, half of it less the per-CTA
     * reservation and the kernel's static shared memory */
    const size_t limit = per_sm == 1 ? (size_t)optin - 8192 : (size_t)per_sm_smem / 2 - 3072;
    const NetDev &d = S.dev[0];
    TileHost th;
    NetTile &tl = S.tile;
    bool ok = false;
    for (int target = tile_target_nodes(); target >= 64 && !ok; target = target * 4 / 5) {
        for (const bool quads : {true, false}) {
            if (build_tile_layout(h, inc, fcodes, d.use_bonds != 0, d.use_triples != 0, per_sm * sms, target, quads, th) !=
                NR_OK)
                return NR_OK;
            tl = NetTile{};
            tl.n_tiles = th.n_tiles;
            tl.n_pos = th.n_pos;
            tl.max_nodes = th.max_nodes;
            tl.max_bonds = th.max_bonds;
            tl.max_tris = th.max_tris;
            tl.max_own = th.max_own;
            tl.max_ro = th.max_ro;
            tl.quads = quads;
            ok = tile_plan_smem(th) <= limit;
            /* quads that do not fit (a hub's list fills up 31 others') */
            if (!ok || tile_smem(tl) <= limit) break;
        }
    }
    if (!ok) return NR_OK;
    /* every tile record is a whole number of 16-byte units at a 16-byte
     * offset, as cp.async.bulk requires */
    for (const TileDesc &td : th.desc)
        if (td.ro_off % 16 != 0 || tile_segs(td).total % 16 != 0)
            return fail(NR_ERR_INVALID, "tile layout: record not 16-byte aligned");
    const int ctas = tile_grid_ctas(tl, threads);
    if (ctas < 1) {
        cudaGetLastError();
        return NR_OK;
    }
    Image img;
    const size_t np = (size_t)th.n_pos;
    const size_t o_desc = img.put(th.desc.data(), th.desc.size());
    const size_t o_ro = img.put(th.ro.data(), th.ro.size());
    const size_t o_nop = img.put(th.node_of_pos.data(), th.node_of_pos.size());
    const size_t o_bid = img.put(th.bid.data(), th.bid.size());
    const size_t o_tid = img.put(th.tid.data(), th.tid.size());
    size_t o_u[2], o_vf[2];
    for (int c = 0; c < 2; ++c) {
        o_u[c] = img.zeros(sizeof(float4) * np);
        o_vf[c] = img.zeros(sizeof(float4) * np);
    }
    const size_t o_fa = img.zeros(sizeof(float4) * np);
    const size_t o_cpart = img.zeros(sizeof(float) * 5 * 2 * (size_t)ctas);
    const size_t o_dpart = img.zeros(sizeof(double) * 2 * (size_t)ctas);
    const size_t o_bar = img.zeros(sizeof(unsigned long long));
    cudaError_t e = cudaMalloc((void **)&S.tile_mem, img.total());
    if (e != cudaSuccess) {
        S.tile_mem = nullptr;
        return fail(e == cudaErrorMemoryAllocation ? NR_ERR_OOM : NR_ERR_CUDA,
                    std::string("cudaMalloc (tile layout): ") + cudaGetErrorString(e));
    }
    char *b = S.tile_mem, *zeros = S.tile_mem + img.zeros_at();
    NR_CUDA_TRY(cudaMemcpyAsync(S.tile_mem, img.data(), img.size(), cudaMemcpyHostToDevice, stream));
    NR_CUDA_TRY(cudaMemsetAsync(zeros, 0, img.zeros_size(), stream));
    NR_CUDA_TRY(cudaStreamSynchronize(stream));
    tl.desc = (const TileDesc *)(b + o_desc);
    tl.ro = (unsigned char *)(b + o_ro);
    tl.node_of_pos = (const int *)(b + o_nop);
    tl.bid = (const int *)(b + o_bid);
    tl.tid = (const int *)(b + o_tid);
    for (int c = 0; c < 2; ++c) {
        tl.u[c] = (float4 *)(zeros + o_u[c]);
        tl.vf[c] = (float4 *)(zeros + o_vf[c]);
    }
    tl.fa = (float4 *)(zeros + o_fa);
    tl.cpart = (float *)(zeros + o_cpart);
    tl.dpart = (double *)(zeros + o_dpart);
    tl.bar = (unsigned long long *)(zeros + o_bar);
    S.tile_ctas = ctas;
    S.tile_threads = threads;
    return NR_OK;
}

/* NR_FP64_KERNEL: res (default), dsm, l2 or grid. */
enum { kFp64Res, kFp64Dsm, kFp64L2, kFp64Grid };
static int fp64_kernel_choice() {
    const char *env = knob("NR_FP64_KERNEL");
    if (env && strcmp(env, "dsm") == 0) return kFp64Dsm;
    if (env && strcmp(env, "l2") == 0) return kFp64L2;
    if (env && strcmp(env, "grid") == 0) return kFp64Grid;
    return kFp64Res;
}

/* FP64, one network.  All kernels give the same bits.  The resident kernel
 * takes whatever fits the SMs' shared memory in one of its modes (about
 * 200 000 nodes of a p = 0.65 lattice).  A cluster of NR_FP64_CLUSTER CTAs
 * (default 16; NR_FP64_KERNEL=dsm or l2, and in the resident kernel's place up
 * to kFp64DsmNodes where that does not fit) takes networks of at most
 * NR_FP64_CLUSTER_NODES nodes: it has the FP64 pipes of 16 SMs, and past that
 * line the cooperative grid kernel on all of them is faster (us a step, dsm /
 * l2 / grid: 4 096 nodes 19 / 28 / 41, 9 216 nodes 37 / 55 / 46, 32 761 nodes
 * 136 / 136 / 41).  0: the grid kernel alone. */
constexpr int kFp64DsmNodes = 4096;
static int fp64_cluster_nodes() {
    const char *env = knob("NR_FP64_CLUSTER_NODES");
    return env ? std::max(0, atoi(env)) : 16384;
}

/* Offsets of the resident FP64 layout in a network's image. */
struct ResOff {
    size_t desc, ro, vf[2], part[2], maxp[2], bar;
};

/* Adds the resident FP64 layout of the (single) network h to the image; false
 * when it does not fit. */
static bool add_res_layout(const nr_host_network &h, const Incidence &inc, const unsigned char *fcodes, bool use_bonds,
                           bool use_triples, const std::vector<int> &eptr, const std::vector<int> &eent,
                           const std::vector<int> &partner, Image &img, ResOff &o, Res64Host &L) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (build_res64_layout(h, inc, fcodes, use_bonds, use_triples, eptr, eent, partner, sms, res64_smem_limit(), L) !=
        NR_OK)
        return false;
    if (!res64_fits(L.n_ctas, L.shape, false, L.mode, L.max_smem) ||
        (h.n_facets() > 0 && !res64_fits(L.n_ctas, L.shape, true, L.mode, L.max_smem)))
        return false;
    o.desc = img.put(L.desc.data(), L.desc.size());
    o.ro = img.add((size_t)L.ro_bytes);
    for (int t = 0; t < L.n_ctas; ++t) memcpy(img.data() + o.ro + L.desc[t].ro_off, L.rec[t].data(), L.rec[t].size());
    for (int c = 0; c < 2; ++c) {
        o.vf[c] = img.zeros(sizeof(double2) * 2 * (size_t)h.n_points);
        o.part[c] = img.zeros(sizeof(double) * 3 * (size_t)L.n_units);
        o.maxp[c] = img.zeros(sizeof(unsigned long long) * (size_t)L.n_ctas);
    }
    o.bar = img.zeros(sizeof(unsigned long long));
    return true;
}

/* May throw. */
static int fill_set(int n, const nr_host_network *const *nets, const double *ks, const double *kb,
                    const unsigned char *const *fcodes_in, cudaStream_t stream, DeviceSet &S) {
    if (n <= 0) return fail(NR_ERR_INVALID, "network count must be positive");
    Image img;
    S.n_nets = n;
    S.node_off.assign(n + 1, 0);
    for (int i = 0; i < n; ++i) {
        if (!nets[i] || nets[i]->n_points <= 0) return fail(NR_ERR_INVALID, "empty network");
        S.node_off[i + 1] = S.node_off[i] + nets[i]->n_points;
    }
    S.total_nodes = S.node_off[n];
    const size_t x_off = img.add(sizeof(double2) * S.total_nodes);
    const size_t v_off = img.zeros(sizeof(double2) * S.total_nodes);
    const size_t f_off = img.zeros(sizeof(double2) * S.total_nodes);
    const size_t u_off = img.zeros(sizeof(float4) * S.total_nodes);
    const size_t vf_off = img.zeros(sizeof(float2) * S.total_nodes);
    const size_t ff_off = img.zeros(sizeof(float2) * S.total_nodes);
    const size_t fah_off = img.zeros(sizeof(float2) * S.total_nodes);
    const size_t fal_off = img.zeros(sizeof(float2) * S.total_nodes);
    std::vector<int> order(n);
    for (int i = 0; i < n; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return nets[a]->n_points > nets[b]->n_points; });
    const size_t order_off = img.put(order.data(), order.size());
    S.order_host = order;
    const size_t order2_off = img.zeros(sizeof(int) * n);
    const size_t st_off = img.zeros(sizeof(FireState) * n);
    const size_t q_off = img.zeros(256);
    const size_t aff_off = img.zeros(sizeof(double4) * n);
    const size_t dev_off = img.add(sizeof(NetDev) * n);
    const size_t dsm_off = img.add(sizeof(NetDsm) * n);
    const size_t gel_off = img.add(sizeof(NetGel) * n);
    S.dsm.assign(n, NetDsm{});
    S.gel.assign(n, NetGel{});
    std::vector<NetOff> off(n);
    const bool want_tile = n == 1 && nets[0]->n_points >= tile_min_nodes();
    const bool want_res = n == 1 && fp64_kernel_choice() == kFp64Res && fp64_cluster_nodes() > 0;
    Incidence inc0;
    std::vector<unsigned char> fc0;
    bool have_res = false;
    ResOff res_off{};
    Res64Host res_host;
    for (int i = 0; i < n; ++i) {
        const nr_host_network &h = *nets[i];
        memcpy(img.data() + x_off + sizeof(double2) * S.node_off[i], h.points.data(),
               sizeof(double) * 2 * h.n_points);
        std::vector<unsigned char> fc(h.n_points);
        if (fcodes_in && fcodes_in[i]) memcpy(fc.data(), fcodes_in[i], h.n_points);
        else nr_host_network_fcodes(&h, fc.data());
        const int ne = h.n_edges(), nt = h.n_triples();
        std::vector<int4> bond(ne);
        for (int e = 0; e < ne; ++e) bond[e] = make_int4(h.edge_ij[2 * e], h.edge_ij[2 * e + 1], h.edge_wrap[e], 0);
        std::vector<int4> tri(nt);
        for (int t = 0; t < nt; ++t)
            tri[t] = make_int4(h.tri_hjk[3 * t], h.tri_hjk[3 * t + 1], h.tri_hjk[3 * t + 2],
                               (h.tri_wrap[2 * t] & 255) | ((h.tri_wrap[2 * t + 1] & 255) << 8));
        Incidence inc;
        build_incidence(h.n_points, h.edge_ij.data(), ne, h.tri_hjk.data(), nt, ks[i] > 0, kb[i] > 0, inc);
        NetOff &o = off[i];
        o.fcode = img.put(fc.data(), fc.size());
        o.bond = img.put(bond.data(), bond.size());
        o.bond_l0 = img.put(h.edge_l0.data(), h.edge_l0.size());
        o.has_bond_k = !h.bond_k.empty();
        o.bond_k = img.put(h.bond_k.data(), h.bond_k.size());
        o.tri = img.put(tri.data(), tri.size());
        o.has_tri_kb = !h.tri_kb.empty();
        o.tri_kb = img.put(h.tri_kb.data(), h.tri_kb.size());
        o.has_tri_phi0 = !h.tri_phi0.empty();
        o.tri_phi0 = img.put(h.tri_phi0.data(), h.tri_phi0.size());
        o.bptr = img.put(inc.bptr.data(), inc.bptr.size());
        o.bent = img.put(inc.bent.data(), inc.bent.size());
        o.tptr = img.put(inc.tptr.data(), inc.tptr.size());
        o.tent = img.put(inc.tent.data(), inc.tent.size());
        /* mixed precision: per-item anchor records and force changes */
        o.mb_data = img.zeros(sizeof(float4) * (size_t)ne);
        o.mb_sk = img.zeros(sizeof(float2) * (size_t)ne);
        o.bdf = img.zeros(sizeof(float2) * (size_t)ne);
        o.mt_arms = img.zeros(sizeof(float4) * (size_t)nt);
        o.mt_pk = img.zeros(sizeof(float2) * (size_t)nt);
        o.tdf = img.zeros(sizeof(float4) * (size_t)nt);
        o.bfrc = img.zeros(sizeof(double2) * (size_t)ne);
        o.tfrc = img.zeros(sizeof(double4) * (size_t)nt);
        /* gel: triangles, inverse matrices (computed on the device after the
         * upload), element terms, per-node element incidence (3 e + role,
         * elements in index order) and duplicate partners */
        const int nf = h.n_facets();
        std::vector<int4> elem(nf);
        for (int f = 0; f < nf; ++f) elem[f] = make_int4(h.facets[3 * f], h.facets[3 * f + 1], h.facets[3 * f + 2], 0);
        std::vector<int> eptr, eent, partner;
        const bool pairs_ok = element_incidence(h, eptr, eent, partner);
        S.gel_ok.push_back(pairs_ok);
        S.minx.push_back(h.minx);
        o.elem = img.put(elem.data(), elem.size());
        o.elem_inv = img.zeros(sizeof(double) * 6 * (size_t)nf);
        o.elem_area = img.put(h.areas.data(), h.areas.size());
        o.efrc = img.zeros(sizeof(double4) * 3 * (size_t)nf);
        o.eptr = img.put(eptr.data(), eptr.size());
        o.eent = img.put(eent.data(), eent.size());
        o.partner = img.put(partner.data(), partner.size());
        build_dsm_layout(h, inc, fc.data(), img, o, S.dsm[i]);
        if (want_res && i == 0)
            have_res = add_res_layout(h, inc, fc.data(), ks[i] > 0, kb[i] > 0, eptr, eent, partner, img, res_off,
                                      res_host);
        if (want_tile && i == 0) {
            inc0 = std::move(inc);
            fc0 = fc;
        }
        if (S.dsm[i].bsub <= 0) S.dsm_ok = false;
        S.max_nodes = std::max(S.max_nodes, h.n_points);
        const int tiles = (h.n_points + kTile - 1) / kTile;
        o.part = img.zeros(sizeof(double) * 4 * (size_t)tiles * 8);
        const int tb = (ne + kTile - 1) / kTile, tt = (nt + kTile - 1) / kTile, tg = (nf + kTile - 1) / kTile;
        o.epart = img.zeros(sizeof(double) * kEpartLists * (size_t)std::max(1, std::max(tb, std::max(tt, tg))));
        S.miny.push_back(h.miny);
        S.maxy.push_back(h.maxy);
    }
    S.arena_bytes = img.total();
    cudaError_t e = cudaMalloc((void **)&S.arena, S.arena_bytes);
    if (e != cudaSuccess) {
        S.arena = nullptr;
        return fail(e == cudaErrorMemoryAllocation ? NR_ERR_OOM : NR_ERR_CUDA,
                    std::string("cudaMalloc: ") + cudaGetErrorString(e));
    }
    char *base = S.arena, *zeros = S.arena + img.zeros_at();
    S.x_all = (double2 *)(base + x_off);
    S.v_all = (double2 *)(zeros + v_off);
    S.f_all = (double2 *)(zeros + f_off);
    S.u_all = (float4 *)(zeros + u_off);
    S.vf_all = (float2 *)(zeros + vf_off);
    S.ff_all = (float2 *)(zeros + ff_off);
    S.fa_hi_all = (float2 *)(zeros + fah_off);
    S.fa_lo_all = (float2 *)(zeros + fal_off);
    S.order = (int *)(base + order_off);
    S.order2 = (int *)(zeros + order2_off);
    S.st = (FireState *)(zeros + st_off);
    S.queue = (int *)(zeros + q_off);
    S.affine_prm = (double4 *)(zeros + aff_off);
    S.dev_array = (NetDev *)(base + dev_off);
    S.dev.resize(n);
    for (int i = 0; i < n; ++i) {
        const nr_host_network &h = *nets[i];
        const NetOff &o = off[i];
        NetDev &d = S.dev[i];
        memset(&d, 0, sizeof(d));
        d.n = h.n_points;
        d.n_edges = h.n_edges();
        d.n_triples = h.n_triples();
        d.n_tiles = (d.n + kTile - 1) / kTile;
        d.use_bonds = ks[i] > 0;
        d.use_triples = kb[i] > 0;
        d.sub = 8;
        d.n_units = d.n_tiles;
        d.width = h.offset;
        d.ks = ks[i];
        d.kb = kb[i];
        d.sqrt_dof = std::sqrt((double)(2L * d.n));
        d.area = h.offset * (h.maxy - h.miny);
        d.x = S.x_all + S.node_off[i];
        d.v = S.v_all + S.node_off[i];
        d.f = S.f_all + S.node_off[i];
        d.u = S.u_all + S.node_off[i];
        d.vf = S.vf_all + S.node_off[i];
        d.ff = S.ff_all + S.node_off[i];
        d.fa_hi = S.fa_hi_all + S.node_off[i];
        d.fa_lo = S.fa_lo_all + S.node_off[i];
        d.mb_data = (float4 *)(zeros + o.mb_data);
        d.mb_sk = (float2 *)(zeros + o.mb_sk);
        d.bdf = (float2 *)(zeros + o.bdf);
        d.mt_arms = (float4 *)(zeros + o.mt_arms);
        d.mt_pk = (float2 *)(zeros + o.mt_pk);
        d.tdf = (float4 *)(zeros + o.tdf);
        d.bfrc = (double2 *)(zeros + o.bfrc);
        d.tfrc = (double4 *)(zeros + o.tfrc);
        d.fcode = (const unsigned char *)(base + o.fcode);
        d.bond = (const int4 *)(base + o.bond);
        d.bond_l0 = (const double *)(base + o.bond_l0);
        d.bond_k = o.has_bond_k ? (const double *)(base + o.bond_k) : nullptr;
        d.tri = (const int4 *)(base + o.tri);
        d.tri_kb = o.has_tri_kb ? (const double *)(base + o.tri_kb) : nullptr;
        d.tri_phi0 = o.has_tri_phi0 ? (const double *)(base + o.tri_phi0) : nullptr;
        d.bptr = (const int *)(base + o.bptr);
        d.bent = (const int *)(base + o.bent);
        d.tptr = (const int *)(base + o.tptr);
        d.tent = (const int *)(base + o.tent);
        d.part = (double *)(zeros + o.part);
        d.epart = (double *)(zeros + o.epart);
        d.st = S.st + i;
        d.n_elems = h.n_facets();
        d.use_gel = 0;
        d.gel = (const NetGel *)(base + gel_off) + i;
        NetGel &g = S.gel[i];
        g.elem = (const int4 *)(base + o.elem);
        g.elem_inv = (double *)(zeros + o.elem_inv);
        g.elem_area = (const double *)(base + o.elem_area);
        g.efrc = (double4 *)(zeros + o.efrc);
        g.eptr = (const int *)(base + o.eptr);
        g.eent = (const int *)(base + o.eent);
        g.partner = (const int *)(base + o.partner);
    }
    S.gel_array = (NetGel *)(base + gel_off);
    memcpy(img.data() + gel_off, S.gel.data(), sizeof(NetGel) * n);
    for (int i = 0; i < n; ++i) {
        const NetOff &o = off[i];
        NetDsm &m = S.dsm[i];
        m.bref = (const int2 *)(base + o.dsm_bref);
        m.bidx = (const int *)(base + o.dsm_bidx);
        m.tref = (const int4 *)(base + o.dsm_tref);
        m.bent = (const int *)(base + o.dsm_bent);
        m.tent = (const int *)(base + o.dsm_tent);
        m.grec = (const int4 *)(base + o.dsm_grec);
        m.xrec = o.has_dsm_quads ? (const int4 *)(base + o.dsm_xrec) : nullptr;
        m.xent = (uint4 *)(zeros + o.dsm_xent);
    }
    S.dsm_array = (NetDsm *)(base + dsm_off);
    memcpy(img.data() + dsm_off, S.dsm.data(), sizeof(NetDsm) * n);
    memcpy(img.data() + dev_off, S.dev.data(), sizeof(NetDev) * n);
    NR_CUDA_TRY(cudaMemcpyAsync(S.arena, img.data(), img.size(), cudaMemcpyHostToDevice, stream));
    NR_CUDA_TRY(cudaMemsetAsync(zeros, 0, img.zeros_size(), stream));
    /* get_inv_mats on the positions as uploaded (network_mesh_relax.cu:1250
     * runs it before dilate) */
    for (int i = 0; i < n; ++i)
        NR_CUDA_TRY(launch_inv_mats((const double *)S.dev[i].x, (const int *)S.gel[i].elem, 4, S.dev[i].n_elems,
                                    S.gel[i].elem_inv, stream));
    NR_CUDA_TRY(cudaStreamSynchronize(stream));
    if (have_res) {
        Res64Dev &r = S.res;
        r.sub = res_host.sub;
        r.n_units = res_host.n_units;
        r.mode = res_host.mode;
        r.shape = res_host.shape;
        r.desc = (const Res64Desc *)(base + res_off.desc);
        r.ro = (const unsigned char *)(base + res_off.ro);
        for (int c = 0; c < 2; ++c) {
            r.vf[c] = (double2 *)(zeros + res_off.vf[c]);
            r.part[c] = (double *)(zeros + res_off.part[c]);
            r.maxp[c] = (unsigned long long *)(zeros + res_off.maxp[c]);
        }
        r.bar = (unsigned long long *)(zeros + res_off.bar);
        S.res_smem = res_host.max_smem;
        r.n_ctas = res_host.n_ctas;
    }
    if (want_tile) return build_tile_set(*nets[0], inc0, fc0.data(), S, stream);
    return NR_OK;
}
static int build_set(int n, const nr_host_network *const *nets, const double *ks, const double *kb,
                     const unsigned char *const *fcodes_in, cudaStream_t stream, DeviceSet &S) {
    return no_throw([&] { return fill_set(n, nets, ks, kb, fcodes_in, stream, S); });
}

/* Energy launch width for network d. */
static int energy_blocks(const NetDev &d, int sms) {
    const int items = std::max(d.n_edges, std::max(d.n_triples, d.n_elems));
    return std::max(1, std::min(2 * sms, (items + kTile - 1) / kTile * 2));
}

static FireParamsDev to_dev(const nr_fire_params &p) {
    FireParamsDev q;
    q.alpha0 = p.alpha0;
    q.falpha = p.falpha;
    q.dt_max = p.dt_max;
    q.finc = p.finc;
    q.fdec = p.fdec;
    q.mass = p.mass;
    q.fcut = p.fcut;
    q.nmin = p.nmin;
    q.max_steps = p.max_steps;
    q.criterion = p.criterion;
    q.precision = p.precision;
    return q;
}

static int check_params(const nr_fire_params *p) {
    if (!p) return fail(NR_ERR_INVALID, "null FIRE parameters");
    if (!(p->mass > 0) || !(p->dt_max > 0) || p->max_steps < 0 || (p->criterion != NR_CRIT_RMS && p->criterion != NR_CRIT_MAX) ||
        (p->precision != NR_FP64 && p->precision != NR_MIXED))
        return fail(NR_ERR_INVALID, "invalid FIRE parameters");
    return NR_OK;
}

static void fill_report(const FireState &st, const NetDev &d, nr_report *rep) {
    rep->rms_force = st.fmag / d.sqrt_dof;
    rep->e_stretch = st.e_stretch;
    rep->e_bend = st.e_bend;
    rep->e_gel = d.use_gel ? st.e_gel : 0.0;
    rep->max_force = st.maxf;
    rep->steps = st.step;
    rep->fp64_steps = st.fp64_steps;
    rep->reserved = 0;
    const double inv_a = d.area > 0 ? 1.0 / d.area : 0.0;
    rep->stress_xx = st.vir[0] * inv_a;
    rep->stress_yy = st.vir[1] * inv_a;
    rep->stress_xy = st.vir[2] * inv_a;
    if (st.abort_flag) rep->status = NR_ERR_TIMEOUT;
    else if (st.status != 0) rep->status = st.status;
    else rep->status = st.converged ? NR_OK : NR_NOT_CONVERGED;
}

static int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

/* Launch plan of one network relaxed by a persistent kernel: the FP64
 * cooperative grid kernel (d.sub and d.n_units set here), the FP64 cluster
 * kernel (cluster > 0) or the mixed cooperative kernel. */
struct GridPlan {
    NetDev d;
    const NetDev *d_dev; /* the network's descriptor in device memory (cluster kernel) */
    int *queue;
    int blocks, energy_blocks, cluster;
    bool mixed;
    bool tile;   /* mixed: the tiled kernel (fire_tile.cu) */
    NetTile tl;
    int tile_threads = 512;
    /* FP64 on a cluster: the distributed-shared-memory kernel (dsm64) with
     * its per-CTA maxima, else the L2 one */
    bool dsm64;
    const NetDsm *m_dev;
    int bmax, emax, tmax;
    /* FP64: the resident kernel */
    bool res;
    Res64Dev rd;
    size_t res_smem;
};

/* Per-CTA maxima of the FP64 distributed-shared-memory kernel for clusters
 * of C CTAs over the networks `subset` of S (all when null); false when the
 * set has no sub-block layout or its state does not fit shared memory. */
static bool fp64_dsm_plan(const DeviceSet &S, int C, int &bmax, int &emax, int &tmax,
                          const std::vector<int> *subset = nullptr) {
    if (!S.dsm_ok || C < 1 || C > kDsmParts) return false;
    const int spr = kDsmParts / C;
    bmax = emax = tmax = 0;
    const int count = subset ? (int)subset->size() : S.n_nets;
    for (int j = 0; j < count; ++j) {
        const int i = subset ? (*subset)[j] : j;
        const NetDsm &m = S.dsm[i];
        const NetDev &d = S.dev[i];
        if (d.use_gel) return false;
        bmax = std::max(bmax, spr * m.bsub);
        for (int r = 0; r < C; ++r) {
            if (d.use_bonds) emax = std::max(emax, m.bo[(r + 1) * spr] - m.bo[r * spr]);
            if (d.use_triples) tmax = std::max(tmax, m.to[(r + 1) * spr] - m.to[r * spr]);
        }
    }
    int active = 0;
    if (dsm64_max_active(C, std::max(bmax, 1), std::max(emax, 1), std::max(tmax, 1), &active) != cudaSuccess ||
        active < 1) {
        cudaGetLastError();
        return false;
    }
    return true;
}

/* Mixed precision, one network: up to kMixedCtaNodes nodes the whole
 * relaxation runs in one CTA with u in shared memory (no grid barriers);
 * larger networks use the cooperative kernel over the whole GPU. */
constexpr int kMixedCtaNodes = 4096;

static int fp64_cluster_ctas() {
    const char *env = knob("NR_FP64_CLUSTER");
    const int c = env ? atoi(env) : 16;
    return c == 1 || c == 2 || c == 4 || c == 8 || c == 16 ? c : 16;
}

static int grid_plan(const DeviceSet &S, int i, bool mixed, GridPlan &g) {
    g.d = S.dev[i];
    g.d_dev = S.dev_array + i;
    g.queue = S.queue;
    g.mixed = mixed;
    g.cluster = 0;
    g.tile = false;
    g.dsm64 = false;
    g.m_dev = S.dsm_array + i;
    g.bmax = g.emax = g.tmax = 0;
    g.res = false;
    const int sms = sm_count();
    const char *mk = knob("NR_MIX_KERNEL");
    if (mixed && S.tile_ctas > 0 && !(mk && strcmp(mk, "grid") == 0)) {
        g.tile = true;
        g.tl = S.tile;
        g.blocks = S.tile_ctas;
        g.tile_threads = S.tile_threads;
    } else if (mixed) {
        g.blocks = mixed_grid_blocks(g.d.n);
        if (g.blocks <= 0) return fail(NR_ERR_CUDA, "occupancy query failed");
        if ((size_t)5 * g.blocks > (size_t)4 * g.d.n_tiles * 8) return fail(NR_ERR_CAPACITY, "reduction scratch too small");
    } else {
        const int choice = fp64_kernel_choice();
        const int line = choice == kFp64Grid ? 0 : fp64_cluster_nodes();
        if (line > 0 && choice == kFp64Res && S.res.n_ctas > 0 && !(g.d.use_gel && g.d.n_elems == 0)) {
            g.res = true;
            g.rd = S.res;
            g.res_smem = S.res_smem;
            g.blocks = S.res.n_ctas;
        } else if (g.d.n <= (choice == kFp64Res ? std::min(line, kFp64DsmNodes) : line)) {
            int c = fp64_cluster_ctas(), active = 0;
            const std::vector<int> one{i};
            if (choice != kFp64L2 && fp64_dsm_plan(S, c, g.bmax, g.emax, g.tmax, &one)) {
                g.dsm64 = true;
            } else {
                while (c > 1 && (fp64_cluster_max_active(c, g.d.use_gel != 0, &active) != cudaSuccess || active < 1)) {
                    cudaGetLastError();
                    c /= 2;
                }
            }
            g.cluster = c;
            g.blocks = c;
        } else {
            int sub = 8;
            while (sub > 1 && g.d.n_tiles * (8 / sub) < sms) sub /= 2;
            g.d.sub = sub;
            g.d.n_units = g.d.n_tiles * (8 / sub);
            int max_blocks = 0;
            NR_CUDA_TRY(fp64_grid_max_blocks(sub, g.d.use_gel != 0, &max_blocks));
            g.blocks = std::max(1, std::min(g.d.n_units, max_blocks));
        }
    }
    g.energy_blocks = energy_blocks(g.d, sms);
    return NR_OK;
}

/* Enqueues one relaxation without waiting for it: the FIRE state zeroed,
 * the persistent kernel, the energies.  Only stream work, so a stream
 * capture records it into a graph. */
static int enqueue_grid(const GridPlan &g, const nr_fire_params &prm, cudaStream_t stream) {
    NR_CUDA_TRY(cudaMemsetAsync(g.d.st, 0, sizeof(FireState), stream));
    if (g.tile)
        NR_CUDA_TRY(
            launch_mixed_tile(g.d, g.tl, to_dev(prm), g.blocks, g.tile_threads, barrier_budget_ns(), stream));
    else if (g.mixed) NR_CUDA_TRY(launch_mixed_grid(g.d, to_dev(prm), g.blocks, barrier_budget_ns(), stream));
    else if (g.res)
        NR_CUDA_TRY(launch_fp64_res(g.d, g.rd, to_dev(prm), g.res_smem, barrier_budget_ns(), stream));
    else if (g.cluster > 0) {
        /* the cluster kernels take their energies themselves */
        if (g.dsm64)
            NR_CUDA_TRY(launch_fp64_dsm(g.d_dev, g.m_dev, 1, g.cluster, g.bmax, g.emax, g.tmax, to_dev(prm), g.queue,
                                        nullptr, stream));
        else
            NR_CUDA_TRY(launch_fp64_cluster(g.d_dev, 1, g.cluster, g.d.use_gel != 0, to_dev(prm), g.queue, nullptr,
                                            stream));
        return NR_OK;
    } else NR_CUDA_TRY(launch_fp64_grid(g.d, to_dev(prm), g.blocks, barrier_budget_ns(), barrier_stall(), stream));
    NR_CUDA_TRY(launch_energies(g.d, g.energy_blocks, stream));
    return NR_OK;
}

/* The report of a finished relaxation and its status (errors recorded). */
static int report_status(const FireState &st, const NetDev &d, nr_report *rep) {
    fill_report(st, d, rep);
    if (rep->status == NR_ERR_TIMEOUT) return fail(NR_ERR_TIMEOUT, "grid barrier wait budget exceeded");
    if (rep->status < 0) return fail(rep->status, "relaxation produced non-finite forces");
    return rep->status;
}

static int relax_grid(const GridPlan &g, const nr_fire_params &prm, cudaStream_t stream, nr_report *rep) {
    int rc = enqueue_grid(g, prm, stream);
    if (rc != NR_OK) return rc;
    FireState st;
    NR_CUDA_TRY(cudaMemcpyAsync(&st, g.d.st, sizeof(FireState), cudaMemcpyDeviceToHost, stream));
    NR_CUDA_TRY(cudaStreamSynchronize(stream));
    return report_status(st, g.d, rep);
}

/* One network over the whole GPU (FP64 cooperative kernel + energies). */
static int relax_single_fp64(DeviceSet &S, int i, const nr_fire_params &prm, cudaStream_t stream, nr_report *rep) {
    GridPlan g;
    int rc = grid_plan(S, i, false, g);
    if (rc != NR_OK) return rc;
    return relax_grid(g, prm, stream, rep);
}

static int relax_set_batch(DeviceSet &S, const nr_fire_params &prm, cudaStream_t stream, nr_report *reps);

static int relax_single_mixed(DeviceSet &S, const nr_fire_params &prm, cudaStream_t stream, nr_report *rep) {
    if (S.dev[0].n <= kMixedCtaNodes) return relax_set_batch(S, prm, stream, rep);
    GridPlan g;
    int rc = grid_plan(S, 0, true, g);
    if (rc != NR_OK) return rc;
    return relax_grid(g, prm, stream, rep);
}

/* Launch plan of the distributed-shared-memory kernel: cluster size and
 * per-CTA maxima (nodes, bonds, triples, incidence entries). */
struct DsmPlan {
    int C, bmax, emax, tmax, ebmax, etmax, resident;
};

/* `forced` C if nonzero, else the smallest C >= `least` (a power of two
 * dividing 16) whose per-CTA state fits in shared memory; the read-only
 * slices go to shared memory as well when they fit too (NR_DSM_RESIDENT=0
 * keeps them in global memory).  False when the batch has no layout,
 * NR_MIX_KERNEL=l2 asks for the global-memory kernels, or nothing fits. */
static bool dsm_plan(const DeviceSet &S, int forced, int least, DsmPlan &pl, const std::vector<int> *subset = nullptr) {
    const char *k = knob("NR_MIX_KERNEL");
    if (!S.dsm_ok || (k && strcmp(k, "l2") == 0)) return false;
    const char *rk = knob("NR_DSM_RESIDENT");
    const bool allow_res = !(rk && atoi(rk) == 0);
    const size_t limit = dsm_smem_limit();
    for (int C = 1; C <= kDsmParts; C *= 2) {
        if (forced ? C != forced : C < least) continue;
        const int spr = kDsmParts / C;
        int bm = 0, em = 0, tm = 0, ebm = 0, etm = 0;
        const int count = subset ? (int)subset->size() : S.n_nets;
        for (int j = 0; j < count; ++j) {
            const int i = subset ? (*subset)[j] : j;
            const NetDsm &m = S.dsm[i];
            const NetDev &d = S.dev[i];
            if (!m.xrec) return false;
            bm = std::max(bm, spr * m.bsub);
            for (int r = 0; r < C; ++r) {
                if (d.use_bonds) {
                    em = std::max(em, m.bo[(r + 1) * spr] - m.bo[r * spr]);
                    ebm = std::max(ebm, m.be[(r + 1) * spr] - m.be[r * spr]);
                }
                if (d.use_triples) {
                    tm = std::max(tm, m.to[(r + 1) * spr] - m.to[r * spr]);
                    etm = std::max(etm, m.te[(r + 1) * spr] - m.te[r * spr]);
                }
            }
        }
        int res = -1;
        if (allow_res && dsm_smem_bytes(bm, em, tm, ebm, etm, 1) <= limit) res = 1;
        else if (dsm_smem_bytes(bm, em, tm, ebm, etm, 0) <= limit) res = 0;
        if (res >= 0) {
            pl = DsmPlan{C, bm, em, tm, ebm, etm, res};
            return true;
        }
    }
    return false;
}

/* Fraction of idle clusters at which running networks escalate to clusters
 * twice as large: NR_ESCALATE (default 0.25; 0 disables). */
static double escalate_fraction() {
    const char *env = knob("NR_ESCALATE");
    const double f = env ? atof(env) : 0.25;
    return f > 0 && f <= 1 ? f : 0.0;
}

/* The distributed-shared-memory kernel in phases: all networks on clusters
 * of C CTAs; when a fraction of the clusters has gone idle (the queue is
 * empty), the networks still running stop at an anchor and the next phase
 * resumes them on clusters twice as large, up to 16 CTAs.  The soft
 * networks that need 10^5-10^6 steps thus end on the widest clusters
 * instead of holding the whole batch on 4 SMs each. */
/* Networks of at most this many nodes run one per CTA beside the clusters
 * in the first phase (NR_SOLO_NODES; 0 disables). */
static int solo_nodes() {
    const char *env = knob("NR_SOLO_NODES");
    return env ? std::max(0, atoi(env)) : 2304;
}

/* First-phase split of a size-ordered batch: the small networks (a suffix
 * of the order) relax one per CTA on a second stream while the others
 * relax on clusters.  A CTA handles a small network with 1.3-1.6x the
 * throughput per SM of a cluster (no cluster barriers), and the single
 * CTAs also use the SMs that clusters of C cannot tile.  SMs are divided by
 * node count, the single CTAs' share weighted by that throughput gain.
 * Returns the number of small networks (0: no split) and their plan. */
static int solo_split(const DeviceSet &S, const DsmPlan &pl, DsmPlan &ps, int &cap_clusters) {
    const int limit = solo_nodes();
    if (pl.C < 2 || limit <= 0 || S.n_nets < 2) return 0;
    std::vector<int> small;
    for (int k = S.n_nets - 1; k >= 0 && S.dev[S.order_host[k]].n <= limit; --k) small.push_back(S.order_host[k]);
    if (small.empty() || (int)small.size() == S.n_nets) return 0;
    if (!dsm_plan(S, 1, 0, ps, &small)) return 0;
    int maxa = 0, dev = 0, sms = 0;
    if (dsm_max_active(pl.C, pl.bmax, pl.emax, pl.tmax, pl.ebmax, pl.etmax, pl.resident, &maxa) != cudaSuccess ||
        maxa < 2)
        return 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    double n_small = 0, n_all = 0;
    for (int i = 0; i < S.n_nets; ++i) n_all += S.dev[i].n;
    for (int i : small) n_small += S.dev[i].n;
    const int want = (int)std::lround(0.6 * sms * n_small / n_all);
    cap_clusters = std::max(1, std::min(maxa, (sms - want) / pl.C));
    return (int)small.size();
}

/* CTAs of the single-CTA launch beside `cap_clusters` clusters of C: the
 * SMs the clusters leave (NR_SOLO_CTAS; 0: one per SM, oversubscribed),
 * so that both launches are resident together from the start and the
 * placement of the clusters does not depend on which launch the hardware
 * schedules first. */
static int solo_ctas(int cap_clusters, int C) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const char *env = knob("NR_SOLO_CTAS");
    if (env) return std::max(0, atoi(env));
    return std::max(1, sms - cap_clusters * C);
}

/* The stream and events of a launch beside the caller's. */
static int side_stream(DeviceSet &S) {
    if (!S.side) {
        NR_CUDA_TRY(cudaStreamCreateWithFlags(&S.side, cudaStreamNonBlocking));
        NR_CUDA_TRY(cudaEventCreateWithFlags(&S.ev_fork, cudaEventDisableTiming));
        NR_CUDA_TRY(cudaEventCreateWithFlags(&S.ev_join, cudaEventDisableTiming));
    }
    return NR_OK;
}

static int relax_dsm_phases(DeviceSet &S, const nr_fire_params &prm, DsmPlan pl, cudaStream_t stream,
                            bool capture = false) {
    /* one network never finds others idle */
    const double frac = S.n_nets > 1 ? escalate_fraction() : 0.0;
    int n_run = S.n_nets;
    const int *order_dev = S.order;
    std::vector<FireState> st;
    std::vector<int> next;
    DsmPlan ps;
    int cap = 0;
    const int n_small = solo_split(S, pl, ps, cap);
    if (n_small > 0) {
        const int rc = side_stream(S);
        if (rc != NR_OK) return rc;
        n_run = S.n_nets - n_small;
    }
    /* Device-side escalation (the default; NR_ESCALATE_HOST=1 steers from
     * the host instead): every later phase is planned now for the whole
     * batch, and a compaction kernel lists the networks that yielded, so the
     * relaxation is stream work only, with no host round trip between
     * phases, and a stream capture records it into a graph.  A phase whose
     * list is empty launches clusters that exit at once. */
    std::vector<DsmPlan> later;
    const char *eh = knob("NR_ESCALATE_HOST");
    bool device_side = frac > 0 && !(eh && atoi(eh) != 0);
    for (int C = 2 * pl.C; device_side && C <= kDsmParts; C *= 2) {
        DsmPlan p2;
        if (!dsm_plan(S, C, 0, p2)) device_side = false;
        else later.push_back(p2);
    }
    if (device_side) {
        if (n_small > 0) NR_CUDA_TRY(cudaEventRecord(S.ev_fork, stream));
        NR_CUDA_TRY(launch_mixed_dsm(S.dev_array, S.dsm_array, n_run, pl.C, pl.bmax, pl.emax, pl.tmax, pl.ebmax,
                                     pl.etmax, pl.resident, later.empty() ? 0.0 : frac, cap, to_dev(prm), S.queue,
                                     order_dev, stream));
        S.launches++;
        if (n_small > 0) {
            NR_CUDA_TRY(cudaStreamWaitEvent(S.side, S.ev_fork, 0));
            NR_CUDA_TRY(launch_mixed_dsm(S.dev_array, S.dsm_array, n_small, 1, ps.bmax, ps.emax, ps.tmax, ps.ebmax,
                                         ps.etmax, ps.resident, later.empty() ? 0.0 : frac, solo_ctas(cap, pl.C),
                                         to_dev(prm), S.queue + 4, S.order + (S.n_nets - n_small), S.side));
            S.launches++;
            NR_CUDA_TRY(cudaEventRecord(S.ev_join, S.side));
            NR_CUDA_TRY(cudaStreamWaitEvent(stream, S.ev_join, 0));
        }
        for (size_t k = 0; k < later.size(); ++k) {
            const DsmPlan &p2 = later[k];
            const bool last = k + 1 == later.size();
            NR_CUDA_TRY(launch_compact_yielded(S.st, S.n_nets, S.order2, S.queue + 8, stream));
            NR_CUDA_TRY(launch_mixed_dsm(S.dev_array, S.dsm_array, S.n_nets, p2.C, p2.bmax, p2.emax, p2.tmax, p2.ebmax,
                                         p2.etmax, p2.resident, last ? 0.0 : frac, 0, to_dev(prm), S.queue, S.order2,
                                         stream, S.queue + 8));
            S.launches += 2;
        }
        return NR_OK;
    }
    if (capture && frac > 0 && pl.C < kDsmParts)
        return fail(NR_ERR_INVALID, "batch relaxation: escalation steered from the host (NR_ESCALATE_HOST, or no "
                                    "plan for the larger clusters) cannot be recorded in a graph");
    for (int phase = 0;; ++phase) {
        const bool last = pl.C >= kDsmParts || frac <= 0;
        /* the side stream starts after the work queued so far, not after
         * the cluster launch below: the two kernels run concurrently */
        if (phase == 0 && n_small > 0) NR_CUDA_TRY(cudaEventRecord(S.ev_fork, stream));
        NR_CUDA_TRY(launch_mixed_dsm(S.dev_array, S.dsm_array, n_run, pl.C, pl.bmax, pl.emax, pl.tmax, pl.ebmax,
                                     pl.etmax, pl.resident, last ? 0.0 : frac, phase == 0 ? cap : 0, to_dev(prm),
                                     S.queue, order_dev, stream));
        S.launches++;
        if (phase == 0 && n_small > 0) {
            /* the small networks (the order's suffix) on single CTAs, on
             * the side stream, with their own queue counters */
            NR_CUDA_TRY(cudaStreamWaitEvent(S.side, S.ev_fork, 0));
            NR_CUDA_TRY(launch_mixed_dsm(S.dev_array, S.dsm_array, n_small, 1, ps.bmax, ps.emax, ps.tmax, ps.ebmax,
                                         ps.etmax, ps.resident, last ? 0.0 : frac, solo_ctas(cap, pl.C),
                                         to_dev(prm), S.queue + 4, S.order + (S.n_nets - n_small), S.side));
            S.launches++;
            NR_CUDA_TRY(cudaEventRecord(S.ev_join, S.side));
            NR_CUDA_TRY(cudaStreamWaitEvent(stream, S.ev_join, 0));
        }
        if (last) return NR_OK;
        st.resize(S.n_nets);
        NR_CUDA_TRY(cudaMemcpyAsync(st.data(), S.st, sizeof(FireState) * S.n_nets, cudaMemcpyDeviceToHost, stream));
        NR_CUDA_TRY(cudaStreamSynchronize(stream));
        next.clear();
        for (int i = 0; i < S.n_nets; ++i)
            if (st[i].yielded) next.push_back(i);
        if (next.empty()) return NR_OK;
        DsmPlan p2;
        if (!dsm_plan(S, 2 * pl.C, 0, p2, &next)) return fail(NR_ERR_CUDA, "escalation: no cluster plan");
        NR_CUDA_TRY(cudaMemcpyAsync(S.order2, next.data(), sizeof(int) * next.size(), cudaMemcpyHostToDevice, stream));
        n_run = (int)next.size();
        order_dev = S.order2;
        pl = p2;
    }
}

/* CTAs per network of an FP64 batch: NR_FP64_BATCH_CLUSTER, else one CTA
 * per network (k_fire_batch) when every network has at most 2304 nodes and
 * clusters of 8 otherwise.  FP64 is the bound of the plain path (1/64 of
 * the FP32 rate on GB300), so the batch's throughput does not depend on the
 * team size, but its makespan is one soft network's 10^5-10^6 steps on its
 * team: a wider team finishes it sooner. */
static int fp64_batch_cluster(int max_nodes) {
    const char *env = knob("NR_FP64_BATCH_CLUSTER");
    if (env) {
        const int c = atoi(env);
        return c == 2 || c == 4 || c == 8 || c == 16 ? c : 1;
    }
    return max_nodes <= 2304 ? 1 : 8;
}

/* The narrow teams beside an FP64 batch's wide ones.  Clusters of 16 leave SMs
 * idle (14 of them, two CTAs an SM, take 112 of 152: a cluster stays within a
 * part of the chip), and a team's step costs about 11 us however small its
 * network.  So teams of 4 on the idle SMs work from the small end of the order
 * while two networks are left for every wide team: a step of theirs takes up to
 * twice as long, and the batch must not end with their last network.  FP64
 * results do not depend on the team.  100 steps of 64 lattices of 16^2 to 96^2
 * nodes 10.8 -> 9.5 ms, of 100 of 8^2 to 40^2 10.1 -> 8.0; run to convergence (up
 * to 20 000 steps), 64 of 16^2 to 48^2 776 -> 672 ms, 40 of 24^2 to 64^2 675 ->
 * 672 (892 with narrow teams until the end). */
struct Fp64Back {
    int n = 0, leave = 0, clusters = 0; /* networks they may take (the order's last), those left alone, teams */
    int bmax = 0, emax = 0, tmax = 0;
};
constexpr int kFp64BackTeam = 4;
static Fp64Back fp64_back(const DeviceSet &S, int C, int bmax, int emax, int tmax) {
    Fp64Back b;
    int dev = 0, sms = 0, per_sm = 0, wide = 0;
    if (C <= kFp64BackTeam || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        dsm64_max_active(C, bmax, emax, tmax, &wide) != cudaSuccess) {
        cudaGetLastError();
        return b;
    }
    b.leave = 2 * wide;
    if (S.n_nets - wide <= b.leave) return b;
    const size_t half = (size_t)per_sm / 2 - 1024; /* two CTAs an SM, 1 KB of each reserved */
    const int used = dsm64_cta_bytes(bmax, emax, tmax) <= half ? (wide * C + 1) / 2 : wide * C;
    b.clusters = std::max(0, sms - used) * 2 / kFp64BackTeam;
    const int spr = kDsmParts / kFp64BackTeam;
    for (int k = S.n_nets - 1; k >= 0 && b.clusters > 0; --k) { /* the order's suffix that fits half an SM a CTA */
        const int i = S.order_host[k];
        const NetDsm &m = S.dsm[i];
        Fp64Back t = b;
        t.bmax = std::max(t.bmax, spr * m.bsub);
        for (int r = 0; r < kFp64BackTeam; ++r) {
            if (S.dev[i].use_bonds) t.emax = std::max(t.emax, m.bo[(r + 1) * spr] - m.bo[r * spr]);
            if (S.dev[i].use_triples) t.tmax = std::max(t.tmax, m.to[(r + 1) * spr] - m.to[r * spr]);
        }
        if (dsm64_cta_bytes(t.bmax, t.emax, t.tmax) > half) break;
        t.n = b.n + 1;
        b = t;
    }
    return b;
}

/* Enqueues one relaxation of every network of S (FIRE states zeroed, the
 * kernels) without waiting for it.  capture: stream work only, as a stream
 * capture needs (fails when escalation would be steered from the host). */
static int enqueue_set_batch(DeviceSet &S, const nr_fire_params &prm, cudaStream_t stream, bool capture) {
    NR_CUDA_TRY(cudaMemsetAsync(S.st, 0, sizeof(FireState) * S.n_nets, stream));
    S.launches = 0;
    if (prm.precision == NR_MIXED) {
        const char *env = knob("NR_CLUSTER");
        const int cluster = env ? std::max(1, std::min(16, atoi(env))) : mixed_cluster_size(S.max_nodes);
        DsmPlan pl;
        if (dsm_plan(S, env ? cluster : 0, cluster, pl)) {
            const int st = relax_dsm_phases(S, prm, pl, stream, capture);
            if (st != NR_OK) return st;
        } else if (cluster > 1) {
            NR_CUDA_TRY(launch_mixed_cluster(S.dev_array, S.n_nets, cluster, to_dev(prm), S.queue, S.order, stream));
            S.launches++;
        } else {
            NR_CUDA_TRY(
                launch_mixed_batch(S.dev_array, S.n_nets, S.max_nodes, to_dev(prm), S.queue, S.order, stream));
            S.launches++;
        }
    } else {
        const int c = fp64_batch_cluster(S.max_nodes);
        int bmax = 0, emax = 0, tmax = 0;
        if (c > 1 && fp64_kernel_choice() <= kFp64Dsm && fp64_dsm_plan(S, c, bmax, emax, tmax)) {
            const Fp64Back b = fp64_back(S, c, bmax, emax, tmax);
            if (b.n > 0) {
                const int st = side_stream(S);
                if (st != NR_OK) return st;
            }
            NR_CUDA_TRY(cudaMemsetAsync(S.queue, 0, 16, stream));
            if (b.n > 0) NR_CUDA_TRY(cudaEventRecord(S.ev_fork, stream));
            NR_CUDA_TRY(launch_fp64_dsm(S.dev_array, S.dsm_array, S.n_nets, c, bmax, emax, tmax, to_dev(prm), S.queue,
                                        S.order, stream, false));
            if (b.n > 0) {
                NR_CUDA_TRY(cudaStreamWaitEvent(S.side, S.ev_fork, 0));
                NR_CUDA_TRY(launch_fp64_dsm(S.dev_array, S.dsm_array, S.n_nets, kFp64BackTeam, b.bmax, b.emax, b.tmax,
                                            to_dev(prm), S.queue, S.order, S.side, false, b.n, b.leave, b.clusters));
                S.launches++;
                NR_CUDA_TRY(cudaEventRecord(S.ev_join, S.side));
                NR_CUDA_TRY(cudaStreamWaitEvent(stream, S.ev_join, 0));
            }
        } else if (c > 1) {
            NR_CUDA_TRY(launch_fp64_cluster(S.dev_array, S.n_nets, c, false, to_dev(prm), S.queue, S.order, stream));
        } else {
            int max_blocks = 0;
            NR_CUDA_TRY(fp64_batch_max_blocks(&max_blocks));
            const int blocks = std::max(1, std::min(S.n_nets, max_blocks));
            NR_CUDA_TRY(launch_fp64_batch(S.dev_array, S.n_nets, to_dev(prm), S.queue, blocks, stream));
        }
        S.launches++;
    }
    return NR_OK;
}

/* Reports of n networks from their FIRE states; the worst status. */
static int reports_of(const DeviceSet &S, const FireState *st, nr_report *reps) {
    int worst = NR_OK;
    for (int i = 0; i < S.n_nets; ++i) {
        fill_report(st[i], S.dev[i], &reps[i]);
        if (reps[i].status < 0) worst = reps[i].status;
        else if (worst == NR_OK && reps[i].status == NR_NOT_CONVERGED) worst = NR_NOT_CONVERGED;
    }
    return worst;
}

static int relax_set_batch(DeviceSet &S, const nr_fire_params &prm, cudaStream_t stream, nr_report *reps) {
    int rc = enqueue_set_batch(S, prm, stream, false);
    if (rc != NR_OK) return rc;
    std::vector<FireState> st(S.n_nets);
    NR_CUDA_TRY(cudaMemcpyAsync(st.data(), S.st, sizeof(FireState) * S.n_nets, cudaMemcpyDeviceToHost, stream));
    NR_CUDA_TRY(cudaStreamSynchronize(stream));
    const int worst = reports_of(S, st.data(), reps);
    if (worst < 0) return fail(worst, "a network in the batch failed");
    return worst;
}

/* Gel arrays of network_mesh_relax.cu's run_fire_md (device pointers). */
struct GelArgs {
    int nelems, n_mpairs;
    double smod, bmod, dilation;
    const int *d_elems;
    const double *d_areas, *d_inv_mats;
    const int *d_mpairs;
};

/* Moduli and preferred dilation of network 0 of S; the gel acts when
 * bmod > 0 (network_mesh_relax.cu:908). */
static int set_gel(DeviceSet &S, double smod, double bmod, double dilation) {
    NetDev &dv = S.dev[0];
    NetGel &g = S.gel[0];
    if (bmod > 0 && !S.gel_ok[0])
        return fail(NR_ERR_INVALID, "gel coupling: a vertex is in more than one duplicate pair (or paired with itself)");
    g.smod = smod;
    g.bmod = bmod;
    g.gdil = dilation;
    dv.use_gel = bmod > 0;
    NR_CUDA_TRY(cudaMemcpy(S.gel_array, &g, sizeof(NetGel), cudaMemcpyHostToDevice));
    NR_CUDA_TRY(cudaMemcpy(S.dev_array, &dv, sizeof(NetDev), cudaMemcpyHostToDevice));
    return NR_OK;
}

/* Checksum of the drop-in's read-only device arrays: every element's bits
 * mixed with its position and its array's tag (SplitMix64's finaliser),
 * summed modulo 2^64 with integer atomics (an order-independent, hence
 * deterministic, total). */
struct DropinArrays {
    const int *pairs;
    const double *lengths;
    const signed char *e_off;
    const int *triples;
    const signed char *t_off;
    const unsigned char *fcodes;
    const int *elems;
    const double *areas;
    const int *mpairs;
    long n[9]; /* element counts, in the order above */
};

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

__global__ void k_dropin_hash(DropinArrays a, long total, unsigned long long *out) {
    unsigned long long acc = 0;
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < total; g += (long)gridDim.x * blockDim.x) {
        long k = g;
        int arr = 0;
        while (k >= a.n[arr]) k -= a.n[arr++];
        unsigned long long v;
        switch (arr) {
        case 0: v = (unsigned)a.pairs[k]; break;
        case 1: v = (unsigned long long)__double_as_longlong(a.lengths[k]); break;
        case 2: v = (unsigned char)a.e_off[k]; break;
        case 3: v = (unsigned)a.triples[k]; break;
        case 4: v = (unsigned char)a.t_off[k]; break;
        case 5: v = a.fcodes[k]; break;
        case 6: v = (unsigned)a.elems[k]; break;
        case 7: v = (unsigned long long)__double_as_longlong(a.areas[k]); break;
        default: v = (unsigned)a.mpairs[k]; break;
        }
        acc += mix64(v ^ mix64((unsigned long long)k * 0x9E3779B97F4A7C15ULL + (unsigned long long)arr));
    }
    for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(kFull, acc, off);
    if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

/* The device image the last drop-in call on this host thread built, and
 * what it was built from: reused while the caller passes the same device
 * arrays with the same sizes, constants and contents (checksum), so a strain
 * sweep that calls run_fire_md once per step (large_strain_relax.cu:931,
 * :973) pays the topology copies, checks and incidence build once. */
struct DropinCache {
    std::unique_ptr<DeviceSet> set;
    int device = -1;
    DropinArrays arrays{};
    int num_dof = 0, use_gel = 0;
    double width = 0, ks = 0, kb = 0;
    unsigned long long hash = 0;
    unsigned long long *d_hash = nullptr; /* 8 bytes of device scratch */
    ~DropinCache() {
        if (d_hash) cudaFree(d_hash);
    }
};
static thread_local DropinCache t_dropin;

/* NR_DROPIN_CACHE=0 rebuilds the device image on every drop-in call. */
static bool dropin_cache_enabled() {
    const char *env = getenv("NR_DROPIN_CACHE");
    return !(env && atoi(env) == 0);
}

static int dropin_hash(const DropinArrays &a, cudaStream_t s, unsigned long long *out) {
    DropinCache &c = t_dropin;
    if (!c.d_hash) NR_CUDA_TRY(cudaMalloc(&c.d_hash, sizeof(unsigned long long)));
    long total = 0;
    for (long v : a.n) total += v;
    NR_CUDA_TRY(cudaMemsetAsync(c.d_hash, 0, sizeof(unsigned long long), s));
    const int blocks = (int)std::max(1L, std::min(2L * sm_count(), (total + 255) / 256));
    k_dropin_hash<<<blocks, 256, 0, s>>>(a, total, c.d_hash);
    NR_CUDA_TRY(cudaGetLastError());
    NR_CUDA_TRY(cudaMemcpyAsync(out, c.d_hash, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    NR_CUDA_TRY(cudaStreamSynchronize(s));
    return NR_OK;
}

/* run_fire_md of large_strain_relax.cu:596 (gel == nullptr) or of
 * network_mesh_relax.cu:865: the caller's device arrays are copied into a
 * device image of the network (or the cached image is reused, see
 * DropinCache), relaxed by the FP64 path with the RMS criterion, and
 * positions, velocities and forces copied back.  report_data: {RMS F, E_s,
 * E_b, E_gel}. */
static int run_fire_md_impl(const char *who, int num_dof, int npairs, int ntriples, double width, double ks, double kb,
                            double *d_pos, double *d_vel, double *d_forces, const int *d_pair_list,
                            const double *d_lengths, const signed char *d_e_offsets, const int *d_triples,
                            const signed char *d_t_offsets, const unsigned char *d_fcodes,
                            const double fire_params[5], double mass, double fcut, int max_steps, int nmin,
                            const GelArgs *gel, double report_data[4], int *step_count, void *stream) {
    const bool use_gel = gel && gel->bmod > 0;
    if (num_dof <= 0 || (num_dof & 1) || npairs < 0 || ntriples < 0 || !d_pos || !d_fcodes || !fire_params ||
        !report_data || !step_count || (npairs > 0 && ks > 0 && (!d_pair_list || !d_lengths || !d_e_offsets)) ||
        (ntriples > 0 && kb > 0 && (!d_triples || !d_t_offsets)) ||
        (use_gel && (gel->nelems < 0 || gel->n_mpairs < 0 ||
                     (gel->nelems > 0 && (!gel->d_elems || !gel->d_areas || !gel->d_inv_mats)) ||
                     (gel->n_mpairs > 0 && !gel->d_mpairs))))
        return fail(NR_ERR_INVALID, std::string(who) + ": bad arguments");
    nr_fire_params p;
    p.alpha0 = fire_params[0];
    p.falpha = fire_params[1];
    p.dt_max = fire_params[2];
    p.finc = fire_params[3];
    p.fdec = fire_params[4];
    p.nmin = nmin;
    p.mass = mass;
    p.fcut = fcut;
    p.max_steps = max_steps;
    p.criterion = NR_CRIT_RMS;
    p.precision = NR_FP64;
    int rc = check_params(&p);
    if (rc != NR_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const int n = num_dof / 2;
    /* the arrays the relaxation reads, as used (a term off means its arrays
     * are not read) */
    const bool bonds = ks > 0 && npairs > 0, tris = kb > 0 && ntriples > 0;
    DropinArrays arr{};
    arr.pairs = bonds ? d_pair_list : nullptr;
    arr.lengths = bonds ? d_lengths : nullptr;
    arr.e_off = bonds ? d_e_offsets : nullptr;
    arr.triples = tris ? d_triples : nullptr;
    arr.t_off = tris ? d_t_offsets : nullptr;
    arr.fcodes = d_fcodes;
    arr.elems = use_gel && gel->nelems > 0 ? gel->d_elems : nullptr;
    arr.areas = use_gel && gel->nelems > 0 ? gel->d_areas : nullptr;
    arr.mpairs = use_gel && gel->n_mpairs > 0 ? gel->d_mpairs : nullptr;
    const long counts[9] = {bonds ? 2L * npairs : 0, bonds ? npairs : 0, bonds ? npairs : 0, tris ? 3L * ntriples : 0,
                            tris ? 2L * ntriples : 0, n, arr.elems ? 3L * gel->nelems : 0,
                            arr.elems ? (long)gel->nelems : 0, arr.mpairs ? 2L * gel->n_mpairs : 0};
    memcpy(arr.n, counts, sizeof(counts));
    int device = 0;
    NR_CUDA_TRY(cudaGetDevice(&device));
    DropinCache &cache = t_dropin;
    const bool caching = dropin_cache_enabled();
    unsigned long long hash = 0;
    bool hit = false;
    if (caching && cache.set && cache.device == device && cache.num_dof == num_dof && cache.use_gel == (int)use_gel &&
        cache.width == width && cache.ks == ks && cache.kb == kb && memcmp(&cache.arrays, &arr, sizeof(arr)) == 0) {
        rc = dropin_hash(arr, s, &hash);
        if (rc != NR_OK) return rc;
        hit = hash == cache.hash;
    }
    if (!hit) {
        cache.set.reset();
        nr_host_network h;
        h.n_points = n;
        h.offset = width;
        h.points.resize(num_dof);
        NR_CUDA_TRY(cudaMemcpyAsync(h.points.data(), d_pos, sizeof(double) * num_dof, cudaMemcpyDeviceToHost, s));
        std::vector<unsigned char> fc(n);
        NR_CUDA_TRY(cudaMemcpyAsync(fc.data(), d_fcodes, n, cudaMemcpyDeviceToHost, s));
        if (bonds) {
            h.edge_ij.resize(2 * (size_t)npairs);
            h.edge_l0.resize(npairs);
            h.edge_wrap.resize(npairs);
            NR_CUDA_TRY(cudaMemcpyAsync(h.edge_ij.data(), d_pair_list, sizeof(int) * 2 * npairs, cudaMemcpyDeviceToHost, s));
            NR_CUDA_TRY(cudaMemcpyAsync(h.edge_l0.data(), d_lengths, sizeof(double) * npairs, cudaMemcpyDeviceToHost, s));
            NR_CUDA_TRY(cudaMemcpyAsync(h.edge_wrap.data(), d_e_offsets, npairs, cudaMemcpyDeviceToHost, s));
        }
        if (tris) {
            h.tri_hjk.resize(3 * (size_t)ntriples);
            h.tri_wrap.resize(2 * (size_t)ntriples);
            NR_CUDA_TRY(cudaMemcpyAsync(h.tri_hjk.data(), d_triples, sizeof(int) * 3 * ntriples, cudaMemcpyDeviceToHost, s));
            NR_CUDA_TRY(cudaMemcpyAsync(h.tri_wrap.data(), d_t_offsets, 2 * (size_t)ntriples, cudaMemcpyDeviceToHost, s));
        }
        if (use_gel) {
            h.facets.resize(3 * (size_t)gel->nelems);
            h.areas.resize(gel->nelems);
            h.mesh_pairs.resize(2 * (size_t)gel->n_mpairs);
            if (gel->nelems > 0) {
                NR_CUDA_TRY(cudaMemcpyAsync(h.facets.data(), gel->d_elems, sizeof(int) * 3 * (size_t)gel->nelems,
                                            cudaMemcpyDeviceToHost, s));
                NR_CUDA_TRY(cudaMemcpyAsync(h.areas.data(), gel->d_areas, sizeof(double) * gel->nelems,
                                            cudaMemcpyDeviceToHost, s));
            }
            if (gel->n_mpairs > 0)
                NR_CUDA_TRY(cudaMemcpyAsync(h.mesh_pairs.data(), gel->d_mpairs, sizeof(int) * 2 * (size_t)gel->n_mpairs,
                                            cudaMemcpyDeviceToHost, s));
        }
        NR_CUDA_TRY(cudaStreamSynchronize(s));
        for (size_t i = 0; i < h.edge_ij.size(); ++i)
            if (h.edge_ij[i] < 0 || h.edge_ij[i] >= n) return fail(NR_ERR_INVALID, std::string(who) + ": bond index out of range");
        for (size_t i = 0; i < h.tri_hjk.size(); ++i)
            if (h.tri_hjk[i] < 0 || h.tri_hjk[i] >= n) return fail(NR_ERR_INVALID, std::string(who) + ": triple index out of range");
        for (size_t i = 0; i < h.facets.size(); ++i)
            if (h.facets[i] < 0 || h.facets[i] >= n) return fail(NR_ERR_INVALID, std::string(who) + ": element index out of range");
        for (size_t i = 0; i < h.mesh_pairs.size(); ++i)
            if (h.mesh_pairs[i] < 0 || h.mesh_pairs[i] >= n) return fail(NR_ERR_INVALID, std::string(who) + ": pair index out of range");
        y_range(h.points, h.miny, h.maxy);
        std::unique_ptr<DeviceSet> S(new DeviceSet());
        const nr_host_network *nets[1] = {&h};
        const unsigned char *fcs[1] = {fc.data()};
        rc = build_set(1, nets, &ks, &kb, fcs, s, *S);
        if (rc != NR_OK) return rc;
        if (caching) {
            rc = dropin_hash(arr, s, &hash);
            if (rc != NR_OK) return rc;
            cache.device = device;
            cache.arrays = arr;
            cache.num_dof = num_dof;
            cache.use_gel = use_gel;
            cache.width = width;
            cache.ks = ks;
            cache.kb = kb;
            cache.hash = hash;
        }
        cache.set = std::move(S);
    } else {
        NR_CUDA_TRY(cudaMemcpyAsync(cache.set->x_all, d_pos, sizeof(double) * num_dof, cudaMemcpyDeviceToDevice, s));
    }
    DeviceSet &S = *cache.set;
    if (use_gel) {
        if (gel->nelems > 0)
            NR_CUDA_TRY(cudaMemcpyAsync(S.gel[0].elem_inv, gel->d_inv_mats, sizeof(double) * 6 * (size_t)gel->nelems,
                                        cudaMemcpyDeviceToDevice, s));
        rc = set_gel(S, gel->smod, gel->bmod, gel->dilation);
        if (rc != NR_OK) return rc;
    }
    nr_report rep;
    rc = relax_single_fp64(S, 0, p, s, &rep);
    if (!caching) {
        /* copy the results out before the image goes */
        if (rc >= 0) {
            NR_CUDA_TRY(cudaMemcpyAsync(d_pos, S.x_all, sizeof(double) * num_dof, cudaMemcpyDeviceToDevice, s));
            if (d_vel) NR_CUDA_TRY(cudaMemcpyAsync(d_vel, S.v_all, sizeof(double) * num_dof, cudaMemcpyDeviceToDevice, s));
            if (d_forces) NR_CUDA_TRY(cudaMemcpyAsync(d_forces, S.f_all, sizeof(double) * num_dof, cudaMemcpyDeviceToDevice, s));
            NR_CUDA_TRY(cudaStreamSynchronize(s));
        }
        cache.set.reset();
        if (rc < 0) return rc;
    } else {
        if (rc < 0) return rc;
        NR_CUDA_TRY(cudaMemcpyAsync(d_pos, S.x_all, sizeof(double) * num_dof, cudaMemcpyDeviceToDevice, s));
        if (d_vel) NR_CUDA_TRY(cudaMemcpyAsync(d_vel, S.v_all, sizeof(double) * num_dof, cudaMemcpyDeviceToDevice, s));
        if (d_forces) NR_CUDA_TRY(cudaMemcpyAsync(d_forces, S.f_all, sizeof(double) * num_dof, cudaMemcpyDeviceToDevice, s));
        NR_CUDA_TRY(cudaStreamSynchronize(s));
    }
    report_data[0] = rep.rms_force;
    report_data[1] = rep.e_stretch;
    report_data[2] = rep.e_bend;
    report_data[3] = rep.e_gel;
    *step_count = rep.steps;
    return rc;
}

/* One strain step of do_relaxation_run's protocol: the affine increment
 * and the values its record reports. */
struct SweepStep {
    double xdisp, ydisp, curr, maxc;
    int is_shear;
};

/* The steps of do_relaxation_run (large_strain_relax.cu:924-999):
 * compression from compr[0] to compr[1] by compr[2], then shear likewise,
 * in units of yrange, with the reference's loop arithmetic (a 1e-10 slack
 * on the bound).  A zero increment makes one step, where the reference
 * loops forever. */
static int sweep_steps(double smult, const double compr[3], const double shear[3], std::vector<SweepStep> &out) {
    constexpr size_t kMaxSteps = (size_t)1 << 24;
    out.clear();
    double min_disp = compr[0] * smult, max_disp = compr[1] * smult, inc = compr[2] * smult;
    double curr_disp = 0.0;
    if (max_disp > 0) {
        for (curr_disp = min_disp; curr_disp <= max_disp + 1e-10; curr_disp += inc) {
            if (out.size() >= kMaxSteps) return fail(NR_ERR_INVALID, "sweep: more than 2^24 strain steps");
            out.push_back({0.0, -inc, 0.0, curr_disp, 0});
            if (!(inc > 0)) break;
        }
    }
    const double max_comp = max_disp > min_disp ? curr_disp - inc : max_disp;
    min_disp = shear[0] * smult;
    max_disp = shear[1] * smult;
    inc = shear[2] * smult;
    if (max_disp > 0) {
        for (curr_disp = min_disp; curr_disp <= max_disp + 1e-10; curr_disp += inc) {
            if (out.size() >= kMaxSteps) return fail(NR_ERR_INVALID, "sweep: more than 2^24 strain steps");
            out.push_back({inc, 0.0, curr_disp, max_comp, 1});
            if (!(inc > 0)) break;
        }
    }
    return NR_OK;
}

static void record_step(const SweepStep &t, const nr_report &rep, nr_step_record &R) {
    R.curr_disp = t.curr;
    R.max_comp = t.maxc;
    R.e_stretch = rep.e_stretch;
    R.e_bend = rep.e_bend;
    R.e_gel = rep.e_gel;
    R.rms_force = rep.rms_force;
    R.max_force = rep.max_force;
    R.steps = rep.steps;
    R.is_shear = t.is_shear;
    R.status = rep.status;
    R.fp64_steps = rep.fp64_steps;
    R.stress_xx = rep.stress_xx;
    R.stress_yy = rep.stress_yy;
    R.stress_xy = rep.stress_xy;
}

/* Stream, graph and buffers of one captured sweep, released on every path
 * (cudaFree waits for the device). */
struct SweepGraphRes {
    cudaStream_t cs = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    FireState *states = nullptr;
    double2 *snaps = nullptr;
    ~SweepGraphRes() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (states) cudaFree(states);
        if (snaps) cudaFree(snaps);
        if (cs) cudaStreamDestroy(cs);
    }
};

/* The whole strain sweep as one CUDA graph.  Per step: the affine
 * increment, the relaxation (enqueue_grid), and device-to-device copies of
 * the FIRE state and, for a recorded shear step, of the positions.  One
 * graph launch, then the host reads all records.  The kernels and their
 * arguments are the step-by-step sweep's, so are the results, bit for bit.
 * After a failed step the graph still runs the later ones; the records
 * stop before the failure, as in the step-by-step sweep. */
static int sweep_graph(DeviceSet &S, const GridPlan &g, double miny, double yrange, const nr_fire_params &prm,
                       const std::vector<SweepStep> &steps, nr_step_record *records, int max_records, int *n_records,
                       double *shear_positions, cudaStream_t user) {
    const size_t n_steps = steps.size();
    const size_t n_rec = std::min(n_steps, (size_t)std::max(max_records, 0));
    const size_t n_nodes = (size_t)S.total_nodes;
    std::vector<long> snap_of(n_rec, -1);
    size_t n_snap = 0;
    if (shear_positions)
        for (size_t k = 0; k < n_rec; k++)
            if (steps[k].is_shear) snap_of[k] = (long)n_snap++;
    SweepGraphRes r;
    NR_CUDA_TRY(cudaStreamSynchronize(user));
    NR_CUDA_TRY(cudaStreamCreateWithFlags(&r.cs, cudaStreamNonBlocking));
    NR_CUDA_TRY(cudaMalloc(&r.states, sizeof(FireState) * n_steps));
    if (n_snap) NR_CUDA_TRY(cudaMalloc(&r.snaps, sizeof(double2) * n_nodes * n_snap));
    NR_CUDA_TRY(cudaStreamBeginCapture(r.cs, cudaStreamCaptureModeThreadLocal));
    int rc = NR_OK;
    for (size_t k = 0; k < n_steps && rc == NR_OK; k++) {
        const SweepStep &t = steps[k];
        cudaError_t e = launch_affine(S.x_all, (int)S.total_nodes, miny, yrange, t.xdisp, t.ydisp, r.cs);
        if (e == cudaSuccess) {
            rc = enqueue_grid(g, prm, r.cs);
            if (rc != NR_OK) break;
            e = cudaMemcpyAsync(r.states + k, g.d.st, sizeof(FireState), cudaMemcpyDeviceToDevice, r.cs);
        }
        if (e == cudaSuccess && k < n_rec && snap_of[k] >= 0)
            e = cudaMemcpyAsync(r.snaps + n_nodes * snap_of[k], S.x_all, sizeof(double2) * n_nodes,
                                cudaMemcpyDeviceToDevice, r.cs);
        if (e != cudaSuccess) rc = fail(NR_ERR_CUDA, std::string("sweep capture: ") + cudaGetErrorString(e));
    }
    const cudaError_t ec = cudaStreamEndCapture(r.cs, &r.graph);
    if (rc != NR_OK) return rc;
    if (ec != cudaSuccess) return fail(NR_ERR_CUDA, std::string("sweep capture: ") + cudaGetErrorString(ec));
    NR_CUDA_TRY(cudaGraphInstantiate(&r.exec, r.graph, 0));
    NR_CUDA_TRY(cudaGraphLaunch(r.exec, r.cs));
    std::vector<FireState> st(n_steps);
    NR_CUDA_TRY(cudaMemcpyAsync(st.data(), r.states, sizeof(FireState) * n_steps, cudaMemcpyDeviceToHost, r.cs));
    NR_CUDA_TRY(cudaStreamSynchronize(r.cs));
    std::vector<nr_report> reps(n_steps);
    size_t n_ok = n_steps;
    int err = NR_OK, worst = NR_OK;
    for (size_t k = 0; k < n_steps; k++) {
        const int s = report_status(st[k], g.d, &reps[k]);
        if (s < 0) {
            n_ok = k;
            err = s;
            break;
        }
        if (s == NR_NOT_CONVERGED) worst = NR_NOT_CONVERGED;
    }
    const size_t n_out = std::min(n_ok, n_rec);
    for (size_t k = 0; k < n_out; k++) {
        record_step(steps[k], reps[k], records[k]);
        if (snap_of[k] >= 0)
            NR_CUDA_TRY(cudaMemcpyAsync(shear_positions + 2 * n_nodes * k, r.snaps + n_nodes * snap_of[k],
                                        sizeof(double2) * n_nodes, cudaMemcpyDefault, r.cs));
    }
    NR_CUDA_TRY(cudaStreamSynchronize(r.cs));
    *n_records = (int)n_out;
    return err != NR_OK ? err : worst;
}

}  // namespace nr

using namespace nr;

struct nr_network {
    DeviceSet set;
};
struct nr_batch {
    DeviceSet set;
};

static cudaStream_t as_stream(void *s) { return (cudaStream_t)s; }

extern "C" {

int nr_network_create(const nr_host_network *net, double ks, double kb, void *stream, nr_network **out) {
    if (!net || !out) return fail(NR_ERR_INVALID, "nr_network_create: null argument");
    *out = nullptr;
    auto *d = new nr_network();
    const nr_host_network *nets[1] = {net};
    int rc = build_set(1, nets, &ks, &kb, nullptr, as_stream(stream), d->set);
    if (rc != NR_OK) {
        delete d;
        return rc;
    }
    *out = d;
    return NR_OK;
}

int nr_network_destroy(nr_network *d) {
    delete d;
    return NR_OK;
}

int nr_network_n_points(const nr_network *d) { return d ? d->set.dev[0].n : 0; }

int nr_network_set_positions(nr_network *d, const double *host_xy, void *stream) {
    if (!d || !host_xy) return fail(NR_ERR_INVALID, "nr_network_set_positions: null argument");
    NR_CUDA_TRY(cudaMemcpyAsync(d->set.x_all, host_xy, sizeof(double2) * d->set.total_nodes, cudaMemcpyDefault,
                                as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    return NR_OK;
}

int nr_network_get_positions(const nr_network *d, double *host_xy, void *stream) {
    if (!d || !host_xy) return fail(NR_ERR_INVALID, "nr_network_get_positions: null argument");
    NR_CUDA_TRY(cudaMemcpyAsync(host_xy, d->set.x_all, sizeof(double2) * d->set.total_nodes, cudaMemcpyDefault,
                                as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    return NR_OK;
}

double *nr_network_positions_device(nr_network *d) { return d ? (double *)d->set.x_all : nullptr; }

int nr_affine_displace(nr_network *d, double miny, double yrange, double xdisp, double ydisp, void *stream) {
    if (!d) return fail(NR_ERR_INVALID, "nr_affine_displace: null network");
    NR_CUDA_TRY(launch_affine(d->set.x_all, (int)d->set.total_nodes, miny, yrange, xdisp, ydisp, as_stream(stream)));
    return NR_OK;
}

int nr_relax(nr_network *d, const nr_fire_params *params, nr_report *report, void *stream) {
    if (!d || !report) return fail(NR_ERR_INVALID, "nr_relax: null argument");
    int rc = check_params(params);
    if (rc != NR_OK) return rc;
    clear_error();
    if (params->precision == NR_MIXED) {
        if (d->set.dev[0].use_gel) return fail(NR_ERR_INVALID, "nr_relax: a gel-coupled network relaxes in FP64 only");
        return relax_single_mixed(d->set, *params, as_stream(stream), report);
    }
    return relax_single_fp64(d->set, 0, *params, as_stream(stream), report);
}

int nr_forces(nr_network *d, double *host_f, void *stream) {
    if (!d || !host_f) return fail(NR_ERR_INVALID, "nr_forces: null argument");
    NR_CUDA_TRY(launch_forces(d->set.dev[0], as_stream(stream)));
    NR_CUDA_TRY(cudaMemcpyAsync(host_f, d->set.f_all, sizeof(double2) * d->set.total_nodes, cudaMemcpyDeviceToHost,
                                as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    return NR_OK;
}

int nr_energies(nr_network *d, double *e_stretch, double *e_bend, void *stream) {
    if (!d || !e_stretch || !e_bend) return fail(NR_ERR_INVALID, "nr_energies: null argument");
    const NetDev &dv = d->set.dev[0];
    NR_CUDA_TRY(launch_energies(dv, energy_blocks(dv, sm_count()), as_stream(stream)));
    FireState st;
    NR_CUDA_TRY(cudaMemcpyAsync(&st, dv.st, sizeof(FireState), cudaMemcpyDeviceToHost, as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    *e_stretch = st.e_stretch;
    *e_bend = st.e_bend;
    return NR_OK;
}

int nr_network_plan(nr_network *d, int precision, char *buf, size_t cap) {
    if (!d || !buf || cap == 0 || (precision != NR_FP64 && precision != NR_MIXED))
        return fail(NR_ERR_INVALID, "nr_network_plan: bad arguments");
    const NetDev &d0 = d->set.dev[0];
    char out[256];
    if (precision == NR_MIXED && d0.n <= kMixedCtaNodes) {
        snprintf(out, sizeof out, "batch kernels, one network (%d nodes <= %d)", d0.n, kMixedCtaNodes);
    } else {
        GridPlan g;
        const int rc = grid_plan(d->set, 0, precision == NR_MIXED, g);
        if (rc != NR_OK) return rc;
        if (g.tile)
            snprintf(out, sizeof out, "k_fire_tile_mixed ctas=%d threads=%d tiles=%d max_tile_nodes=%d", g.blocks,
                     g.tile_threads, g.tl.n_tiles, g.tl.max_nodes);
        else if (g.mixed) snprintf(out, sizeof out, "k_fire_grid_mixed ctas=%d", g.blocks);
        else if (g.res) 
            snprintf(out, sizeof out, "k_fire_res64 ctas=%d sub=%d smem=%zu%s", g.blocks, g.rd.sub, g.res_smem,
                     g.rd.mode == kResPairs ? " pairs" : g.rd.mode == kResStream ? " stream" : "");
        else if (g.cluster > 0) snprintf(out, sizeof out, "%s cluster=%d", g.dsm64 ? "k_fire_dsm64" : "k_fire_cluster", g.cluster);
        else snprintf(out, sizeof out, "k_fire_grid ctas=%d sub=%d", g.blocks, g.d.sub);
    }
    snprintf(buf, cap, "%s", out);
    return NR_OK;
}

int nr_batch_plan(nr_batch *b, int precision, char *buf, size_t cap) {
    if (!b || !buf || cap == 0 || (precision != NR_FP64 && precision != NR_MIXED))
        return fail(NR_ERR_INVALID, "nr_batch_plan: bad arguments");
    const DeviceSet &S = b->set;
    char out[256];
    if (precision == NR_MIXED) {
        const char *env = knob("NR_CLUSTER");
        const int cluster = env ? std::max(1, std::min(16, atoi(env))) : mixed_cluster_size(S.max_nodes);
        DsmPlan pl, ps;
        if (dsm_plan(S, env ? cluster : 0, cluster, pl)) {
            int cap_clusters = 0;
            const int n_small = solo_split(S, pl, ps, cap_clusters);
            const char *eh = knob("NR_ESCALATE_HOST");
            snprintf(out, sizeof out,
                     "k_fire_dsm_mixed cluster=%d clusters=%d resident=%d solo_networks=%d solo_ctas=%d escalation=%g "
                     "(%s)",
                     pl.C, cap_clusters, pl.resident, n_small, n_small > 0 ? solo_ctas(cap_clusters, pl.C) : 0,
                     escalate_fraction(), eh && atoi(eh) != 0 ? "host" : "device");
        } else {
            snprintf(out, sizeof out, "%s cluster=%d", cluster > 1 ? "k_fire_cluster_mixed" : "k_fire_batch_mixed",
                     cluster);
        }
    } else {
        const int c = fp64_batch_cluster(S.max_nodes);
        int bmax = 0, emax = 0, tmax = 0;
        if (c > 1 && fp64_kernel_choice() <= kFp64Dsm && fp64_dsm_plan(S, c, bmax, emax, tmax))
        {
            const Fp64Back b = fp64_back(S, c, bmax, emax, tmax);
            if (b.n > 0)
                snprintf(out, sizeof out, "k_fire_dsm64 cluster=%d beside cluster=%d clusters=%d networks=%d", c,
                         kFp64BackTeam, b.clusters, b.n);
            else snprintf(out, sizeof out, "k_fire_dsm64 cluster=%d", c);
        }
        else if (c > 1) snprintf(out, sizeof out, "k_fire_cluster cluster=%d", c);
        else snprintf(out, sizeof out, "k_fire_batch (one CTA per network)");
    }
    snprintf(buf, cap, "%s", out);
    return NR_OK;
}

int nr_stress(nr_network *d, double stress[3], double energies[2], void *stream) {
    if (!d || !stress || !energies) return fail(NR_ERR_INVALID, "nr_stress: null argument");
    const NetDev &dv = d->set.dev[0];
    NR_CUDA_TRY(launch_energies(dv, energy_blocks(dv, sm_count()), as_stream(stream)));
    FireState st;
    NR_CUDA_TRY(cudaMemcpyAsync(&st, dv.st, sizeof(FireState), cudaMemcpyDeviceToHost, as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    const double inv_a = dv.area > 0 ? 1.0 / dv.area : 0.0;
    for (int c = 0; c < 3; ++c) stress[c] = st.vir[c] * inv_a;
    energies[0] = st.e_stretch;
    energies[1] = st.e_bend;
    return NR_OK;
}

int nr_sweep(nr_network *d, double miny, double yrange, const nr_fire_params *params, const double compr[3],
             const double shear[3], nr_step_record *records, int max_records, int *n_records,
             double *shear_positions, void *stream) {
    if (!d || !compr || !shear || !n_records || (max_records > 0 && !records))
        return fail(NR_ERR_INVALID, "nr_sweep: null argument");
    int rc = check_params(params);
    if (rc != NR_OK) return rc;
    if (!(yrange > 0)) return fail(NR_ERR_INVALID, "nr_sweep: yrange must be positive");
    *n_records = 0;
    std::vector<SweepStep> steps;
    rc = sweep_steps(yrange, compr, shear, steps);
    if (rc != NR_OK) return rc;
    const size_t n2 = 2 * (size_t)d->set.total_nodes;
    int worst = NR_OK;
    for (const SweepStep &t : steps) {
        rc = nr_affine_displace(d, miny, yrange, t.xdisp, t.ydisp, stream);
        if (rc != NR_OK) return rc;
        nr_report rep;
        rc = nr_relax(d, params, &rep, stream);
        if (rc < 0) return rc;
        if (rc == NR_NOT_CONVERGED) worst = NR_NOT_CONVERGED;
        if (*n_records < max_records) {
            record_step(t, rep, records[*n_records]);
            if (t.is_shear && shear_positions) {
                rc = nr_network_get_positions(d, shear_positions + n2 * (size_t)(*n_records), stream);
                if (rc != NR_OK) return rc;
            }
            (*n_records)++;
        }
    }
    return worst;
}

int nr_sweep_graph(nr_network *d, double miny, double yrange, const nr_fire_params *params, const double compr[3],
                   const double shear[3], nr_step_record *records, int max_records, int *n_records,
                   double *shear_positions, void *stream) {
    if (!d || !compr || !shear || !n_records || (max_records > 0 && !records))
        return fail(NR_ERR_INVALID, "nr_sweep_graph: null argument");
    int rc = check_params(params);
    if (rc != NR_OK) return rc;
    if (!(yrange > 0)) return fail(NR_ERR_INVALID, "nr_sweep_graph: yrange must be positive");
    const bool mixed = params->precision == NR_MIXED;
    const NetDev &d0 = d->set.dev[0];
    if (mixed && d0.use_gel) return fail(NR_ERR_INVALID, "nr_sweep_graph: a gel-coupled network relaxes in FP64 only");
    /* A small network's mixed relaxation is steered between launches by the
     * host (one CTA, escalation): it is swept step by step. */
    if (mixed && d0.n <= kMixedCtaNodes)
        return nr_sweep(d, miny, yrange, params, compr, shear, records, max_records, n_records, shear_positions,
                        stream);
    *n_records = 0;
    std::vector<SweepStep> steps;
    rc = sweep_steps(yrange, compr, shear, steps);
    if (rc != NR_OK || steps.empty()) return rc;
    clear_error();
    GridPlan g;
    rc = grid_plan(d->set, 0, mixed, g);
    if (rc != NR_OK) return rc;
    return sweep_graph(d->set, g, miny, yrange, *params, steps, records, max_records, n_records, shear_positions,
                       as_stream(stream));
}

int nr_run_fire_md(int num_dof, int npairs, int ntriples, double width, double ks, double kb, double *d_pos,
                   double *d_vel, double *d_forces, const int *d_pair_list, const double *d_lengths,
                   const signed char *d_e_offsets, const int *d_triples, const signed char *d_t_offsets,
                   const unsigned char *d_fcodes, const double fire_params[5], double mass, double fcut,
                   int max_steps, int nmin, double report_data[3], int *step_count, void *stream) {
    if (!report_data) return fail(NR_ERR_INVALID, "nr_run_fire_md: bad arguments");
    double rep4[4];
    const int rc = run_fire_md_impl("nr_run_fire_md", num_dof, npairs, ntriples, width, ks, kb, d_pos, d_vel, d_forces,
                                    d_pair_list, d_lengths, d_e_offsets, d_triples, d_t_offsets, d_fcodes,
                                    fire_params, mass, fcut, max_steps, nmin, nullptr, rep4, step_count, stream);
    if (rc >= 0) memcpy(report_data, rep4, 3 * sizeof(double));
    return rc;
}

int nr_mesh_run_fire_md(int num_dof, int npairs, int ntriples, int nelems, double width, double ks, double kb,
                        double smod, double bmod, double dilation, double *d_pos, double *d_vel, double *d_forces,
                        const int *d_pair_list, const double *d_lengths, const signed char *d_e_offsets,
                        const int *d_triples, const signed char *d_t_offsets, const int *d_elems,
                        const double *d_areas, const double *d_inv_mats, const int *d_mpairs, int n_mpairs,
                        const unsigned char *d_fcodes, const double fire_params[5], double mass, double fcut,
                        int max_steps, int nmin, double report_data[4], int *step_count, void *stream) {
    GelArgs g{nelems, n_mpairs, smod, bmod, dilation, d_elems, d_areas, d_inv_mats, d_mpairs};
    return run_fire_md_impl("nr_mesh_run_fire_md", num_dof, npairs, ntriples, width, ks, kb, d_pos, d_vel, d_forces,
                            d_pair_list, d_lengths, d_e_offsets, d_triples, d_t_offsets, d_fcodes, fire_params, mass,
                            fcut, max_steps, nmin, &g, report_data, step_count, stream);
}

int nr_network_set_gel(nr_network *d, double smod, double bmod, double dilation) {
    if (!d) return fail(NR_ERR_INVALID, "nr_network_set_gel: null network");
    return set_gel(d->set, smod, bmod, dilation);
}

int nr_network_gel_inv_mats(nr_network *d, void *stream) {
    if (!d) return fail(NR_ERR_INVALID, "nr_network_gel_inv_mats: null network");
    const DeviceSet &S = d->set;
    NR_CUDA_TRY(launch_inv_mats((const double *)S.dev[0].x, (const int *)S.gel[0].elem, 4, S.dev[0].n_elems,
                                S.gel[0].elem_inv, as_stream(stream)));
    return NR_OK;
}

int nr_dilate(nr_network *d, double minx, double miny, double factor, void *stream) {
    if (!d) return fail(NR_ERR_INVALID, "nr_dilate: null network");
    NR_CUDA_TRY(launch_dilate(d->set.x_all, (int)d->set.total_nodes, minx, miny, factor, as_stream(stream)));
    return NR_OK;
}

int nr_mesh_energies(nr_network *d, double energies[3], void *stream) {
    if (!d || !energies) return fail(NR_ERR_INVALID, "nr_mesh_energies: null argument");
    const NetDev &dv = d->set.dev[0];
    NR_CUDA_TRY(launch_energies(dv, energy_blocks(dv, sm_count()), as_stream(stream)));
    FireState st;
    NR_CUDA_TRY(cudaMemcpyAsync(&st, dv.st, sizeof(FireState), cudaMemcpyDeviceToHost, as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    energies[0] = st.e_stretch;
    energies[1] = st.e_bend;
    energies[2] = dv.use_gel ? st.e_gel : 0.0;
    return NR_OK;
}

int nr_get_inv_mats(int n_facets, const double *d_pos, const int *d_facets, double *d_inv_mats, void *stream) {
    if (n_facets < 0 || (n_facets > 0 && (!d_pos || !d_facets || !d_inv_mats)))
        return fail(NR_ERR_INVALID, "nr_get_inv_mats: bad arguments");
    NR_CUDA_TRY(launch_inv_mats(d_pos, d_facets, 3, n_facets, d_inv_mats, as_stream(stream)));
    return NR_OK;
}

int nr_mesh_prepare(nr_network *d, double smod, double bmod, double dilation, double area, double *pref_dilation,
                    void *stream) {
    if (!d || !pref_dilation) return fail(NR_ERR_INVALID, "nr_mesh_prepare: null argument");
    DeviceSet &S = d->set;
    int rc = nr_dilate(d, S.minx[0], S.miny[0], std::sqrt(1 + dilation), stream);
    if (rc != NR_OK) return rc;
    double net_bmod = 0;
    if (S.dev[0].use_bonds) {
        double es = 0, eb = 0;
        rc = nr_energies(d, &es, &eb, stream);
        if (rc != NR_OK) return rc;
        net_bmod = es;
        net_bmod *= 2 / area / (dilation * dilation);
    }
    const double pref_d = dilation * (bmod + net_bmod) / bmod;
    *pref_dilation = pref_d;
    return set_gel(S, smod, bmod, pref_d);
}

int nr_mesh_sweep(nr_network *d, double miny, double height, const nr_fire_params *params, const double compr[3],
                  const double shear[3], nr_step_record *records, int max_records, int *n_records,
                  double *shear_positions, void *stream) {
    if (!d || !compr || !shear || !n_records || (max_records > 0 && !records))
        return fail(NR_ERR_INVALID, "nr_mesh_sweep: null argument");
    int rc = check_params(params);
    if (rc != NR_OK) return rc;
    if (!(height > 0)) return fail(NR_ERR_INVALID, "nr_mesh_sweep: height must be positive");
    *n_records = 0;
    const double smult = height;
    double range = height;
    const size_t n2 = 2 * (size_t)d->set.total_nodes;
    int worst = NR_OK;
    auto relax_record = [&](double curr, double maxc, int is_shear) -> int {
        nr_report rep;
        int r = nr_relax(d, params, &rep, stream);
        if (r < 0) return r;
        if (r == NR_NOT_CONVERGED) worst = NR_NOT_CONVERGED;
        if (*n_records < max_records) {
            nr_step_record &R = records[*n_records];
            R.curr_disp = curr;
            R.max_comp = maxc;
            R.e_stretch = rep.e_stretch;
            R.e_bend = rep.e_bend;
            R.e_gel = rep.e_gel;
            R.rms_force = rep.rms_force;
            R.max_force = rep.max_force;
            R.steps = rep.steps;
            R.is_shear = is_shear;
            R.status = rep.status;
            R.fp64_steps = rep.fp64_steps;
            R.stress_xx = rep.stress_xx;
            R.stress_yy = rep.stress_yy;
            R.stress_xy = rep.stress_xy;
            if (is_shear && shear_positions) {
                r = nr_network_get_positions(d, shear_positions + n2 * (size_t)(*n_records), stream);
                if (r != NR_OK) return r;
            }
            (*n_records)++;
        }
        return NR_OK;
    };
    double min_disp = compr[0] * smult, max_disp = compr[1] * smult, inc = compr[2] * smult;
    double curr_disp = 0.0;
    if (max_disp > 0) {
        rc = nr_affine_displace(d, miny, range, 0, -min_disp, stream);
        if (rc != NR_OK) return rc;
        range -= min_disp;
        for (curr_disp = min_disp; curr_disp <= max_disp + 1e-10; curr_disp += inc) {
            rc = relax_record(0.0, curr_disp, 0);
            if (rc < 0) return rc;
            if (curr_disp < max_disp) {
                rc = nr_affine_displace(d, miny, range, 0, -inc, stream);
                if (rc != NR_OK) return rc;
                range -= inc;
            }
            if (!(inc > 0)) break; /* the reference loops forever when inc == 0 */
        }
    }
    const double max_comp = max_disp > min_disp ? curr_disp - inc : max_disp;
    min_disp = shear[0] * smult;
    max_disp = shear[1] * smult;
    inc = shear[2] * smult;
    if (max_disp > 0) {
        rc = nr_affine_displace(d, miny, range, min_disp, 0, stream);
        if (rc != NR_OK) return rc;
        for (curr_disp = min_disp; curr_disp <= max_disp + 1e-10; curr_disp += inc) {
            rc = relax_record(curr_disp, max_comp, 1);
            if (rc < 0) return rc;
            if (curr_disp < max_disp) {
                rc = nr_affine_displace(d, miny, range, inc, 0, stream);
                if (rc != NR_OK) return rc;
            }
            if (!(inc > 0)) break;
        }
    }
    return worst;
}

int nr_batch_create(int n, const nr_host_network *const *nets, const double *ks, const double *kb, void *stream,
                    nr_batch **out) {
    if (n <= 0 || !nets || !ks || !kb || !out) return fail(NR_ERR_INVALID, "nr_batch_create: bad arguments");
    *out = nullptr;
    auto *b = new nr_batch();
    int rc = build_set(n, nets, ks, kb, nullptr, as_stream(stream), b->set);
    if (rc != NR_OK) {
        delete b;
        return rc;
    }
    *out = b;
    return NR_OK;
}

int nr_batch_destroy(nr_batch *b) {
    delete b;
    return NR_OK;
}
int nr_batch_size(const nr_batch *b) { return b ? b->set.n_nets : 0; }
int nr_batch_last_launches(const nr_batch *b) { return b ? b->set.launches : 0; }
int nr_batch_total_points(const nr_batch *b) { return b ? (int)b->set.total_nodes : 0; }

int nr_batch_set_positions(nr_batch *b, const double *host_xy, void *stream) {
    if (!b || !host_xy) return fail(NR_ERR_INVALID, "nr_batch_set_positions: null argument");
    NR_CUDA_TRY(cudaMemcpyAsync(b->set.x_all, host_xy, sizeof(double2) * b->set.total_nodes, cudaMemcpyDefault,
                                as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    return NR_OK;
}

int nr_batch_get_positions(const nr_batch *b, double *host_xy, void *stream) {
    if (!b || !host_xy) return fail(NR_ERR_INVALID, "nr_batch_get_positions: null argument");
    NR_CUDA_TRY(cudaMemcpyAsync(host_xy, b->set.x_all, sizeof(double2) * b->set.total_nodes, cudaMemcpyDefault,
                                as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    return NR_OK;
}

double *nr_batch_positions_device(nr_batch *b) { return b ? (double *)b->set.x_all : nullptr; }

int nr_batch_affine_displace(nr_batch *b, const double *miny, const double *yrange, const double *xdisp,
                             const double *ydisp, void *stream) {
    if (!b || !miny || !yrange || !xdisp || !ydisp) return fail(NR_ERR_INVALID, "nr_batch_affine_displace: null argument");
    std::vector<double4> prm(b->set.n_nets);
    for (int i = 0; i < b->set.n_nets; ++i) prm[i] = make_double4(miny[i], yrange[i], xdisp[i], ydisp[i]);
    NR_CUDA_TRY(cudaMemcpyAsync(b->set.affine_prm, prm.data(), sizeof(double4) * prm.size(), cudaMemcpyHostToDevice,
                                as_stream(stream)));
    NR_CUDA_TRY(launch_affine_batch(b->set.dev_array, b->set.affine_prm, b->set.n_nets, as_stream(stream)));
    NR_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    return NR_OK;
}

int nr_batch_sweep(nr_batch *b, const nr_fire_params *params, const double compr[3], const double shear[3],
                   nr_step_record *records, int max_steps, int *n_steps, int graph, void *stream) {
    if (!b || !compr || !shear || !n_steps || (max_steps > 0 && !records))
        return fail(NR_ERR_INVALID, "nr_batch_sweep: null argument");
    int rc = check_params(params);
    if (rc != NR_OK) return rc;
    clear_error();
    *n_steps = 0;
    DeviceSet &S = b->set;
    const int n = S.n_nets;
    std::vector<SweepStep> steps;
    rc = sweep_steps(1.0, compr, shear, steps); /* in strain units: the same steps for every network */
    if (rc != NR_OK || steps.empty()) return rc;
    /* per network and kind of step, the affine increment in its own
     * displacement units (strain x (maxy - miny)) */
    std::vector<double4> prm(2 * (size_t)n);
    for (int i = 0; i < n; ++i) {
        const double H = S.maxy[i] - S.miny[i];
        for (int kind = 0; kind < 2; ++kind) {
            const SweepStep *t = nullptr;
            for (const SweepStep &q : steps)
                if (q.is_shear == kind) {
                    t = &q;
                    break;
                }
            prm[(size_t)kind * n + i] = make_double4(S.miny[i], H, t ? t->xdisp * H : 0.0, t ? t->ydisp * H : 0.0);
        }
    }
    cudaStream_t user = as_stream(stream);
    struct Res {
        cudaStream_t cs = nullptr;
        cudaGraph_t g = nullptr;
        cudaGraphExec_t e = nullptr;
        double4 *prm = nullptr;
        FireState *st = nullptr;
        ~Res() {
            if (e) cudaGraphExecDestroy(e);
            if (g) cudaGraphDestroy(g);
            if (prm) cudaFree(prm);
            if (st) cudaFree(st);
            if (cs) cudaStreamDestroy(cs);
        }
    } r;
    const size_t ns = steps.size();
    NR_CUDA_TRY(cudaStreamSynchronize(user));
    NR_CUDA_TRY(cudaMalloc(&r.prm, sizeof(double4) * prm.size()));
    NR_CUDA_TRY(cudaMalloc(&r.st, sizeof(FireState) * n * ns));
    NR_CUDA_TRY(cudaMemcpy(r.prm, prm.data(), sizeof(double4) * prm.size(), cudaMemcpyHostToDevice));
    NR_CUDA_TRY(cudaStreamCreateWithFlags(&r.cs, cudaStreamNonBlocking));
    if (graph) NR_CUDA_TRY(cudaStreamBeginCapture(r.cs, cudaStreamCaptureModeThreadLocal));
    int launches = 0;
    for (size_t k = 0; k < ns && rc == NR_OK; ++k) {
        cudaError_t e = launch_affine_batch(S.dev_array, r.prm + (size_t)steps[k].is_shear * n, n, r.cs);
        if (e != cudaSuccess) {
            rc = fail(NR_ERR_CUDA, std::string("nr_batch_sweep: ") + cudaGetErrorString(e));
            break;
        }
        rc = enqueue_set_batch(S, *params, r.cs, graph != 0);
        if (rc != NR_OK) break;
        launches += 1 + S.launches;
        e = cudaMemcpyAsync(r.st + k * n, S.st, sizeof(FireState) * n, cudaMemcpyDeviceToDevice, r.cs);
        if (e != cudaSuccess) rc = fail(NR_ERR_CUDA, std::string("nr_batch_sweep: ") + cudaGetErrorString(e));
    }
    if (graph) {
        const cudaError_t ec = cudaStreamEndCapture(r.cs, &r.g);
        if (rc != NR_OK) return rc;
        if (ec != cudaSuccess) return fail(NR_ERR_CUDA, std::string("nr_batch_sweep capture: ") + cudaGetErrorString(ec));
        NR_CUDA_TRY(cudaGraphInstantiate(&r.e, r.g, 0));
        NR_CUDA_TRY(cudaGraphLaunch(r.e, r.cs));
    } else if (rc != NR_OK) {
        cudaStreamSynchronize(r.cs);
        return rc;
    }
    std::vector<FireState> st(n * ns);
    NR_CUDA_TRY(cudaMemcpyAsync(st.data(), r.st, sizeof(FireState) * n * ns, cudaMemcpyDeviceToHost, r.cs));
    NR_CUDA_TRY(cudaStreamSynchronize(r.cs));
    S.launches = launches;
    int worst = NR_OK;
    std::vector<nr_report> reps(n);
    for (size_t k = 0; k < ns; ++k) {
        const int w = reports_of(S, st.data() + k * n, reps.data());
        if (w < 0 && worst >= 0) worst = w;
        else if (w == NR_NOT_CONVERGED && worst == NR_OK) worst = w;
        if ((int)k < max_steps)
            for (int i = 0; i < n; ++i) {
                const double H = S.maxy[i] - S.miny[i];
                SweepStep t = steps[k];
                t.curr *= H;
                t.maxc *= H;
                record_step(t, reps[i], records[k * n + i]);
            }
    }
    *n_steps = (int)ns;
    if (worst < 0) return fail(worst, "nr_batch_sweep: a network failed");
    return worst;
}

int nr_batch_relax(nr_batch *b, const nr_fire_params *params, nr_report *reports, void *stream) {
    if (!b || !reports) return fail(NR_ERR_INVALID, "nr_batch_relax: null argument");
    int rc = check_params(params);
    if (rc != NR_OK) return rc;
    clear_error();
    return relax_set_batch(b->set, *params, as_stream(stream), reports);
}

}  // extern "C"

extern "C" int nr_dsm_layout_check(const nr_host_network *h, long long stats[4]) {
    if (!h || !stats) return fail(NR_ERR_INVALID, "nr_dsm_layout_check: null argument");
    for (int k = 0; k < 4; ++k) stats[k] = 0;
    const int n = h->n_points, ne = h->n_edges(), nt = h->n_triples();
    Incidence inc;
    build_incidence(n, h->edge_ij.data(), ne, h->tri_hjk.data(), nt, true, true, inc);
    std::vector<unsigned char> fc(n);
    nr_host_network_fcodes(h, fc.data());
    Image img;
    NetOff o;
    memset(&o, 0, sizeof o);
    NetDsm m;
    build_dsm_layout(*h, inc, fc.data(), img, o, m);
    if (m.bsub <= 0) return NR_ERR_CAPACITY;
    const char *base = img.data();
    const int2 *bref = (const int2 *)(base + o.dsm_bref);
    const int *bidx = (const int *)(base + o.dsm_bidx);
    const int4 *tref = (const int4 *)(base + o.dsm_tref);
    const int *bent = (const int *)(base + o.dsm_bent);
    const int *tent = (const int *)(base + o.dsm_tent);
    const int4 *grec = (const int4 *)(base + o.dsm_grec);
    const int4 *xrec = (const int4 *)(base + o.dsm_xrec);
    const long long xquads = (long long)(img.zeros_size() / sizeof(uint4));
    const int bsub = m.bsub;
    long long bad = o.has_dsm_quads != (bsub <= kDsmMaxSubBlock) || (!o.has_dsm_quads && img.zeros_size() > 0);
    auto ref_of = [&](int v) { return ((v / bsub) << 16) | (v % bsub); };
    std::vector<int> seen(n, 0);
    int parts = 0;
    for (int g = 0; g * bsub < n; ++g) {
        ++parts;
        const int v0 = g * bsub, v1 = std::min(n, v0 + bsub);
        for (int k = v0; k < v1; ++k) {
            const int4 r = grec[k];
            const int v = r.x & 0x0fffffff, f = (int)((unsigned)r.x >> 28);
            /* the group's record: the same node, room for its entries, the
             * same place for all 32 lanes and no other group's */
            if (o.has_dsm_quads) {
                const int4 xr = xrec[k], x0 = xrec[k - (k - v0) % 32];
                if (xr.x != r.x || xr.y != x0.y || xr.z != x0.z ||
                    4 * xr.z < (r.z & 0xffff) + (int)((unsigned)r.z >> 16) || xr.y + 32LL * xr.z > xquads ||
                    (k > v0 && (k - v0) % 32 == 0 && xr.y < xrec[k - 1].y + 32 * xrec[k - 1].z))
                    ++bad;
            }
            if (v < v0 || v >= v1) {
                ++bad;
                continue;
            }
            seen[v]++;
            const int nbe = inc.bptr[v + 1] - inc.bptr[v], nte = inc.tptr[v + 1] - inc.tptr[v];
            if (f != (fc[v] & 3) || r.y != inc.bptr[v] || r.w != inc.tptr[v] || (r.z & 0xffff) != nbe ||
                ((unsigned)r.z >> 16) != (unsigned)nte)
                ++bad;
            if (k > v0) {
                const int u = grec[k - 1].x & 0x0fffffff;
                if (u >= v0 && u < v1) {
                    const int pnb = inc.bptr[u + 1] - inc.bptr[u], pnt = inc.tptr[u + 1] - inc.tptr[u];
                    if (pnt < nte || (pnt == nte && pnb < nbe)) ++bad; /* order: decreasing (triples, bonds) */
                }
            }
        }
    }
    for (int v = 0; v < n; ++v)
        if (seen[v] != 1) ++bad;
    /* item slots: owned by the sub-block of the bond's first node / the
     * triple's hinge, with that item's node references */
    for (int g = 0; g < kDsmParts; ++g) {
        for (int sl = m.bo[g]; sl < m.bo[g + 1]; ++sl) {
            const int b = bidx[sl];
            if (b < 0 || b >= ne) {
                ++bad;
                continue;
            }
            const int i = h->edge_ij[2 * b], j = h->edge_ij[2 * b + 1];
            if (i / bsub != g || bref[sl].x != ref_of(i) || bref[sl].y != ref_of(j)) ++bad;
        }
        for (int sl = m.to[g]; sl < m.to[g + 1]; ++sl) {
            const int4 r = tref[sl];
            if (r.w < 0 || r.w >= nt) {
                ++bad;
                continue;
            }
            const int hh = h->tri_hjk[3 * r.w], jj = h->tri_hjk[3 * r.w + 1], kk = h->tri_hjk[3 * r.w + 2];
            if (hh / bsub != g || r.x != ref_of(hh) || r.y != ref_of(jj) || r.z != ref_of(kk)) ++bad;
        }
    }
    /* resolved incidence entries: owner sub-block, slot, role of the entry
     * they replace */
    for (size_t e = 0; e < inc.bent.size(); ++e) {
        const unsigned c = (unsigned)bent[e];
        const int g = (int)(c >> 28), sl = (int)((c >> 1) & 0x7ffffffu);
        const int b = inc.bent[e] >> 1;
        if ((int)(c & 1u) != (inc.bent[e] & 1) || sl < m.bo[g] || sl >= m.bo[g + 1] || bidx[sl] != b) ++bad;
    }
    for (size_t e = 0; e < inc.tent.size(); ++e) {
        const unsigned c = (unsigned)tent[e];
        const int g = (int)(c >> 28), sl = (int)((c >> 2) & 0x3ffffffu);
        const int t = inc.tent[e] >> 2;
        if ((int)(c & 3u) != (inc.tent[e] & 3) || sl < m.to[g] || sl >= m.to[g + 1] || tref[sl].w != t) ++bad;
    }
    stats[0] = bsub;
    stats[1] = parts;
    stats[2] = n;
    stats[3] = bad;
    return NR_OK;
}

