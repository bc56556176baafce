// Streamed step: many fused steps in one launch, for meshes too large for the
// resident step (resident.cu) whose tables still fit in L2.
//
// One block per node tile, three (FP64) or four (mixed) blocks per SM, every
// tile's block resident for the whole launch.  A tile's positions and its
// halo's, its velocities, mass terms and force accumulators stay in shared
// memory; the triangles' tables stream from L2 in the node-tiled step's chunk
// records (NodeTilePlan), the next chunk's -- across the step's end too -- while
// the block adds up the current one's runs.  Positions are gathered from
// shared memory by 16-bit local ids, and tiles exchange them as the resident
// step does (packets.cuh; the same argument that no packet is overwritten
// early holds, tile adjacency being the same).  Every node's contributions are
// added in ascending triangle order from zero, with the arithmetic of the
// other paths: the same bits.
//
// What bounds it: the SM, at 12 (FP64) or 16 warps: 2,100 clocks per chunk of
// 128 triangles, of which FP64 takes half and shared-memory accesses two
// thirds, plus a node phase and one exchange per step.  Per step, FP64 (mixed),
// against the two-kernel step in graphs: 50,310 triangles 6.7 (6.3) us against
// 11.1 (10.0), 72,364 8.8 (6.8) against 13.2 (11.0), 147,922 14.6 (11.7)
// against 19.0 (15.9).  A component of a run per thread, four values ahead of
// the adds, was slower (15.9 us): three times the entries' loads.
//
// The launch is cooperative; every wait is bounded; the state a launch starts
// from stays untouched, and the steps of one that tripped the force guard or was
// given up run again one by one, as for the resident step.
//
// The batch runs stretches of steps in which no instance changes its status or
// checks for equilibrium the same way (BATCH): the union is the mesh, a tile
// keeps its instances' scalars in shared memory, and their dial values of
// every step come from a table.  Done and failed instances' triangles and
// nodes are left alone, except that their nodes keep publishing.
#include <algorithm>
#include <climits>

#include "internal.cuh"
#include "node_tile_walk.cuh"
#include "packets.cuh"
#include "step_common.cuh"
#include "tile_copy.cuh"
#include "tri_contrib.cuh"

namespace msb {
namespace {

using namespace packets;
using namespace stepdev;
using namespace tiles;
using namespace tridev;

constexpr int kPolls = 4;  // halo components a thread has under way together

// Shared memory of a block: staging area, two node sections, then per node of
// the tile accumulator, velocity (3 doubles each), dt / m and the damping
// term, positions of the tile and its halo, flags.
// For the batch: its instances' scalars, and each node's instance.
struct StInst {
    double ks, kb, igmh, nu, dt, force_limit;
    double lam[2], pw[2];  // of this step and the next, by the step's parity
    int frozen;
};
template <bool MIXED>
struct StSmem {
    static constexpr size_t stage = NtSmem<MIXED>::stage;
    __host__ __device__ static size_t bytes(size_t stride, int nodes, int halo, int insts) {
        return stage + 2 * NtSmem<MIXED>::ns_cap(stride) + 8 * (8 * (size_t)nodes + 3 * ((size_t)nodes + halo)) +
               ((size_t)nodes + 15) / 16 * 16 +
               (insts ? sizeof(StInst) * (size_t)insts + ((size_t)nodes * 2 + 15) / 16 * 16 : 0);
    }
};

// Loads that pass L1 by (tables are read once per step) and stay in L2.
__device__ __forceinline__ unsigned ld_l2(const unsigned* p) {
    unsigned v;
    asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_l2(const float* p) {
    float v;
    asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_l2(const double* p) {
    double v;
    asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Slot i's tables of chunk c: local patch ids (two to a word), weights, area,
// and the director trigonometry or the metric in force (abar, bbar).
template <int DIAL, bool MIXED>
struct StTables {
    using R = typename Real<MIXED>::T;
    static constexpr int kMet = DIAL == DIAL_LCE ? 3 : 6;
    unsigned lid[3];
    R cf[24];
    double area, met[kMet];
    int tag;  // the slot's instance (batch)

    __device__ __forceinline__ void load(const NodeTilePlan& q, const StreamPlan& sp, int c, int i) {
        using L = TileLayout<MIXED>;
        const unsigned char* rec = q.rec + (size_t)c * q.stride;
        const R* coef = reinterpret_cast<const R*>(rec + L::ids);
        const double* aux = reinterpret_cast<const double*>(rec + L::ids + L::coef);
#pragma unroll
        for (int k = 0; k < 3; ++k) lid[k] = ld_l2(sp.local + ((size_t)c * 3 + k) * kTile + i);
#pragma unroll
        for (int k = 0; k < 24; ++k) cf[k] = ld_l2(coef + k * kTile + i);
        area = ld_l2(aux + i);
#pragma unroll
        for (int k = 0; k < kMet; ++k)
            met[k] = DIAL == DIAL_LCE ? ld_l2(aux + (k + 1) * kTile + i)
                                      : ld_l2(sp.metric + ((size_t)c * 6 + k) * kTile + i);
        tag = q.chunk_tag ? __ldg(q.chunk_tag + (size_t)c * kTile + i) : 0;
    }
};

// The metric in force of every slot, field-major per chunk, for a launch that
// reads abar and bbar from the arrays (they do not change while it runs).
__global__ void k_stream_metric(const DevMesh m, const NodeTilePlan q, double* __restrict__ out) {
    const int c = blockIdx.x, i = threadIdx.x;
    const int t = q.chunk_tri[(size_t)c * kTile + i];
    const size_t T = m.T;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        out[((size_t)c * 6 + k) * kTile + i] = t >= 0 ? m.abar[k * T + t] : 0.0;
        out[((size_t)c * 6 + 3 + k) * kTile + i] = t >= 0 ? m.bbar[k * T + t] : 0.0;
    }
}

template <int DIAL, bool MIXED, bool BATCH>
__global__ void __launch_bounds__(kTile, MIXED ? 4 : 3)
    k_streamed(const DevMesh m, const NodeTilePlan q, const StreamPlan sp, const BatchStream bs, const DevState s,
               const StepScalars sc, int steps, unsigned tag0) {
    using R = typename Real<MIXED>::T;
    int g0 = 0;
    if constexpr (!BATCH) {
        g0 = global_step(s.err, sc.step);
        // An earlier launch tripped the guard or was given up: uniform over the grid.
        if (stale(s.err, g0)) return;
    }
    auto give_up = [&]() {
        if constexpr (BATCH) atomicExch(bs.trip, 5);
        else record_timeout(s, g0);
    };
    extern __shared__ __align__(128) unsigned char st_smem[];
    __shared__ uint64_t bar;
    const int NT = q.nodes, N = m.N, ld = NT + sp.halo;
    const size_t ns_cap = NtSmem<MIXED>::ns_cap(q.stride);
    R* stage = reinterpret_cast<R*>(st_smem);
    unsigned char* nsec = st_smem + StSmem<MIXED>::stage;
    double* acc = reinterpret_cast<double*>(nsec + 2 * ns_cap);  // [NT][3]
    double* svel = acc + 3 * NT;                                 // [3][NT]
    double* sk2 = svel + 3 * NT;
    double* sdm = sk2 + NT;
    double* spos = sdm + NT;                                     // [3][ld]: own nodes, then the halo
    // 1: constrained, 2: others read it, 4: its instance is done or failed.
    unsigned char* sflag = reinterpret_cast<unsigned char*>(spos + 3 * ld);
    StInst* sinst = reinterpret_cast<StInst*>(sflag + (NT + 15) / 16 * 16);
    unsigned short* sni = reinterpret_cast<unsigned short*>(sinst + bs.insts);  // [NT] node's instance in sinst

    const int b = blockIdx.x, i = threadIdx.x;
    const int n0 = b * NT, nn = min(NT, N - n0), nh = __ldg(sp.halo_count + b);
    const int* halo_id = sp.halo_id + (size_t)b * sp.halo;
    const int c0 = __ldg(q.tile_chunk + b), c1 = __ldg(q.tile_chunk + b + 1);
    const double* pos = pos_buf(s, sc.parity);
    const double* vel = vel_buf(s, sc.parity);
    if (i == 0) {
        bar_init(&bar);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    int i_lo = 0, i_n = 0;
    if constexpr (BATCH) {
        i_lo = __ldg(bs.node_inst + n0);
        i_n = __ldg(bs.node_inst + n0 + nn - 1) - i_lo + 1;
        for (int k = i; k < i_n; k += kTile) {
            const InstParams& p = bs.ip[i_lo + k];
            StInst& o = sinst[k];
            o.ks = p.ks;
            o.kb = p.kb;
            o.igmh = p.igmh;
            o.nu = p.nu;
            o.dt = p.dt;
            o.force_limit = p.force_limit;
            o.frozen = bs.is[i_lo + k].status >= INST_DONE;
            const double2 d = __ldg(bs.dials + i_lo + k);
            o.lam[0] = d.x;
            o.pw[0] = d.y;
        }
    }
    for (int j = i; j < nn; j += kTile) {
        const double mass = __ldg(m.mass + n0 + j);
        int frozen = 0;
        if constexpr (BATCH) {
            const int inst = __ldg(bs.node_inst + n0 + j);
            const InstParams& p = bs.ip[inst];
            const double damping = bs.is[inst].damping;
            sni[j] = (unsigned short)(inst - i_lo);
            sk2[j] = p.dt / mass;
            sdm[j] = -damping * mass / p.rho_hh;
            frozen = bs.is[inst].status >= INST_DONE ? 4 : 0;
        } else {
            sk2[j] = sc.dt / mass;
            // Gradient descent divides by damping m instead.
            sdm[j] = sc.gd ? sc.damping * mass : -sc.damping * mass / sc.rho_hh;
        }
        sflag[j] = (__ldg(m.fixed + n0 + j) ? 1 : 0) | (__ldg(sp.border + n0 + j) ? 2 : 0) | frozen;
        for (int c = 0; c < 3; ++c) {
            spos[c * ld + j] = pos[(size_t)c * N + n0 + j];
            svel[c * NT + j] = vel[(size_t)c * N + n0 + j];
            acc[3 * j + c] = 0.0;
        }
    }
    for (int j = i; j < nh; j += kTile) {
        const int n = __ldg(halo_id + j);
        for (int c = 0; c < 3; ++c) spos[c * ld + NT + j] = pos[(size_t)c * N + n];
    }
    __syncthreads();
    auto fetch = [&](int c, int slot) {
        bulk_load(nsec + slot * ns_cap, q.rec + (size_t)c * q.stride + NtSmem<MIXED>::fixed,
                  __ldg(q.chunk_bytes + c) - (uint32_t)NtSmem<MIXED>::fixed, &bar);
    };
    if (i == 0) fetch(c0, 0);
    StTables<DIAL, MIXED> tb;
    tb.load(q, sp, c0, i);
    TriMat<double> mt;
    mt.h = m.h_uniform;
    mt.mu = m.mu_uniform;
    mt.ks = m.ks_uniform;
    mt.kb = m.kb_uniform;
    mt.igmh = m.igmh_uniform;
    double lam = 0.0, pw = 0.0, nu = m.nu;
    if (DIAL == DIAL_LCE && !BATCH) {
        lam = __ldg(s.dials + 3 * (size_t)g0 + 1);
        pw = __ldg(s.dials + 3 * (size_t)g0 + 2);
    }
    uint32_t phase = 0u;
    int slot = 0;
    bool tripped = false;
    double fmax = -1.0, vmax = -1.0;
    int fnode = INT_MAX, vnode = INT_MAX;

    for (int it = 0; it < steps; ++it) {
        const bool last = it + 1 == steps;
        for (int c = c0; c < c1; ++c) {
            const int nc = c + 1 < c1 ? c + 1 : last ? -1 : c0;
            // This barrier also ends the previous chunk's runs.
            const int ok = __syncthreads_and(bar_wait(&bar, phase) ? 1 : 0);
            phase ^= 1u;
            if (!ok) {
                if (i == 0) give_up();  // no other copy is in flight
                return;
            }
            if (i == 0 && nc >= 0) fetch(nc, slot ^ 1);
            const unsigned char* ns = nsec + slot * ns_cap;
            const int4 hd = *reinterpret_cast<const int4*>(ns);  // R, E, ntri
            bool live = i < hd.z;
            if constexpr (BATCH) {
                // The chunk's triangles are of the tile's instances: each
                // touches one of its nodes.
                const StInst& o = sinst[live ? tb.tag - i_lo : 0];
                live = live && !o.frozen;
                mt.ks = o.ks;
                mt.kb = o.kb;
                mt.igmh = o.igmh;
                nu = o.nu;
                lam = o.lam[it & 1];
                pw = o.pw[it & 1];
            }
            if (live) {
                mt.area = tb.area;
                if (DIAL == DIAL_LCE) {
                    lce_metric(tb.met[0], tb.met[1], tb.met[2], __dmul_rn(lam, lam), pw, mt);
                } else {
                    constexpr int k = StTables<DIAL, MIXED>::kMet;  // 6
                    mt.abar0 = tb.met[0];
                    mt.abar1 = tb.met[1];
                    mt.abar2 = tb.met[2];
                    mt.bbar0 = tb.met[k - 3];
                    mt.bbar1 = tb.met[k - 2];
                    mt.bbar2 = tb.met[k - 1];
                }
                double P[6][3];
#pragma unroll
                for (int sl = 0; sl < 6; ++sl) {
                    const unsigned id = sl & 1 ? tb.lid[sl / 2] >> 16 : tb.lid[sl / 2] & 0xffffu;
#pragma unroll
                    for (int k = 0; k < 3; ++k) P[sl][k] = spos[k * ld + id];
                }
                R f[18];
                tri_forces<MIXED>(P, tb.cf, mt, nu, f);
#pragma unroll
                for (int k = 0; k < 18; ++k) stage[k * kTile + i] = f[k];
            }
            __syncthreads();
            if (nc >= 0) tb.load(q, sp, nc, i);
            // Runs, as in node_tile_walk.
            const unsigned short* rn = reinterpret_cast<const unsigned short*>(ns + 16);
            const unsigned short* re = rn + hd.x;
            const unsigned short* en = re + hd.x;
            for (int r = i; r < hd.x; r += kTile) {
                const int j = rn[r] & ~kRunFinal;
                int e = r ? re[r - 1] : 0;
                const int e1 = re[r];
                double a0 = acc[3 * j], a1 = acc[3 * j + 1], a2 = acc[3 * j + 2];
                for (; e < e1; ++e) {
                    const R* v = stage + en[e];
                    a0 += (double)v[0];
                    a1 += (double)v[kTile];
                    a2 += (double)v[2 * kTile];
                }
                acc[3 * j] = a0;
                acc[3 * j + 1] = a1;
                acc[3 * j + 2] = a2;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            slot ^= 1;
        }
        __syncthreads();
        if constexpr (BATCH) {
            if (!last)
                for (int k = i; k < i_n; k += kTile) {
                    const double2 d = __ldg(bs.dials + (size_t)(it + 1) * bs.n_inst + i_lo + k);
                    sinst[k].lam[(it + 1) & 1] = d.x;
                    sinst[k].pw[(it + 1) & 1] = d.y;
                }
        }
        if (DIAL == DIAL_LCE && !BATCH && !last) {
            lam = __ldg(s.dials + 3 * (size_t)(g0 + it + 1) + 1);
            pw = __ldg(s.dials + 3 * (size_t)(g0 + it + 1) + 2);
        }
        // The tile's nodes.
        const unsigned tag = tag0 + (unsigned)it + 1u;
        ulonglong2* pk = sp.packets + (tag & 1u) * 3 * (size_t)N;
        for (int j = i; j < nn; j += kTile) {
            const int flag = sflag[j];
            double dt = sc.dt, limit = sc.force_limit;
            if constexpr (BATCH) {
                const StInst& o = sinst[sni[j]];
                dt = o.dt;
                limit = o.force_limit;
            }
            double F[3], v[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                F[c] = acc[3 * j + c];
                acc[3 * j + c] = 0.0;
                v[c] = svel[c * NT + j];
                if (!sc.gd) F[c] += sdm[j] * v[c];
                if (flag & 1) F[c] = 0.0;
                double x = spos[c * ld + j];
                if (!BATCH || !(flag & 4)) {
                    if (!(fabs(F[c]) < limit) && !tripped) {
                        tripped = true;
                        if constexpr (BATCH) atomicExch(bs.trip, 1);
                        else record_guard(s, g0 + it, (long long)c * N + n0 + j);
                    }
                    double nv;
                    if (!sc.gd) nv = v[c] + sk2[j] * F[c];
                    else nv = sc.rho_hh * F[c] / sdm[j];
                    x += dt * nv;
                    if (last) {
                        pos_buf(s, sc.parity ^ 1)[(size_t)c * N + n0 + j] = x;
                        vel_buf(s, sc.parity ^ 1)[(size_t)c * N + n0 + j] = nv;
                    } else {
                        svel[c * NT + j] = nv;
                        spos[c * ld + j] = x;
                    }
                }
                if (!last && (flag & 2)) put_packet(pk + (size_t)c * N + n0 + j, x, tag);
            }
            if (sc.check && last) {
                eq_merge(fmax, fnode, sqrt(F[0] * F[0] + F[1] * F[1] + F[2] * F[2]), n0 + j);
                eq_merge(vmax, vnode, sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]), n0 + j);
            }
        }
        if (last) break;
        // Halo positions of the next step.
        int ok = 1;
        long long t0 = 0;
        int spin = 0;
        for (int k0 = i; ok && k0 < 3 * nh; k0 += kPolls * kTile) {
            int src[kPolls], dst[kPolls];
#pragma unroll
            for (int u = 0; u < kPolls; ++u) {
                const int k = k0 + u * kTile;
                src[u] = -1;
                dst[u] = 0;
                if (k < 3 * nh) {
                    const int c = k / nh, j = k - c * nh;
                    src[u] = c * N + __ldg(halo_id + j);
                    dst[u] = c * ld + NT + j;
                }
            }
            for (;;) {
                unsigned long long lo[kPolls], hi[kPolls];
                bool wait = false;
#pragma unroll
                for (int u = 0; u < kPolls; ++u)
                    if (src[u] >= 0) get_packet(pk + src[u], lo[u], hi[u]);
#pragma unroll
                for (int u = 0; u < kPolls; ++u)
                    if (src[u] >= 0) {
                        if (packet_is(lo[u], hi[u], tag)) {
                            spos[dst[u]] = packet_value(lo[u], hi[u]);
                            src[u] = -1;
                        } else {
                            wait = true;
                        }
                    }
                if (!wait) break;
                if (wait_is_over(spin++, sp.patience, t0, sp.wait)) {
                    ok = 0;
                    break;
                }
            }
        }
        if (!__syncthreads_and(ok)) {
            if (i == 0) {
                give_up();
                bar_wait(&bar, phase);  // the next step's first node section is on its way
            }
            return;
        }
    }
    if (sc.check) {
        const EqPartial r = eq_block_reduce<kTile>(fmax, fnode, vmax, vnode);
        eq_store_and_fold<kTile>(s, r, b, gridDim.x, gridDim.x);
    }
}

template <int DIAL, bool MIXED, bool BATCH>
cudaError_t prepare_one(const NodeTilePlan& q, const StreamPlan& sp, int insts, int& blocks) {
    const size_t smem = StSmem<MIXED>::bytes(q.stride, q.nodes, sp.halo, insts);
    cudaError_t e = allow_shared((const void*)k_streamed<DIAL, MIXED, BATCH>, smem);
    if (e != cudaSuccess) return e;
    int b = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_streamed<DIAL, MIXED, BATCH>, kTile, smem);
    blocks = std::min(blocks, b);
    return e;
}

template <int DIAL, bool MIXED, bool BATCH>
cudaError_t launch_one(const DevMesh& m, const NodeTilePlan& q, const StreamPlan& sp, const BatchStream& bs,
                       const DevState& s, const StepScalars& sc, int steps, unsigned tag0, cudaStream_t st) {
    if (DIAL != DIAL_LCE) {
        k_stream_metric<<<q.nchunks, kTile, 0, st>>>(m, q, sp.metric);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(q.ntiles);
    cfg.blockDim = dim3(kTile);
    cfg.dynamicSmemBytes = StSmem<MIXED>::bytes(q.stride, q.nodes, sp.halo, bs.insts);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_streamed<DIAL, MIXED, BATCH>, m, q, sp, bs, s, sc, steps, tag0);
}

}  // namespace

size_t stream_smem(size_t stride, int nodes, int halo, int insts, int mixed) {
    return mixed ? StSmem<true>::bytes(stride, nodes, halo, insts) : StSmem<false>::bytes(stride, nodes, halo, insts);
}

int stream_blocks_target(int mixed) { return mixed ? 4 : 3; }

cudaError_t prepare_streamed(const NodeTilePlan& q, const StreamPlan& sp, int insts, int mixed, int* blocks_per_sm) {
    int b = INT_MAX;
    cudaError_t e;
    if (insts > 0) {
        e = mixed ? prepare_one<DIAL_LCE, true, true>(q, sp, insts, b)
                  : prepare_one<DIAL_LCE, false, true>(q, sp, insts, b);
    } else {
        e = mixed ? prepare_one<DIAL_LCE, true, false>(q, sp, 0, b) : prepare_one<DIAL_LCE, false, false>(q, sp, 0, b);
        if (e == cudaSuccess)
            e = mixed ? prepare_one<DIAL_ARRAYS, true, false>(q, sp, 0, b)
                      : prepare_one<DIAL_ARRAYS, false, false>(q, sp, 0, b);
    }
    *blocks_per_sm = e == cudaSuccess ? b : 0;
    return e;
}

cudaError_t launch_streamed(const DevMesh& m, const NodeTilePlan& q, const StreamPlan& sp, const DevState& s,
                            const StepScalars& sc, int dial_mode, int mixed, int steps, unsigned tag0,
                            cudaStream_t st) {
    const BatchStream no{};
    if (dial_mode == DIAL_LCE)
        return mixed ? launch_one<DIAL_LCE, true, false>(m, q, sp, no, s, sc, steps, tag0, st)
                     : launch_one<DIAL_LCE, false, false>(m, q, sp, no, s, sc, steps, tag0, st);
    return mixed ? launch_one<DIAL_ARRAYS, true, false>(m, q, sp, no, s, sc, steps, tag0, st)
                 : launch_one<DIAL_ARRAYS, false, false>(m, q, sp, no, s, sc, steps, tag0, st);
}

cudaError_t launch_batch_streamed(const DevMesh& m, const NodeTilePlan& q, const StreamPlan& sp,
                                  const BatchStream& bs, const DevState& s, int parity, int mixed, int steps,
                                  unsigned tag0, cudaStream_t st) {
    StepScalars sc{};
    sc.parity = parity;
    return mixed ? launch_one<DIAL_LCE, true, true>(m, q, sp, bs, s, sc, steps, tag0, st)
                 : launch_one<DIAL_LCE, false, true>(m, q, sp, bs, s, sc, steps, tag0, st);
}

}  // namespace msb
