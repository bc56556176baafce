// Resident step: many fused steps in one launch, for meshes whose triangles
// fit one thread each on the device.
//
// The nodes (Morton order) are cut into at most one tile of consecutive
// nodes per SM, one block per tile.  A block computes every triangle whose
// patch touches one of its nodes, one thread per triangle, and keeps what
// does not change between steps on chip for the whole launch: the triangle's
// weights and director trigonometry in its thread's registers, the tile's
// positions and its halo's (the other nodes of its triangles' patches) in
// shared memory, a node component's velocity, mass terms and flags in the
// registers of the thread that updates it.  A step is then
//   triangles   18 contributions per thread, from positions in shared
//               memory, staged field-major in shared memory;
//   nodes       one thread per node component: its contributions in
//               ascending triangle order from zero (the order, and so the
//               bits, of the node kernel's gather), damping, constraint,
//               force guard, symplectic Euler (the arithmetic of node_core);
//   exchange    a node that other tiles read is published as three 16-byte
//               packets, and each halo component is polled from its owner's
//               packet.  Both 8-byte halves of a packet carry the step's tag
//               beside half of the double, so a packet is complete when both
//               tags match: no fence, no flag and no grid-wide barrier, one
//               trip through L2 per step.
// What bounds it: latency.  Of a step of the 18,086-triangle disk (147 tiles
// of 63 nodes, 256 threads) about 1,750 SM clocks go to the triangles (two
// FP64 warps on each sub-partition; 1,000 with one), 800 to the nodes'
// dependent sums and 1,400 to the trip of a position through L2.  Per step
// against the two-kernel step captured in graphs (FP64 / mixed): 687
// triangles 1.9 / 1.8 us against 8.0 / 7.6, 18,086 triangles 2.6 / 2.4
// against 9.3 / 8.5, 32,219 triangles 3.4 / 3.0 against 9.9 / 9.1.
//
// Packets are double-buffered by the tag's parity.  Tile adjacency is
// symmetric (a triangle that makes A read a node of B touches nodes of both,
// so B computes it and reads A), and a block publishes step s + 1 only after
// all its threads have read step s of its halo; a tile that overwrites a
// step-s packet has read step s + 1 of every tile that could still want it.
//
// The launch is cooperative, so its blocks are resident together.  Every
// wait is bounded (about a second of SM clock); a block that gives up
// records it and returns, and so do its neighbours in turn.  The state the
// launch starts from stays untouched in its buffer (only the last step writes
// the other one), so the steps of a launch that tripped the force guard or
// was given up run again one by one: the call gives the same result, and finds
// and reports the step that trips.
#include <algorithm>
#include <climits>

#include "internal.cuh"
#include "packets.cuh"
#include "step_common.cuh"
#include "tri_contrib.cuh"

namespace msb {
namespace {

using namespace packets;
using namespace stepdev;
using namespace tridev;

// Threads of a block: one per triangle slot and, in the node phase, one per
// node component.  Up to 256 threads a thread may hold 255 registers; at 384,
// 168 (as the node-tiled step's, a few bytes of spills in FP64).
constexpr int kLarge = 384;
constexpr int kHaloItems = 2;  // halo components a thread polls at most
constexpr int kHeld = 16;      // entries of a node kept in registers
constexpr int kBatch = 8;      // of which this many are loaded together
// SM clocks from a node's update to its thread's first poll: the trip
// through L2 takes longer, and a poll that comes too early costs one more.
// Per step with 0 / 200 / 400 / 500 / 600 / 700 clocks: 687 triangles 1.91 /
// 1.89 / 1.81 / 1.80 / 1.86 / 1.90 us, 18,086 triangles 2.58 / 2.55 / 2.50 /
// 2.49 / 2.48 / 2.46 us, 32,219 triangles 3.57 / 3.49 / 3.40 / 3.38 / 3.35 /
// 3.36 us.
constexpr unsigned kFirstPoll = 500;

template <int DIAL, bool MIXED, int TH>
__global__ void __launch_bounds__(TH, 1)
    k_resident(const DevMesh m, const ClusterPlan p, const ResidentPlan q, const DevState s, const StepScalars sc,
               int steps, unsigned tag0) {
    using R = typename Real<MIXED>::T;
    const int g0 = global_step(s.err, sc.step);
    // An earlier launch tripped the guard or was given up: uniform over the grid.
    if (stale(s.err, g0)) return;
    extern __shared__ __align__(16) unsigned char rs_smem[];
    constexpr int S = TH;
    const int NT = q.nodes, N = m.N;
    const int ld = NT + q.halo;  // positions per component: own nodes, then the halo
    R* stage = reinterpret_cast<R*>(rs_smem);                          // [18][S]
    double* spos = reinterpret_cast<double*>(rs_smem + 18 * sizeof(R) * S);  // [3][ld]
    double* sfv = spos + 3 * ld;                                       // [6][NT]: F and v of a check step
    unsigned short* sent = reinterpret_cast<unsigned short*>(sfv + 6 * NT);  // [width][NT]

    // At 168 registers a thread's area and metric terms wait in shared memory.
    constexpr bool kSpare = TH <= 256;
    __shared__ double smet[kSpare ? 1 : 7][kSpare ? 1 : TH];

    const int b = blockIdx.x, i = threadIdx.x;
    const int n0 = b * NT, nn = min(NT, N - n0);
    const int4 hd = __ldg(q.head + b);  // triangles, halo nodes
    const double* pos = pos_buf(s, sc.parity);
    const double* vel = vel_buf(s, sc.parity);

    // This thread's triangle: tables in registers for the whole launch.
    const bool live = i < hd.x;
    int lid[6];
    R c[24];
    double area = 0.0, m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0, m4 = 0.0, m5 = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) lid[k] = 0;
#pragma unroll
    for (int k = 0; k < 24; ++k) c[k] = R(0);
    if (live) {
        const int t = __ldg(q.tri + (size_t)b * S + i);
#pragma unroll
        for (int k = 0; k < 6; ++k) lid[k] = __ldg(q.local + ((size_t)b * 6 + k) * S + i);
        if constexpr (MIXED) {
#pragma unroll
            for (int k = 0; k < 24; ++k) c[k] = __ldg(p.coef_aos_f + 24 * (size_t)t + k);
        } else {
#pragma unroll
            for (int k = 0; k < 24; ++k) c[k] = __ldg(p.coef_aos + 24 * (size_t)t + k);
        }
        area = __ldg(m.area + t);
        if (DIAL == DIAL_LCE) {
            const double2* ap = reinterpret_cast<const double2*>(p.tri_aux + t);
            const double2 a01 = __ldg(ap), a23 = __ldg(ap + 1);
            m0 = a01.y;
            m1 = a23.x;
            m2 = a23.y;
        } else {
            const size_t T = m.T;
            m0 = __ldg(m.abar + t);
            m1 = __ldg(m.abar + T + t);
            m2 = __ldg(m.abar + 2 * T + t);
            m3 = __ldg(m.bbar + t);
            m4 = __ldg(m.bbar + T + t);
            m5 = __ldg(m.bbar + 2 * T + t);
        }
    }
    if constexpr (!kSpare) {
        const double mv[7] = {m0, m1, m2, m3, m4, m5, area};
#pragma unroll
        for (int k = 0; k < 7; ++k) smet[k][i] = mv[k];
    }
    // This thread's node component.
    const int nc = i / NT, nj = i - nc * NT;
    const bool owner = nc < 3 && nj < nn;
    double v = 0.0, k2 = 0.0, dm = 0.0, gden = 0.0;
    bool fixed = false, border = false;
    int width = 0;
    if (owner) {
        const int n = n0 + nj;
        v = vel[(size_t)nc * N + n];
        const double mass = __ldg(m.mass + n);
        k2 = sc.dt / mass;
        dm = -sc.damping * mass / sc.rho_hh;
        gden = sc.damping * mass;
        fixed = __ldg(m.fixed + n) != 0;
        border = __ldg(q.border + n) != 0;
        width = __ldg(q.count + n);
        spos[nc * ld + nj] = pos[(size_t)nc * N + n];
    }
    // Its first kHeld entries, two to a register where there is room; the
    // rest in shared memory.
    unsigned held[kHeld / 2];
#pragma unroll
    for (int k = 0; k < kHeld / 2; ++k) held[k] = 0;
    for (int k = i; k < q.width * NT; k += S) sent[k] = q.entries[(size_t)b * q.width * NT + k];
    __syncthreads();
    if (kSpare && owner) {
#pragma unroll
        for (int k = 0; k < kHeld; ++k)
            if (k < width) held[k / 2] |= (unsigned)sent[k * NT + nj] << (16 * (k & 1));
    }
    const int wmax = __reduce_max_sync(0xffffffffu, width);
    // This thread's halo components.
    int hsrc[kHaloItems], hdst[kHaloItems];
#pragma unroll
    for (int u = 0; u < kHaloItems; ++u) {
        const int k = i + u * S;
        hsrc[u] = -1;
        hdst[u] = 0;
        if (k < 3 * hd.y) {
            const int hc = k / hd.y, hj = k - hc * hd.y;
            const int n = __ldg(q.halo_id + (size_t)b * q.halo + hj);
            hsrc[u] = hc * N + n;
            hdst[u] = hc * ld + NT + hj;
            spos[hdst[u]] = pos[hsrc[u]];
        }
    }
    TriMat<double> mt;
    mt.h = m.h_uniform;
    mt.mu = m.mu_uniform;
    mt.ks = m.ks_uniform;
    mt.kb = m.kb_uniform;
    mt.igmh = m.igmh_uniform;
    double lam = 0.0, pw = 0.0;
    if (DIAL == DIAL_LCE) {
        lam = __ldg(s.dials + 3 * (size_t)g0 + 1);
        pw = __ldg(s.dials + 3 * (size_t)g0 + 2);
    }
    bool tripped = false;
    __syncthreads();

    for (int it = 0; it < steps; ++it) {
        const bool last = it + 1 == steps;
        if (live) {
            auto met = [&](int k, double reg) { return kSpare ? reg : smet[kSpare ? 0 : k][kSpare ? 0 : i]; };
            mt.area = met(6, area);
            if (DIAL == DIAL_LCE) {
                lce_metric(met(0, m0), met(1, m1), met(2, m2), __dmul_rn(lam, lam), pw, mt);
            } else {
                mt.abar0 = met(0, m0);
                mt.abar1 = met(1, m1);
                mt.abar2 = met(2, m2);
                mt.bbar0 = met(3, m3);
                mt.bbar1 = met(4, m4);
                mt.bbar2 = met(5, m5);
            }
            double P[6][3];
#pragma unroll
            for (int sl = 0; sl < 6; ++sl)
#pragma unroll
                for (int k = 0; k < 3; ++k) P[sl][k] = spos[k * ld + lid[sl]];
            R f[18];
            tri_forces<MIXED>(P, c, mt, m.nu, f);
#pragma unroll
            for (int k = 0; k < 18; ++k) stage[k * S + i] = f[k];
        }
        __syncthreads();
        // The next step's dial values load while the nodes are summed.
        if (DIAL == DIAL_LCE && !last) {
            lam = __ldg(s.dials + 3 * (size_t)(g0 + it + 1) + 1);
            pw = __ldg(s.dials + 3 * (size_t)(g0 + it + 1) + 2);
        }
        const unsigned tag = tag0 + (unsigned)it + 1u;
        ulonglong2* pk = q.packets + (tag & 1u) * 3 * (size_t)N;
        if (owner) {
            // Contributions in ascending triangle order; kBatch loads in
            // flight ahead of the adds, which depend on one another.
            const R* st = stage + nc * S;
            double F = 0.0;
#pragma unroll
            for (int k0 = 0; k0 < kHeld; k0 += kBatch) {
                if (k0 < wmax) {
                    R val[kBatch];
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        unsigned e = 0;
                        if constexpr (kSpare) e = (held[(k0 + k) / 2] >> (16 * (k & 1))) & 0xffffu;
                        else if (k0 + k < width) e = sent[(k0 + k) * NT + nj];
                        val[k] = st[e];
                    }
#pragma unroll
                    for (int k = 0; k < kBatch; ++k)
                        if (k0 + k < width) F += (double)val[k];
                }
            }
            for (int k = kHeld; k < width; ++k) F += (double)st[sent[k * NT + nj]];
            if (!sc.gd) F += dm * v;
            if (fixed) F = 0.0;
            if (sc.check && last) {
                sfv[nc * NT + nj] = F;
                sfv[(3 + nc) * NT + nj] = v;
            }
            if (!(fabs(F) < sc.force_limit) && !tripped) {
                tripped = true;
                record_guard(s, g0 + it, (long long)nc * N + n0 + nj);
            }
            double nv;
            if (!sc.gd) nv = v + k2 * F;
            else nv = sc.rho_hh * F / gden;
            const double x = spos[nc * ld + nj] + sc.dt * nv;
            v = nv;
            if (last) {
                pos_buf(s, sc.parity ^ 1)[(size_t)nc * N + n0 + nj] = x;
                vel_buf(s, sc.parity ^ 1)[(size_t)nc * N + n0 + nj] = nv;
            } else {
                spos[nc * ld + nj] = x;
                if (border) put_packet(pk + (size_t)nc * N + n0 + nj, x, tag);
            }
        }
        if (last) break;
        // Halo positions of the next step.
        int ok = 1;
        {
            bool need[kHaloItems];
#pragma unroll
            for (int u = 0; u < kHaloItems; ++u) need[u] = hsrc[u] >= 0;
            long long t0 = 0;
            const unsigned c0 = (unsigned)clock();
            while ((unsigned)clock() - c0 < kFirstPoll) {
            }
            for (int spin = 0;; ++spin) {
                unsigned long long lo[kHaloItems], hi[kHaloItems];
                bool wait = false;
#pragma unroll
                for (int u = 0; u < kHaloItems; ++u)
                    if (need[u]) get_packet(pk + hsrc[u], lo[u], hi[u]);
#pragma unroll
                for (int u = 0; u < kHaloItems; ++u)
                    if (need[u]) {
                        if (packet_is(lo[u], hi[u], tag)) {
                            spos[hdst[u]] = packet_value(lo[u], hi[u]);
                            need[u] = false;
                        } else {
                            wait = true;
                        }
                    }
                if (!wait) break;
                if (wait_is_over(spin, q.patience, t0, q.wait)) {
                    ok = 0;
                    break;
                }
            }
        }
        if (!__syncthreads_and(ok)) {
            if (i == 0) record_timeout(s, g0);
            return;
        }
    }
    if (sc.check) {
        __syncthreads();
        double f = -1.0, w = -1.0;
        int fn = INT_MAX, wn = INT_MAX;
        if (i < nn) {
            const double Fx = sfv[i], Fy = sfv[NT + i], Fz = sfv[2 * NT + i];
            const double vx = sfv[3 * NT + i], vy = sfv[4 * NT + i], vz = sfv[5 * NT + i];
            eq_merge(f, fn, sqrt(Fx * Fx + Fy * Fy + Fz * Fz), n0 + i);
            eq_merge(w, wn, sqrt(vx * vx + vy * vy + vz * vz), n0 + i);
        }
        const EqPartial r = eq_block_reduce<TH>(f, fn, w, wn);
        eq_store_and_fold<TH>(s, r, b, gridDim.x, gridDim.x);
    }
}

size_t smem_bytes(const ResidentPlan& q, int mixed) {
    return (size_t)18 * (mixed ? 4 : 8) * q.threads + 24 * (size_t)(q.nodes + q.halo) + 48 * (size_t)q.nodes +
           2 * (size_t)q.width * q.nodes;
}

template <int DIAL, bool MIXED, int TH>
cudaError_t prepare_one(const ResidentPlan& q, int& blocks) {
    const size_t smem = smem_bytes(q, MIXED);
    cudaError_t e = allow_shared((const void*)k_resident<DIAL, MIXED, TH>, smem);
    if (e != cudaSuccess) return e;
    int b = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_resident<DIAL, MIXED, TH>, q.threads, smem);
    blocks = std::min(blocks, b);
    return e;
}

template <int DIAL, bool MIXED>
cudaError_t prepare_th(const ResidentPlan& q, int& blocks) {
    return q.threads == 128   ? prepare_one<DIAL, MIXED, 128>(q, blocks)
           : q.threads == 256 ? prepare_one<DIAL, MIXED, 256>(q, blocks)
                              : prepare_one<DIAL, MIXED, kLarge>(q, blocks);
}

template <int DIAL, bool MIXED, int TH>
cudaError_t launch_one(const DevMesh& m, const ClusterPlan& p, const ResidentPlan& q, const DevState& s,
                       const StepScalars& sc, int steps, unsigned tag0, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(q.ntiles);
    cfg.blockDim = dim3(q.threads);
    cfg.dynamicSmemBytes = smem_bytes(q, MIXED);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_resident<DIAL, MIXED, TH>, m, p, q, s, sc, steps, tag0);
}

template <int DIAL, bool MIXED>
cudaError_t launch_th(const DevMesh& m, const ClusterPlan& p, const ResidentPlan& q, const DevState& s,
                      const StepScalars& sc, int steps, unsigned tag0, cudaStream_t st) {
    return q.threads == 128   ? launch_one<DIAL, MIXED, 128>(m, p, q, s, sc, steps, tag0, st)
           : q.threads == 256 ? launch_one<DIAL, MIXED, 256>(m, p, q, s, sc, steps, tag0, st)
                              : launch_one<DIAL, MIXED, kLarge>(m, p, q, s, sc, steps, tag0, st);
}

// Which of n items are in which of K tiles, a bit each.
struct TileBits {
    size_t words = 0;
    std::vector<unsigned long long> bits;
    void clear(int K, int n) {
        words = ((size_t)n + 63) / 64;
        bits.assign(K * words, 0);
    }
    void set(int k, int i) { bits[k * words + i / 64] |= 1ULL << (i % 64); }
    // A tile's items, ascending.
    template <typename F>
    void each(int k, F f) const {
        for (size_t w = 0; w < words; ++w)
            for (unsigned long long b = bits[k * words + w]; b; b &= b - 1) f((int)(64 * w) + __builtin_ctzll(b));
    }
    int most(int K) const {
        int m = 0;
        for (int k = 0; k < K; ++k) {
            int c = 0;
            for (size_t w = 0; w < words; ++w) c += __builtin_popcountll(bits[k * words + w]);
            m = std::max(m, c);
        }
        return m;
    }
};

// Tiles of NT nodes: each tile's triangles and halo nodes, and the most of each
// a tile has.  Bits need no look whether a triangle or node is on a list
// already, and no sort: the plan of 18,086 triangles takes 1.1 ms, with
// sorted lists 3.2.
struct Cut {
    int K = 0, tris = 0, halo = 0;
    TileBits tri, hal;
};

Cut cut_tiles(const int* patch, int N, int T, int NT) {
    Cut x;
    x.K = (N + NT - 1) / NT;
    std::vector<int> tile(N);
    for (int k = 0; k < x.K; ++k) std::fill(tile.begin() + k * NT, tile.begin() + std::min(N, (k + 1) * NT), k);
    x.tri.clear(x.K, T);
    x.hal.clear(x.K, N);
    for (int t = 0; t < T; ++t) {
        const int* p = patch + 6LL * t;
        int k[6], differ = 0;
        for (int j = 0; j < 6; ++j) {
            k[j] = tile[p[j]];
            differ |= k[j] ^ k[0];
            x.tri.set(k[j], t);
        }
        if (!differ) continue;
        for (int j = 0; j < 6; ++j)
            if (j == 0 || k[j] != k[j - 1])
                for (int i = 0; i < 6; ++i)
                    if (k[i] != k[j]) x.hal.set(k[j], p[i]);
    }
    x.tris = x.tri.most(x.K);
    x.halo = x.hal.most(x.K);
    return x;
}

int threads_for(const Cut& x, int NT) { return (std::max(x.tris, 3 * NT) + 127) / 128 * 128; }

}  // namespace

bool resident_layout(const int* patch, int N, int T, int sms, const std::vector<int>& off, const std::vector<int>& ent,
                     ResidentLayout& L) {
    L = ResidentLayout();
    // A tile needs at least a thread per node component, and a triangle's
    // thread; far larger meshes are not looked at further.
    if (N > sms * (kLarge / 3) || T > sms * kLarge) return false;
    auto fits = [&](const Cut& x, int NT) {
        const int th = threads_for(x, NT);
        return th <= kLarge && 3 * x.halo <= kHaloItems * th;
    };
    int NT = (N + sms - 1) / sms;
    Cut x = cut_tiles(patch, N, T, NT);
    // Small meshes: larger tiles on fewer SMs as long as a block stays at
    // four warps, one per SM sub-partition; a step then takes no longer and
    // fewer tiles exchange.  (A tile's triangles grow with its nodes, so the
    // largest such tile is found by halving.)
    if (threads_for(x, NT) <= 128) {
        for (int lo = NT, hi = 128 / 3 + 1; hi - lo > 1;) {
            const int mid = (lo + hi) / 2;
            Cut y = cut_tiles(patch, N, T, mid);
            if (threads_for(y, mid) <= 128 && fits(y, mid)) {
                lo = NT = mid;
                x = std::move(y);
            } else {
                hi = mid;
            }
        }
    }
    if (!fits(x, NT)) return false;
    L.nodes = NT;
    L.ntiles = x.K;
    L.halo = std::max(1, x.halo);
    L.threads = threads_for(x, NT);
    const int S = L.threads;
    for (int n = 0; n < N; ++n) L.width = std::max(L.width, off[n + 1] - off[n]);
    if (L.width > 255) return false;  // counts are bytes
    L.head.assign(4ULL * x.K, 0);
    L.tri.assign((size_t)x.K * S, 0);
    L.local.assign((size_t)x.K * 6 * S, 0);
    L.halo_id.assign((size_t)x.K * L.halo, 0);
    L.entries.assign((size_t)x.K * L.width * NT, 0);
    L.border.assign(N, 0);
    L.count.assign(N, 0);
    std::vector<int> slot(T, 0), place(N, 0);  // of the current tile's triangles, its nodes and its halo
    for (int k = 0; k < x.K; ++k) {
        const int n0 = k * NT, n1 = std::min(N, n0 + NT);
        for (int n = n0; n < n1; ++n) place[n] = n - n0;
        int nh = 0, nt = 0;
        x.hal.each(k, [&](int n) {
            place[n] = NT + nh;
            L.halo_id[(size_t)k * L.halo + nh++] = n;
            L.border[n] = 1;
        });
        x.tri.each(k, [&](int t) {
            slot[t] = nt;
            L.tri[(size_t)k * S + nt] = t;
            for (int j = 0; j < 6; ++j) L.local[((size_t)k * 6 + j) * S + nt] = (unsigned short)place[patch[6LL * t + j]];
            ++nt;
        });
        L.head[4ULL * k] = nt;
        L.head[4ULL * k + 1] = nh;
        for (int n = n0; n < n1; ++n) {
            L.count[n] = (unsigned char)(off[n + 1] - off[n]);
            for (int e = off[n]; e < off[n + 1]; ++e)
                L.entries[((size_t)k * L.width + (e - off[n])) * NT + (n - n0)] =
                    (unsigned short)(3 * (ent[e] % 6) * S + slot[ent[e] / 6]);
        }
    }
    return true;
}

cudaError_t prepare_resident(const ResidentPlan& q, int mixed, int* blocks_per_sm) {
    int b = INT_MAX;
    cudaError_t e = mixed ? prepare_th<DIAL_LCE, true>(q, b) : prepare_th<DIAL_LCE, false>(q, b);
    if (e == cudaSuccess) e = mixed ? prepare_th<DIAL_ARRAYS, true>(q, b) : prepare_th<DIAL_ARRAYS, false>(q, b);
    *blocks_per_sm = e == cudaSuccess ? b : 0;
    return e;
}

cudaError_t launch_resident(const DevMesh& m, const ClusterPlan& p, const ResidentPlan& q, const DevState& s,
                            const StepScalars& sc, int dial_mode, int mixed, int steps, unsigned tag0,
                            cudaStream_t st) {
    if (dial_mode == DIAL_LCE)
        return mixed ? launch_th<DIAL_LCE, true>(m, p, q, s, sc, steps, tag0, st)
                     : launch_th<DIAL_LCE, false>(m, p, q, s, sc, steps, tag0, st);
    return mixed ? launch_th<DIAL_ARRAYS, true>(m, p, q, s, sc, steps, tag0, st)
                 : launch_th<DIAL_ARRAYS, false>(m, p, q, s, sc, steps, tag0, st);
}

}  // namespace msb
