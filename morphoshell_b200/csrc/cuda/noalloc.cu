// Deformation forces without any device allocation (ms_deformation_forces_noalloc
// in include/morphoshell_gpu.h).
//
// Who needs it: callers that cannot call cudaMalloc -- host frameworks that
// route every device allocation through their own pool and forbid others
// (an allocation behind the pool's back breaks its accounting and can fail
// once the pool holds the memory), and real-time loops that must not
// allocate after start-up (cudaMalloc can block on the device and take
// unbounded time).  They already hold device buffers for the mesh tables, the
// positions and the forces; this entry point computes forces = -D^T dE/dcq
// from them using a fixed scratch area that lives in this library's static
// device memory.
//
// Scratch: one file-scope __device__ array sized for meshes of up to
// kMaxTris triangles and kMaxNodes nodes (about 16 MB, held by every GPU
// that loads the library until the process exits).  Larger meshes are
// rejected.  Every call shares the array and it keeps the last call's
// contents, so two calls that overlap on the GPU (different streams, or
// different host threads on the same device) race and corrupt each other;
// serialise them.  The nodes' counts are cleared at the start of every call.
//
// The node sums are deterministic: a node's entries are listed as they come
// (one atomic add each), sorted by triangle when the node is summed, and added
// in ascending triangle order, as in the main path.
//
// Two kernels: k_na_tri (lists, and the triangles' contributions) and
// k_na_gather (sort and sum).  What bounds them: the tables' one trip from HBM,
// and a node's three dependent trips to L2 (count, entries, contributions).
// Per call for 50,310 triangles: incidence lists built by counting, a one-block
// scan, filling and sorting in five more launches 114 us; entries chained, a
// dozen dependent trips along a chain, 53; listed, and the triangles' weights
// in flight together, 43.
#include <climits>
#include <cstddef>
#include <cstdio>
#include <cstring>

#include "../../../include/morphoshell_gpu.h"
#include "tri_physics.cuh"

namespace {

constexpr int kMaxTris = 65536;
constexpr int kMaxNodes = 65536;
constexpr int kListed = 32;          // entries of a node listed, and sorted in shared memory, at most
constexpr int kLists = 12 * 65536;   // room for the lists: kLists / N entries of a node (23 at T = 2 N = kMaxTris)

struct Scratch {
    double contrib[kMaxTris * 18];  // per (triangle, slot) force contribution
    int list[kLists];               // [entry of the node][N] 6 t + slot, in the order of arrival
    int next[kMaxTris * 6];         // entry 6 t + slot beyond a full list: its chain's next entry + 1, or 0
    int entries[kMaxTris * 6];      // sorted entries of the nodes with chains
    int bad;                        // patch ids outside [0, num_nodes) seen this call
    int used;                       // of entries
    int2 node[kMaxNodes];           // a node's entries, and its chain's first entry + 1, or 0 (bad, used and node are
                                    // cleared every call)
};

static __device__ __align__(256) unsigned char ms_noalloc_scratch[sizeof(Scratch)];

// Device address of the scratch array in the current context, looked up on
// every call (a table lookup once the module is loaded), so that an address
// never outlives the context it belongs to, e.g. across cudaDeviceReset.
cudaError_t scratch_address(Scratch** out) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, ms_noalloc_scratch);
    if (e != cudaSuccess) return e;
    *out = static_cast<Scratch*>(p);
    return cudaSuccess;
}

constexpr int kTriBlock = 128;
constexpr int kNodeBlock = 64;

__host__ __device__ inline int listed(int N) { return kListed < kLists / N ? kListed : kLists / N; }

__global__ void __launch_bounds__(kTriBlock)
    k_na_tri(Scratch* s, int N, int T, const int* __restrict__ patch, const double* __restrict__ coef,
             const double* __restrict__ area, const double* __restrict__ thick, const double* __restrict__ shear,
             const double* __restrict__ abar, const double* __restrict__ bbar, double nu, double gamma,
             const double* __restrict__ dofs) {
    using namespace msb::dev;
    // The block's weights in one run, then its contributions: rows of 24 and
    // 18 doubles would be 32 separate lines per warp access.
    __shared__ double rows[kTriBlock * 24];
    const int t0 = blockIdx.x * kTriBlock, i = threadIdx.x, t = t0 + i;
    const int live = min(kTriBlock, T - t0);
    // All of them on their way at once (8 bytes each: the caller's array has a
    // double's alignment), past the node lists and the positions.
    for (int e = i; e < 24 * live; e += kTriBlock)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(rows + e)),
                     "l"(coef + 24 * (size_t)t0 + e)
                     : "memory");
    double c[24], f[18], P[6][3];
    TriMat<double> m;
    if (i < live) {
        const int slots = listed(N);
        m.abar0 = abar[3 * (size_t)t];
        m.abar1 = abar[3 * (size_t)t + 1];
        m.abar2 = abar[3 * (size_t)t + 2];
        m.bbar0 = bbar[3 * (size_t)t];
        m.bbar1 = bbar[3 * (size_t)t + 1];
        m.bbar2 = bbar[3 * (size_t)t + 2];
        m.h = thick[t];
        m.mu = shear[t];
        m.area = area[t];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            int id = patch[6 * (size_t)t + k];
            if (id < 0 || id >= N) {
                // Reported; never read out of range, on no list.
                atomicAdd(&s->bad, 1);
                id = 0;
            } else {
                const int at = atomicAdd(&s->node[id].x, 1);
                if (at < slots) s->list[(size_t)at * N + id] = 6 * t + k;
                else s->next[6 * t + k] = atomicExch(&s->node[id].y, 6 * t + k + 1);
            }
            P[k][0] = dofs[id];
            P[k][1] = dofs[(size_t)N + id];
            P[k][2] = dofs[2 * (size_t)N + id];
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (i < live) {
#pragma unroll
        for (int k = 0; k < 24; ++k) c[k] = rows[24 * i + k];
        double rx[3], ry[3], rxx[3], rxy[3], ryy[3];
        for (int d = 0; d < 3; ++d) {
            rx[d] = c[0] * P[0][d] + c[1] * P[1][d] + c[2] * P[2][d];
            ry[d] = c[3] * P[0][d] + c[4] * P[1][d] + c[5] * P[2][d];
            double sxx = 0, sxy = 0, syy = 0;
            for (int k = 0; k < 6; ++k) {
                sxx += c[6 + 3 * k] * P[k][d];
                sxy += c[7 + 3 * k] * P[k][d];
                syy += c[8 + 3 * k] * P[k][d];
            }
            rxx[d] = sxx;
            rxy[d] = sxy;
            ryy[d] = syy;
        }
        Cq<double> q;
        q.rx = {rx[0], rx[1], rx[2]};
        q.ry = {ry[0], ry[1], ry[2]};
        q.rxx = {rxx[0], rxx[1], rxx[2]};
        q.rxy = {rxy[0], rxy[1], rxy[2]};
        q.ryy = {ryy[0], ryy[1], ryy[2]};
        material_coefs(m.h, m.mu, nu, gamma, m.ks, m.kb, m.igmh);
        CqGrad<double> g;
        energy_gradient<double>(q, m, nu, g);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const double mxx = c[6 + 3 * k], mxy = c[7 + 3 * k], myy = c[8 + 3 * k];
            double fx = mxx * g.rxx.x + mxy * g.rxy.x + myy * g.ryy.x;
            double fy = mxx * g.rxx.y + mxy * g.rxy.y + myy * g.ryy.y;
            double fz = mxx * g.rxx.z + mxy * g.rxy.z + myy * g.ryy.z;
            if (k < 3) {
                fx += c[k] * g.rx.x + c[3 + k] * g.ry.x;
                fy += c[k] * g.rx.y + c[3 + k] * g.ry.y;
                fz += c[k] * g.rx.z + c[3 + k] * g.ry.z;
            }
            f[3 * k] = -fx;
            f[3 * k + 1] = -fy;
            f[3 * k + 2] = -fz;
        }
    }
    __syncthreads();
    if (i < live)
#pragma unroll
        for (int k = 0; k < 18; ++k) rows[18 * i + k] = f[k];
    __syncthreads();
    double* o = s->contrib + 18 * (size_t)t0;
    for (int e = i; e < 18 * live; e += kTriBlock) o[e] = rows[e];
}

__global__ void __launch_bounds__(kNodeBlock) k_na_gather(Scratch* s, int N, double* __restrict__ forces) {
    __shared__ int list[kListed][kNodeBlock];
    const int n = blockIdx.x * kNodeBlock + threadIdx.x, i = threadIdx.x;
    if (n >= N) return;
    const int2 node = s->node[n];
    const int count = node.x, slots = listed(N);
    double fx = 0.0, fy = 0.0, fz = 0.0;
    auto add = [&](int e) {
        const double* c = s->contrib + 3 * (size_t)e;
        fx += c[0];
        fy += c[1];
        fz += c[2];
    };
    if (count <= slots) {
        // Into ascending order.  Most nodes have at most kRanked entries: loaded
        // together, their ranks counted in registers (independent compares;
        // insertion's chain of shared-memory steps, as long as the warp's worst
        // lane, took half of the kernel).
        constexpr int kRanked = 16;
        if (count <= kRanked) {
            int e[kRanked], rank[kRanked];
#pragma unroll
            for (int u = 0; u < kRanked; ++u) {
                e[u] = u < count && u < slots ? s->list[(size_t)u * N + n] : INT_MAX;
                rank[u] = 0;
            }
#pragma unroll
            for (int u = 1; u < kRanked; ++u)
#pragma unroll
                for (int w = 0; w < u; ++w) {
                    const bool after = e[w] < e[u];
                    rank[u] += after;
                    rank[w] += !after;
                }
#pragma unroll
            for (int u = 0; u < kRanked; ++u)
                if (u < count) list[rank[u]][i] = e[u];
        } else {
            for (int k = 0; k < count; ++k) {
                const int e = s->list[(size_t)k * N + n];
                int b = k;
                while (b > 0 && list[b - 1][i] > e) {
                    list[b][i] = list[b - 1][i];
                    --b;
                }
                list[b][i] = e;
            }
        }
        // Several entries' contributions are under way together.
        constexpr int kAhead = 8;
        for (int k0 = 0; k0 < count; k0 += kAhead) {
            double c[kAhead][3];
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (k0 + u < count) {
                    const double* from = s->contrib + 3 * (size_t)list[k0 + u][i];
#pragma unroll
                    for (int d = 0; d < 3; ++d) c[u][d] = from[d];
                }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (k0 + u < count) {
                    fx += c[u][0];
                    fy += c[u][1];
                    fz += c[u][2];
                }
        }
    } else {
        // The list, and the chain laid out from its end: nearly in order,
        // then insertion.
        int* a = s->entries + atomicAdd(&s->used, count);
        int k = count;
        for (int e = node.y; e != 0; e = s->next[e - 1]) a[--k] = e - 1;
        while (--k >= 0) a[k] = s->list[(size_t)k * N + n];
        for (k = 1; k < count; ++k) {
            const int e = a[k];
            int b = k;
            while (b > 0 && a[b - 1] > e) {
                a[b] = a[b - 1];
                --b;
            }
            a[b] = e;
        }
        for (k = 0; k < count; ++k) add(a[k]);
    }
    forces[n] = fx;
    forces[(size_t)N + n] = fy;
    forces[2 * (size_t)N + n] = fz;
}

void set_msg(char* err, size_t len, const char* msg) {
    if (err && len) {
        std::strncpy(err, msg, len - 1);
        err[len - 1] = 0;
    }
}

}  // namespace

extern "C" ms_status ms_deformation_forces_noalloc(int32_t num_nodes, int32_t num_tris, const int32_t* patch_ids,
                                                   const double* deriv_coeffs, const double* ref_area,
                                                   const double* ref_thickness, const double* ref_shear_modulus,
                                                   const double* abar, const double* bbar, double def_poisson_ratio,
                                                   double bend_stiffening_scale_factor, const double* dofs,
                                                   double* forces, void* stream, char* err, size_t err_len) {
    set_msg(err, err_len, "");
    if (num_nodes <= 0 || num_tris <= 0 || !patch_ids || !deriv_coeffs || !ref_area || !ref_thickness ||
        !ref_shear_modulus || !abar || !bbar || !dofs || !forces) {
        set_msg(err, err_len, "ms_deformation_forces_noalloc: null pointer or non-positive size");
        return MS_ERR_INVALID_ARGUMENT;
    }
    if (num_tris > kMaxTris || num_nodes > kMaxNodes) {
        char buf[200];
        std::snprintf(buf, sizeof buf,
                      "ms_deformation_forces_noalloc: mesh of %d nodes / %d triangles exceeds the static scratch "
                      "limit of %d nodes / %d triangles",
                      (int)num_nodes, (int)num_tris, kMaxNodes, kMaxTris);
        set_msg(err, err_len, buf);
        return MS_ERR_INVALID_ARGUMENT;
    }
    Scratch* s = nullptr;
    cudaError_t e = scratch_address(&s);
    if (e != cudaSuccess) {
        set_msg(err, err_len, cudaGetErrorString(e));
        return e == cudaErrorNoDevice ? MS_ERR_NO_DEVICE : MS_ERR_CUDA;
    }
    // An error left pending by the caller's earlier work is not this call's:
    // report it without clearing it, and launch nothing.
    e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        char buf[200];
        std::snprintf(buf, sizeof buf, "ms_deformation_forces_noalloc: a CUDA error was pending before the call (%s)",
                      cudaGetErrorString(e));
        set_msg(err, err_len, buf);
        return MS_ERR_CUDA;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int N = num_nodes, T = num_tris;
    // Each launch is checked on its own so the message names the kernel that
    // failed; the error is ours, so it is cleared.
    auto launched = [&](const char* name) -> bool {
        const cudaError_t le = cudaGetLastError();
        if (le == cudaSuccess) return true;
        char buf[200];
        std::snprintf(buf, sizeof buf, "ms_deformation_forces_noalloc: launch of %s failed (%s)", name,
                      cudaGetErrorString(le));
        set_msg(err, err_len, buf);
        return false;
    };
    e = cudaMemsetAsync(&s->bad, 0, offsetof(Scratch, node) - offsetof(Scratch, bad) + sizeof(int2) * (size_t)N, st);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_msg(err, err_len, cudaGetErrorString(e));
        return MS_ERR_CUDA;
    }
    k_na_tri<<<(T + kTriBlock - 1) / kTriBlock, kTriBlock, 0, st>>>(
        s, N, T, patch_ids, deriv_coeffs, ref_area, ref_thickness, ref_shear_modulus, abar, bbar, def_poisson_ratio,
        bend_stiffening_scale_factor, dofs);
    if (!launched("k_na_tri")) return MS_ERR_CUDA;
    k_na_gather<<<(N + kNodeBlock - 1) / kNodeBlock, kNodeBlock, 0, st>>>(s, N, forces);
    if (!launched("k_na_gather")) return MS_ERR_CUDA;
    // Wait for the result and check the ids (a plain host int: no allocation).
    int bad = 0;
    e = cudaMemcpyAsync(&bad, &s->bad, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        set_msg(err, err_len, cudaGetErrorString(e));
        return MS_ERR_CUDA;
    }
    if (bad) {
        set_msg(err, err_len, "ms_deformation_forces_noalloc: patch ids outside [0, num_nodes); forces incomplete");
        return MS_ERR_INVALID_ARGUMENT;
    }
    return MS_OK;
}
