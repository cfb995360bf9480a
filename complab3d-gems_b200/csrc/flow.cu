// flow.cu -- D3Q19 incompressible BGK flow lattice on the AA in-place pattern.
//
// Reference behaviour (Palabos dynamics installed by NSdomainSetup,
// complab_functions.hh:296-345, driven by complab.cpp:1095-1206):
//   IncBGK collision with per-material omega (pore, biofilm: omega_bio =
//   1/(permRatio (1/omega - 1/2) + 1/2), :323), BounceBack walls (full-way: populations are
//   held one step in the wall node), NoDynamics solids (no collision, populations stream
//   through), Palabos' local regularized density boundary on the planes x = 0 (rho = 1) and
//   x = nx-1 (rho = 1 - 3 dP), reflection of populations whose source lies outside the box.
//
// Layout: only collide-or-stream nodes are stored (sparse.cuh): f[19][K] of the storage type
// in lexicographic node order, plus one link slot per (node, direction into a wall). One array,
// updated in place with the AA pattern:
//   even step: node a reads f[i][a], collides, writes outgoing i to f[opp(i)][a];
//   odd step:  node a reads incoming i from f[opp(i)][a - c_i], collides, writes outgoing
//              i to f[i][a + c_i].
// Each slot is read and written by exactly one node per step, so a step needs no second array
// and no synchronisation. A full-way bounce-back node is the identity on its AA slots, so it is
// never launched; each link from a stored node into a wall is a two-step delay line held in the
// node's own opposite slot on odd steps and in a link slot on even steps (sparse.cuh). A source
// or destination outside the box maps to the node's own opposite slot: Palabos' reflection at the
// block edge. The even step touches only the node's own slots and its link slots; the odd step
// gathers and scatters through the precomputed neighbour-row offsets and writes every stored slot
// exactly once.
//
// Algorithmic bytes per node update: 2 * 19 * sizeof(storage). Metadata read per node: 1 byte
// material code and 4 bytes wall mask + link offset (even step); 1 byte code, 8 bytes masks and
// 16 bytes neighbour-row offsets (odd step).
#include "batch.cuh"
#include "flow_node.cuh"
#include "grid_sync.cuh"
#include "step_chain.cuh"
#include "tma.cuh"

#include <algorithm>
#include <cstddef>
#include <type_traits>
#include <vector>
#include <cmath>
#include <cstring>

namespace clb {

constexpr int FLOW_THREADS = 256;
constexpr int PIPE_THREADS = 256;  // CTA of the pipelined odd step (shared memory per thread: 2 nodes)


// Block-wide FP64 sum; result valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0;
    if (threadIdx.x == 0)
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) r += sh[k];
    __syncthreads();
    return r;
}

// The stored average energy of a step from its sum of |u|^2, `count` iterations, and the tracer: by every
// thread of the step's last block.
__device__ void settle_step(Tracer* tr, double tot, int64_t n_bgk, int trace, int count) {
    __shared__ double sh[32];
    double v;
    __shared__ double s_mean;
    __shared__ int s_count;
    if (threadIdx.x == 0) {
        double e = n_bgk > 0 ? 0.5 * tot / (double)n_bgk : 0.0;
        tr->energy = e;
        tr->iterations += count;
        tr->done_blocks = 0;
        s_count = 0;
        if (trace) {
            tr->ring[tr->head] = e;
            tr->head = (tr->head + 1) % TRACER_WINDOW;
            if (tr->count < TRACER_WINDOW) tr->count += 1;
            s_count = tr->count;
        }
    }
    __syncthreads();
    if (!trace || s_count < TRACER_WINDOW) return;
    v = 0;
    for (int k = threadIdx.x; k < TRACER_WINDOW; k += blockDim.x) v += tr->ring[k];
    double sum = block_sum(v, sh);
    if (threadIdx.x == 0) s_mean = sum / (double)TRACER_WINDOW;
    __syncthreads();
    v = 0;
    for (int k = threadIdx.x; k < TRACER_WINDOW; k += blockDim.x) {
        double d = tr->ring[k] - s_mean;
        v += d * d;
    }
    double sq = block_sum(v, sh);
    if (threadIdx.x == 0) {
        double sd = sqrt(sq / (double)(TRACER_WINDOW - 1));
        double r = sd / s_mean;
        if (isnan(r) || fabs(r) < tr->eps) tr->converged = 1;
    }
}

// The last block of a step turns the partial sums into the stored average energy and runs
// the tracer. Deterministic: fixed grid, fixed reduction order.
__device__ void finish_step(Tracer* tr, double* partials, double block_total, int64_t n_bgk, int trace, int count = 1) {
    __shared__ bool s_last;
    __shared__ double sh[32];
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = block_total;
        __threadfence();
        unsigned t = atomicAdd(&tr->done_blocks, 1u);
        s_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double v = 0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) v += ((volatile double*)partials)[k];
    double tot = block_sum(v, sh);
    settle_step(tr, tot, n_bgk, trace, count);
}

// Odd AA step with the gathers of the next node in flight while a node is collided: each thread
// stages a node's 19 incoming populations in its own two shared-memory slots with asynchronous
// copies (4- and 8-byte storage), one node ahead, and the node after that has its metadata
// loading. The odd step is an in-place permutation: outgoing population j of node k goes to the
// slot incoming opp(j) came from, so the 19 slot offsets computed for the gathers are kept in
// registers (two sets, the loop unrolled by two nodes) and reused by the stores. Same arithmetic
// as the plain step.
template <typename TS, typename TC, int MINB>
__global__ void __launch_bounds__(PIPE_THREADS, MINB)
    k_flow_odd_pipe(TS* __restrict__ f, TS* __restrict__ link, const SparseView S, const FlowParams P,
                    Tracer* __restrict__ tr, double* __restrict__ partials, int trace, int64_t k_west_end,
                    int64_t k_east_begin) {
    if (trace && tr->converged) return;
    extern __shared__ __align__(16) unsigned char flow_smem[];
    const int tid = threadIdx.x, nt = blockDim.x;
    TS* buf = reinterpret_cast<TS*>(flow_smem);  // [2][19][nt]
    const int64_t K = S.K;
    const uint32_t K32 = (uint32_t)S.KS;
    const int64_t stride = (int64_t)gridDim.x * nt;
    double esum = 0;
    uint32_t A[19], B[19];
    auto issue = [&](int64_t kk, const FlowMeta& M, int q, uint32_t (&ad)[19]) {
        const OddRows R = odd_rows(S, kk, M);
        TS* dst = buf + (q * 19) * nt + tid;
#pragma unroll
        for (int i = 0; i < 19; ++i) {
            ad[i] = odd_src(i, kk, R, K32);
            cp_async<sizeof(TS)>(dst + i * nt, f + ad[i]);
        }
    };
    int64_t k = (int64_t)blockIdx.x * nt + tid;
    FlowMeta cur, nxt;
    if (k < K) {
        cur = flow_meta<true>(S, k);
        issue(k, cur, 0, A);
    }
    cp_async_commit();
    int64_t kn = k + stride;
    if (kn < K) nxt = flow_meta<true>(S, kn);
    // one node: gathers of the next node issued into the other slot, then this node collided
    auto node = [&](int q, uint32_t (&ac)[19], uint32_t (&an)[19]) {
        if (kn < K) issue(kn, nxt, q ^ 1, an);
        cp_async_commit();
        const int64_t knn = kn + stride;
        FlowMeta nn;
        if (knn < K) nn = flow_meta<true>(S, knn);
        cp_async_wait_group<1>();  // this node's populations have landed
        const int code = cur.code;
        if (P.dyn[code] != DYN_BB) {  // a stored bounce-back node: identity on AA slots
            TC g[19];
            const TS* src = buf + (q * 19) * nt + tid;
#pragma unroll
            for (int i = 0; i < 19; ++i) g[i] = ld<TS, TC>(src + i * nt);
            if (P.dyn[code] == DYN_BGK) {
                if (k < k_west_end) regularize19<TC>(g, -1, (TC)(P.rho_w - 1.0));
                else if (k >= k_east_begin) regularize19<TC>(g, 1, (TC)(P.rho_e - 1.0));
                esum += (double)bgk19<TC>(g, (TC)P.omega[code]);
            }
#pragma unroll
            for (int i = 0; i < 19; ++i) st<TS, TC>(f + ac[q19opp(i)], g[i]);
        }
        k = kn;
        kn = knn;
        cur = nxt;
        nxt = nn;
    };
    while (k < K) {
        node(0, A, B);
        if (k >= K) break;
        node(1, B, A);
    }
    cp_async_wait_group<0>();
    __shared__ double sh[32];
    double bt = block_sum(esum, sh);
    finish_step(tr, partials, bt, P.n_bgk, trace);
}

template <typename TS, typename TC, bool ODD, int MINB>
__global__ void __launch_bounds__(FLOW_THREADS, MINB)
    k_flow_aa(TS* __restrict__ f, TS* __restrict__ link, const SparseView S, const FlowParams P,
              Tracer* __restrict__ tr, double* __restrict__ partials, int trace, int64_t k_west_end,
              int64_t k_east_begin) {
    if (trace && tr->converged) return;  // a batch continues past convergence as no-ops
    const int64_t K = S.K;
    double esum = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    FlowMeta cur;
    if (k < K) cur = flow_meta<ODD>(S, k);
    while (k < K) {
        const int64_t kn = k + stride;
        FlowMeta nxt;
        if (kn < K) nxt = flow_meta<ODD>(S, kn);  // the next node's metadata in flight meanwhile
        esum += flow_node_m<TS, TC, ODD>(f, link, S, P, k, k_west_end, k_east_begin, cur);
        cur = nxt;
        k = kn;
    }
    __shared__ double sh[32];
    double bt = block_sum(esum, sh);
    finish_step(tr, partials, bt, P.n_bgk, trace);
}


// Even AA step through shared memory: a persistent CTA walks 256-node tiles; one thread moves the
// tile's 19 population rows (contiguous, 16-byte aligned thanks to the padded row stride) into
// shared memory with bulk copies completing on an mbarrier, keeping NSTAGE-1 tiles in flight
// ahead of the one being collided. Each thread collides its node in place in shared memory; the
// rows go back with bulk stores. A wall link (a, i) takes its incoming opp(i) from its even-step
// slot X (a global load issued alongside the tile's), writes outgoing i to X, and leaves its
// odd-step slot Y = f[opp(i)][a] untouched in the tile, so the bulk store rewrites it unchanged.
constexpr int NSTAGE = 2;  // 2 stages x 4 resident CTAs (4-byte storage) beat 3 x 3 on B200

template <typename TS, typename TC>
__global__ void __launch_bounds__(TILE, sizeof(TS) == 8 ? 2 : 4)
    k_flow_even_tma(TS* __restrict__ f, TS* __restrict__ link, const SparseView S, const FlowParams P,
                    Tracer* __restrict__ tr, double* __restrict__ partials, int trace, int64_t k_west_end,
                    int64_t k_east_begin) {
    if (trace && tr->converged) return;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    TS* stages = reinterpret_cast<TS*>(smem_raw);
    __shared__ __align__(8) uint64_t full[NSTAGE];
    __shared__ int s_abort;
    const int tid = threadIdx.x;
    const int64_t K = S.K, KS = S.KS;
    const int ntiles = (int)((K + TILE - 1) / TILE);
    const uint32_t row_bytes = TILE * sizeof(TS);
    if (tid == 0) {
        for (int q = 0; q < NSTAGE; ++q) mbar_init(&full[q], 1);
        fence_mbar_init();
        s_abort = 0;
    }
    __syncthreads();
    auto issue_load = [&](int t, int q) {
        TS* dst = stages + (size_t)q * 19 * TILE;
        mbar_expect_tx(&full[q], 19 * row_bytes);
        for (int i = 0; i < 19; ++i) bulk_g2s(dst + i * TILE, f + (int64_t)i * KS + (int64_t)t * TILE, row_bytes, &full[q]);
    };
    double esum = 0;
    if (tid == 0)
        for (int q = 0; q < NSTAGE - 1; ++q) {
            const int t = blockIdx.x + q * gridDim.x;
            if (t < ntiles) issue_load(t, q);
        }
    int j = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++j) {
        const int q = j % NSTAGE;
        TS* buf = stages + (size_t)q * 19 * TILE;
        // keep NSTAGE-1 tiles in flight: refill the stage of the previous tile once its bulk store
        // has read it
        const int tn = t + (NSTAGE - 1) * gridDim.x;
        if (tid == 0 && tn < ntiles) {
            bulk_wait_read_all();
            issue_load(tn, (j + NSTAGE - 1) % NSTAGE);
        }
        const int64_t k = (int64_t)t * TILE + tid;
        int code = 0;
        if (k < K) code = S.code[k];
        // a stored bounce-back node leaves its tile slots and links as they are (identity)
        const bool live = k < K && P.dyn[code] != DYN_BB;
        uint32_t wm = 0;
        int lb = 0;
        TC xv[19];
        if (live) {
            const uint32_t m0 = S.meta[2 * k];
            wm = m0 & 0x7FFFFu;
            lb = S.tlb[t] + (int)(m0 >> 19);
            int r = 0;
#pragma unroll
            for (int i = 1; i < 19; ++i) {
                const bool wl = (wm >> i) & 1u;
                xv[q19opp(i)] = wl ? ld<TS, TC>(link + lb + r) : (TC)0;
                r += wl;
            }
        }
        if (!mbar_wait(&full[q], (uint32_t)((j / NSTAGE) & 1))) {
            if (tid == 0) { tr->gave_up = 1; s_abort = 1; }
        }
        __syncthreads();
        if (s_abort) break;
        if (live) {
            TC g[19];
#pragma unroll
            for (int i = 0; i < 19; ++i) {
                const bool wsrc = i != 0 && ((wm >> q19opp(i)) & 1u);
                g[i] = wsrc ? xv[i] : ld<TS, TC>(buf + i * TILE + tid);
            }
            if (P.dyn[code] == DYN_BGK) {
                if (k < k_west_end) regularize19<TC>(g, -1, (TC)(P.rho_w - 1.0));
                else if (k >= k_east_begin) regularize19<TC>(g, 1, (TC)(P.rho_e - 1.0));
                esum += (double)bgk19<TC>(g, (TC)P.omega[code]);
            }
            int r = 0;
#pragma unroll
            for (int i = 0; i < 19; ++i) {
                const bool wl = (wm >> i) & 1u;
                if (wl) st<TS, TC>(link + lb + r, g[i]);
                else st<TS, TC>(buf + q19opp(i) * TILE + tid, g[i]);
                r += wl;
            }
        }
        fence_async_smem();  // this thread's writes to the tile, ordered before the bulk stores read it
        __syncthreads();
        if (tid == 0) {
            for (int i = 0; i < 19; ++i) bulk_s2g(f + (int64_t)i * KS + (int64_t)t * TILE, buf + i * TILE, row_bytes);
            bulk_commit();
        }
    }
    if (tid == 0) bulk_wait_all();
    __shared__ double sh[32];
    double bt = block_sum(esum, sh);
    finish_step(tr, partials, bt, P.n_bgk, trace);
}

// ------------------------------------------------------------------ one node per thread

constexpr int STREAM_FLOW_THREADS = 128;

// Resident blocks the registers are budgeted for: 64 registers with 4-byte storage (8 blocks run); 5
// blocks with 8- and 2-byte storage (FP64 83 us per step on 199x143x131, 87 at 6 and 105 at 8 blocks,
// which spill; FP16 36.7 us, 37.8 and 40.1).
template <typename TS>
constexpr int stream_flow_blocks() { return sizeof(TS) == 4 ? 6 : 5; }

// The stored average energy of a streamed step from its warps' sums, and the tracer (a launch after the
// step's: inside it, a barrier, a fence and a counter per 128-node block cost the FP32 256^3 pack 125 us of a
// 226 us step).
__global__ void __launch_bounds__(256) k_flow_energy(const double* warp_sums, int64_t n, Tracer* tr, double* partials,
                                                     int64_t n_bgk, int trace, int count) {
    step_wait();
    if (trace && tr->converged) return;
    __shared__ double sh[32];
    double v = 0;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) v += warp_sums[q];
    const double bt = block_sum(v, sh);
    finish_step(tr, partials, bt, n_bgk, trace, count);
}

// One AA step, one node per thread, no staging: both steps are in-place permutations of 19 slots of one
// buffer (the lattice's rows, then its link slots), so a node is 19 offsets, 19 gathers in flight
// together, the collision and 19 stores. Blocks of 128 nodes in launch order keep the blocks in flight
// next to one another in every row. ENERGY: the step's stored average energy is wanted (by the tracer
// after every step, else after the last one of a call): the warps' sums of |u|^2 go to warp_sums.
//
// Bound by HBM and the two round trips of a node (metadata, then the gathers). Against the tiled even and
// the pipelined odd step, us per step: 256x128x128 pack (1.5 M nodes) FP32 60.5 -> 52.4; 384x256x256
// (8.7 M) FP32 316 -> 292 (4.2 -> 4.6 TB/s of algorithmic traffic); 199x143x131 (1.4 M) FP64 103 -> 83 (5.3
// TB/s), FP16 71 -> 37. Two to sixteen nodes per thread with the next one's metadata prefetched: 54 to 65
// us instead of 52.4.
// The node's |u|^2 where it is a BGK node, else 0; nothing is stored where *converged is set.
template <typename TS, typename TC, bool ODD>
__device__ __forceinline__ double flow_stream_node(TS* __restrict__ f, const SparseView& S, const FlowParams& P, int64_t k,
                                                   int64_t k_west_end, int64_t k_east_begin, const int* converged) {
    const uint32_t K32 = (uint32_t)S.KS;
    const FlowMeta M = flow_meta<ODD>(S, k);
    uint32_t off[19];
    if (ODD) {
        const OddRows R = odd_rows(S, k, M);
#pragma unroll
        for (int i = 0; i < 19; ++i) off[i] = odd_src(i, k, R, K32);
    } else {
        const uint32_t wm = M.m0 & 0x7FFFFu;
        const uint32_t lb = 19u * K32 + (uint32_t)(S.tlb[(int)(k >> 8)] + (int)(M.m0 >> 19));  // the links follow the rows
#pragma unroll
        for (int i = 0; i < 19; ++i) {
            const int oi = q19opp(i);
            off[i] = (i != 0 && ((wm >> oi) & 1u)) ? lb + (uint32_t)__popc(wm & ((1u << oi) - 1u))
                                                   : (uint32_t)(i * K32) + (uint32_t)k;
        }
    }
    const int dyn = P.dyn[M.code];
    step_wait();
    // a batch continues past convergence as no-ops: used before the stores only, so the load is not a
    // round trip of its own
    const int settled = converged ? *(volatile const int*)converged : 0;
    if (dyn == DYN_BB) return 0.0;  // a stored bounce-back node: the identity on AA slots
    double e = 0;
    TC g[19];
#pragma unroll
    for (int i = 0; i < 19; ++i) g[i] = gather<TS, TC>(f + off[i]);
    if (dyn == DYN_BGK) {
        if (k < k_west_end) regularize19<TC>(g, -1, (TC)(P.rho_w - 1.0));
        else if (k >= k_east_begin) regularize19<TC>(g, 1, (TC)(P.rho_e - 1.0));
        e = (double)bgk19<TC>(g, (TC)P.omega[M.code]);
    }
    if (!settled) {
#pragma unroll
        for (int i = 0; i < 19; ++i) st<TS, TC>(f + off[q19opp(i)], g[i]);
    }
    return e;
}

template <typename TS, typename TC, bool ODD, bool ENERGY>
__global__ void __launch_bounds__(STREAM_FLOW_THREADS, (stream_flow_blocks<TS>()))
    k_flow_stream(TS* __restrict__ f, const SparseView S, const FlowParams P, const Tracer* tr,
                  double* __restrict__ warp_sums, int trace, int64_t k_west_end, int64_t k_east_begin) {
    const int* converged = ENERGY && trace ? &tr->converged : nullptr;
    const int64_t k = (int64_t)blockIdx.x * STREAM_FLOW_THREADS + threadIdx.x;
    if (k >= S.K) step_wait();
    double e = k < S.K ? flow_stream_node<TS, TC, ODD>(f, S, P, k, k_west_end, k_east_begin, converged) : 0.0;
    if (ENERGY) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
        if ((threadIdx.x & 31) == 0) warp_sums[((int64_t)blockIdx.x * STREAM_FLOW_THREADS + threadIdx.x) >> 5] = e;
    }
}

// ------------------------------------------------------------------ many steps of a small lattice

// `steps` AA steps in one cooperative launch, for lattices small enough that a step is mostly latency:
// launch, ramp-up and metadata are paid once, and between steps the blocks meet at a grid-wide barrier.
// ONE: every node has a resident thread, which keeps its node's slots of both parities in registers
// (both steps are in-place permutations of 19 slots); otherwise the resident threads walk the nodes
// with the per-step code. The barrier also carries the blocks' energy sums, which every block adds up
// in the same order, so each runs the tracer on its own copy of the window and all stop at the same
// step; the tracer's sums of a step run while the next step's populations are on their way, its
// decision before that step's first store.
constexpr int MULTI_THREADS = 256;

template <typename TS, typename TC, bool ONE>
__global__ void __launch_bounds__(MULTI_THREADS, 2)
    k_flow_multi(TS* f, TS* link, const SparseView S, const FlowParams P, Tracer* tr, double* partials, GridSync* gs, int steps,
                 int odd, int64_t k_west_end, int64_t k_east_begin, uint32_t polls) {
    __shared__ double sh[32];
    __shared__ double ring[TRACER_WINDOW];
    __shared__ int s_conv;  // the tracer's decision: set once, before the step after the one it settles
    if (tr->converged) return;  // a batch continues past convergence as no-ops
    const int tid = threadIdx.x;
    if (tid == 0) s_conv = 0;
    const int64_t k = (int64_t)blockIdx.x * MULTI_THREADS + tid, stride = (int64_t)gridDim.x * MULTI_THREADS;
    const uint32_t K32 = (uint32_t)S.KS;
    bool live = ONE && k < S.K;
    uint32_t od[19], wm = 0;
    TS* lk = link;
    int code = 0;
    if (live) {
        const FlowMeta M = flow_meta<true>(S, k);
        code = M.code;
        live = P.dyn[code] != DYN_BB;  // a stored bounce-back node: the identity on AA slots
        const OddRows R = odd_rows(S, k, M);
#pragma unroll
        for (int i = 0; i < 19; ++i) od[i] = odd_src(i, k, R, K32);
        wm = M.m0 & 0x7FFFFu;
        lk = link + S.tlb[(int)(k >> 8)] + (int)(M.m0 >> 19);
    }
    const bool bgk = live && P.dyn[code] == DYN_BGK;
    const int side = k < k_west_end ? -1 : (k >= k_east_begin ? 1 : 0);
    const TC rho = (TC)((side < 0 ? P.rho_w : P.rho_e) - 1.0), omega = (TC)P.omega[code];
    for (int q = tid; q < TRACER_WINDOW; q += MULTI_THREADS) ring[q] = tr->ring[q];
    int head = tr->head, count = tr->count;
    double energy = 0;
    // the stored average energy of step `n` (1, 2, ...) from the blocks' sums, the tracer's window and its
    // criterion. By warp 0 alone, while the other warps collide.
    auto warp_total = [](double v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    auto trace = [&](int n) {
        const double* part = partials + (n & 1) * gridDim.x;
        double v = 0;
        for (int q = tid; q < (int)gridDim.x; q += 32) v += __ldcg(part + q);
        v = warp_total(v);
        energy = P.n_bgk > 0 ? 0.5 * v / (double)P.n_bgk : 0.0;
        if (tid == 0) ring[head] = energy;
        __syncwarp();
        head = (head + 1) % TRACER_WINDOW;
        if (count < TRACER_WINDOW) ++count;
        if (count < TRACER_WINDOW) return;
        v = 0;
        for (int q = tid; q < TRACER_WINDOW; q += 32) v += ring[q];
        const double mean = warp_total(v) / (double)TRACER_WINDOW;
        v = 0;
        for (int q = tid; q < TRACER_WINDOW; q += 32) {
            const double d = ring[q] - mean;
            v += d * d;
        }
        const double r = sqrt(warp_total(v) / (double)(TRACER_WINDOW - 1)) / mean;
        if (tid == 0 && (isnan(r) || fabs(r) < tr->eps)) s_conv = 1;
    };
    int done = 0;
    bool ok = true;
    while (done < steps) {
        const bool odd_step = ((odd + done) & 1) != 0;
        TC g[19];
        if (live) {
            if (odd_step) {
#pragma unroll
                for (int i = 0; i < 19; ++i) g[i] = ld<TS, TC>(f + od[i]);
            } else {
#pragma unroll
                for (int i = 0; i < 19; ++i) {
                    const int oi = q19opp(i);
                    const bool wall = i != 0 && ((wm >> oi) & 1u);
                    g[i] = ld<TS, TC>(wall ? lk + __popc(wm & ((1u << oi) - 1u)) : f + (uint32_t)(i * K32) + k);
                }
            }
        }
        if (done > 0 && tid < 32) trace(done);
        double e = 0;
        if (bgk) {
            if (side < 0) regularize19<TC>(g, -1, rho);
            else if (side > 0) regularize19<TC>(g, 1, rho);
            e = (double)bgk19<TC>(g, omega);
        }
        __syncthreads();
        if (s_conv) break;
        if (live) {
            if (odd_step) {
#pragma unroll
                for (int i = 0; i < 19; ++i) st<TS, TC>(f + od[q19opp(i)], g[i]);
            } else {
#pragma unroll
                for (int i = 0; i < 19; ++i) {
                    const bool wall = i != 0 && ((wm >> i) & 1u);
                    st<TS, TC>(wall ? lk + __popc(wm & ((1u << i) - 1u)) : f + (uint32_t)(q19opp(i) * K32) + k, g[i]);
                }
            }
        }
        if (!ONE) {
            if (odd_step) {
                for (int64_t j = k; j < S.K; j += stride)
                    e += flow_node<TS, TC, true>(f, link, S, P, j, k_west_end, k_east_begin);
            } else {
                for (int64_t j = k; j < S.K; j += stride)
                    e += flow_node<TS, TC, false>(f, link, S, P, j, k_west_end, k_east_begin);
            }
        }
        ++done;
        const double bt = block_sum(e, sh);
        if (tid == 0) partials[(done & 1) * gridDim.x + blockIdx.x] = bt;
        if (!(ok = grid_barrier(gs, (unsigned)done, polls))) break;
    }
    if (!ok) {
        if (tid == 0) tr->gave_up = 1;
        return;
    }
    if (blockIdx.x != 0) return;
    __syncthreads();
    if (tid < 32 && !s_conv) trace(done);
    __syncthreads();
    for (int q = tid; q < TRACER_WINDOW; q += MULTI_THREADS) tr->ring[q] = ring[q];
    if (tid == 0) {
        tr->energy = energy;
        tr->iterations += done;
        tr->head = head;
        tr->count = count;
        if (s_conv) tr->converged = 1;
    }
}

// ------------------------------------------------------------------ batched step of many domains

// One AA step of every domain's flow lattice: one block per tile of the table, which takes its domain's
// flow part to shared memory and steps the tile 128 nodes at a time with the single-domain streamed step's
// code. 96 uneven domains (2.9 M nodes, FP32): 131 us per step; the tiled and pipelined steps over runs of
// the table took 145.
template <typename TS, typename TC, bool ODD>
__global__ void __launch_bounds__(STREAM_FLOW_THREADS, (stream_flow_blocks<TS>())) k_flow_stream_batch(const BatchView B) {
    constexpr int WORDS = (int)(offsetof(BatchDomain, g) / 8);
    __shared__ __align__(16) uint64_t words[WORDS];
    const BatchTile T = B.ftiles[blockIdx.x];
    const uint64_t* src = reinterpret_cast<const uint64_t*>(B.dom + T.d);
    for (int q = threadIdx.x; q < WORDS; q += STREAM_FLOW_THREADS) words[q] = src[q];
    __syncthreads();
    const BatchDomain& D = *reinterpret_cast<const BatchDomain*>(words);  // its members before g only
    for (int i = threadIdx.x; i < T.count; i += STREAM_FLOW_THREADS)
        flow_stream_node<TS, TC, ODD>((TS*)D.f, D.fs, D.fp, T.first + i, D.fkw, D.fke, nullptr);
}

void launch_flow_batch(const BatchView& B, int prec, bool odd, cudaStream_t st) {
    if (B.nft == 0) return;
#define CLB_FB(TS, TC)                                                                          \
    if (odd) k_flow_stream_batch<TS, TC, true><<<B.nft, STREAM_FLOW_THREADS, 0, st>>>(B);       \
    else k_flow_stream_batch<TS, TC, false><<<B.nft, STREAM_FLOW_THREADS, 0, st>>>(B);
    switch (prec) {
        case CLB_F64: CLB_FB(double, double); break;
        case CLB_F32: CLB_FB(float, float); break;
        default: CLB_FB(__half, float); break;
    }
#undef CLB_FB
}

// PressureGradient equilibrium (complab_functions.hh:82-94): BGK nodes t_i (rho(x) - 1),
// no-dynamics nodes zero (BounceBack / NoDynamics equilibria are zero). For a wall link (a, i)
// the even-step slot X holds a's equilibrium incoming opp(i) and the odd-step slot
// Y = f[opp(i)][a] the wall's initial (zero) population.
template <typename TS>
__global__ void k_flow_init(TS* __restrict__ f, TS* __restrict__ link, const SparseView S, const FlowParams P,
                            double delta_p) {
    const Geom G = P.g;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < S.K; k += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(S.node[k] / G.plane);
        const double rho = 1.0 - delta_p * 3.0 / (double)(G.nx - 1) * (double)x;
        const bool bgk = P.dyn[S.code[k]] == DYN_BGK;
        const uint32_t wm = S.wall[k];
#pragma unroll
        for (int i = 0; i < 19; ++i) {
            const double eq = bgk ? q19w(i) * (rho - 1.0) : 0.0;
            const bool wall_src = i != 0 && ((wm >> q19opp(i)) & 1u);
            const double v = wall_src ? 0.0 : eq;
            if constexpr (std::is_same<TS, __half>::value) f[(int64_t)i * S.KS + k] = to_half(v);
            else f[(int64_t)i * S.KS + k] = (TS)v;
            if (wall_src) {
                TS* x_ = link_slot(S, link, (int)k, q19opp(i));
                if constexpr (std::is_same<TS, __half>::value) *x_ = to_half(eq);
                else *x_ = (TS)eq;
            }
        }
    }
}

// computeVelocity of the voxel n at x: BGK u = j; pressure-plane BGK nodes (j_x from the known
// populations, 0, 0); others 0.
template <typename TS, typename TC>
__device__ __forceinline__ void node_velocity(const TS* __restrict__ f, const TS* __restrict__ link, const SparseView& S,
                                              const int8_t* __restrict__ mat, const FlowParams& P, int odd, int64_t n, int x,
                                              TC& jx, TC& jy, TC& jz) {
    jx = jy = jz = 0;
    if (P.dyn[mat[n]] != DYN_BGK) return;
    const int k = S.idx_of[n];
    if (k < 0) return;
    TC g[19];
    flow_incoming<TS, TC>(S, f, link, k, odd, g);
    if (x == 0 || x == P.g.nx - 1) {
        const int o = (x == 0) ? -1 : 1;
        const TC rb = (TC)((x == 0 ? P.rho_w : P.rho_e) - 1.0);
        TC r0 = 0, rn = 0;
#pragma unroll
        for (int i = 0; i < 19; ++i) {
            if (q19cx(i) == 0) r0 += g[i];
            else if (q19cx(i) == o) rn += g[i];
        }
        jx = (TC)o * (r0 + (TC)2 * rn - rb);
    } else {
#pragma unroll
        for (int i = 0; i < 19; ++i) {
            jx += (TC)q19cx(i) * g[i];
            jy += (TC)q19cy(i) * g[i];
            jz += (TC)q19cz(i) * g[i];
        }
    }
}

// The velocity at the voxels `nodes[0..count)`; output u[3][stride] at position t.
template <typename TS, typename TC, typename TO>
__global__ void __launch_bounds__(256) k_flow_velocity_at(const TS* __restrict__ f, const TS* __restrict__ link, const SparseView S,
                                   const int8_t* __restrict__ mat, const FlowParams P, int odd,
                                   const int32_t* __restrict__ nodes, int64_t count, TO* __restrict__ u, int64_t stride) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
        const int n = nodes[t];
        TC jx, jy, jz;
        node_velocity<TS, TC>(f, link, S, mat, P, odd, n, n / P.g.plane, jx, jy, jz);
        u[t] = (TO)jx;
        u[stride + t] = (TO)jy;
        u[2 * stride + t] = (TO)jz;
    }
}

// The velocity of every voxel of rows [r0, r1) of the box; output u[3][stride], the rows' first voxel
// at position 0. Bound by HBM (the field written, the lattice read once): found through the inverse
// index with 64-bit divisions it took 522 us on the 256x128x128 pack (FP32), here 95 us.
template <typename TS, typename TC, typename TO>
__global__ void __launch_bounds__(256) k_flow_velocity(const TS* __restrict__ f, const TS* __restrict__ link, const SparseView S,
                                const int8_t* __restrict__ mat, const FlowParams P, int odd, int r0, int r1,
                                TO* __restrict__ u, int64_t stride) {
    const int64_t n0 = (int64_t)r0 * P.g.nz;
    for_each_voxel(P.g, r0, r1, [&](int64_t n, int x, int, int) {
        TC jx, jy, jz;
        node_velocity<TS, TC>(f, link, S, mat, P, odd, n, x, jx, jy, jz);
        TO* o = u + (n - n0);
        o[0] = (TO)jx;
        o[stride] = (TO)jy;
        o[2 * stride] = (TO)jz;
    });
}

template <typename TS>
__global__ void k_flow_get_pops(const TS* __restrict__ f, const TS* __restrict__ link, const SparseView S,
                                const Geom G, int odd, double* __restrict__ out) {
    const double zero[19] = {};
    for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < G.N; n += (int64_t)gridDim.x * blockDim.x) {
        double g[19];
        natural<TS, double, 19>(S, G, f, link, n, odd, zero, g);
        for (int i = 0; i < 19; ++i) out[(int64_t)i * G.N + n] = g[i];
    }
}

template <typename TS>
__global__ void k_flow_set_pops(TS* __restrict__ f, TS* __restrict__ link, const SparseView S, const Geom G, int odd,
                                const double* __restrict__ in) {
    for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < G.N; n += (int64_t)gridDim.x * blockDim.x) {
        double g[19];
        for (int i = 0; i < 19; ++i) g[i] = in[(int64_t)i * G.N + n];
        put_natural<TS, 19>(S, G, f, link, n, odd, g);
    }
}

__global__ void k_flow_vstats(const double* __restrict__ u, const Geom G, double* __restrict__ acc) {
    // acc[0] sum |u| over x=1..nx-2, acc[1] max u_x (as ordered bits), acc[2] sum u_x on x=nx-2
    __shared__ double sh[32];
    double s_norm = 0, s_out = 0, m = -1e300;
    for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < G.N; n += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(n / G.plane);
        if (x < 1 || x > G.nx - 2) continue;
        const double ux = u[n], uy = u[G.N + n], uz = u[2 * G.N + n];
        s_norm += sqrt(ux * ux + uy * uy + uz * uz);
        m = fmax(m, ux);
        if (x == G.nx - 2) s_out += ux;
    }
    double a = block_sum(s_norm, sh);
    double b = block_sum(s_out, sh);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    __shared__ double smax[32];
    if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double mm = -1e300;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) mm = fmax(mm, smax[k]);
        atomicAdd(&acc[0], a);
        atomicAdd(&acc[2], b);
        // max of doubles via the ordered-integer trick
        long long bits = __double_as_longlong(mm);
        long long key = bits >= 0 ? bits : (bits ^ 0x7fffffffffffffffLL);
        atomicMax((long long*)&acc[1], key);
    }
}

// ------------------------------------------------------------------ host side

static int64_t flow_tiles(const clb_handle* h) { return (h->flow_sp.K + STREAM_FLOW_THREADS - 1) / STREAM_FLOW_THREADS; }

static size_t storage_size(int prec) { return prec == CLB_F64 ? 8 : (prec == CLB_F32 ? 4 : 2); }

template <typename TS>
static size_t even_smem() {
    return (size_t)NSTAGE * 19 * TILE * sizeof(TS);
}

// two slots of 19 populations per thread for the pipelined odd step
template <typename TS>
static size_t pipe_smem() {
    return (size_t)2 * 19 * PIPE_THREADS * sizeof(TS);
}

// resident-CTA grid of the pipelined odd step (0: not available for 2-byte storage, whose
// populations are below the 4-byte granule of the asynchronous copy)
template <typename TS, typename TC>
static int pipe_grid_of(clb_handle* h) {
    if (sizeof(TS) < 4) return 0;
    int per_sm = 0;
    const size_t sm = pipe_smem<TS>();
    cudaFuncSetAttribute(k_flow_odd_pipe<TS, TC, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_flow_odd_pipe<TS, TC, 2>, PIPE_THREADS, sm);
    return h->num_sms * std::min(16, std::max(1, per_sm));
}


template <typename F>
static int grid_for(clb_handle* h, F kernel, int threads) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0);
    if (per_sm < 1) per_sm = 1;
    return h->num_sms * per_sm;
}

void flow_free(clb_handle* h) {
    cudaFree(h->d_f); h->d_f = nullptr;
    h->d_flink = nullptr;  // inside d_f
    sparse_free(h->flow_sp);
    cudaFree(h->d_tracer); h->d_tracer = nullptr;
    cudaFree(h->d_partials); h->d_partials = nullptr;
    h->flow_ready = false;
}

static int flow_gather_grid(clb_handle* h) {
    switch (h->flow_prec) {
        case CLB_F64: return h->flow_minb == 2 ? grid_for(h, k_flow_aa<double, double, true, 2>, FLOW_THREADS) : grid_for(h, k_flow_aa<double, double, true, 3>, FLOW_THREADS);
        case CLB_F32: return h->flow_minb == 2 ? grid_for(h, k_flow_aa<float, float, true, 2>, FLOW_THREADS) : grid_for(h, k_flow_aa<float, float, true, 3>, FLOW_THREADS);
        default: return h->flow_minb == 2 ? grid_for(h, k_flow_aa<__half, float, true, 2>, FLOW_THREADS) : grid_for(h, k_flow_aa<__half, float, true, 3>, FLOW_THREADS);
    }
}

// Blocks of k_flow_multi for this lattice, 0 where a launch per step is faster; h->flow_multi_one: every
// node has a resident thread. us per traced step, one launch per step -> many steps per launch, by nodes:
//   11 k: FP64 13.5 -> 9.2, FP32 10.4 -> 4.8, FP16 12.6 -> 5.7;  91 k (walked): 17.0 -> 12.6, 13.4 -> 10.8, 17.9 -> 11.7;
//   214 k: 23.2 -> 17.7, 17.0 -> 14.2, 22.3 -> 16.1;             482 k: 35.9 -> 37.5, 22.5 -> 24.6, 27.9 -> 27.7.
// Steps without the tracer need no grid-wide sum and go one to a chained launch at every size (many steps per
// launch: 27 k nodes FP32 3.2 against 2.95, 91 k 7.3 against 4.9, 214 k FP64 14.7 against 12.0).
constexpr int64_t MULTI_MAX_NODES = 400000;

template <typename TS, typename TC>
static int flow_multi_blocks(clb_handle* h) {
    int one = 0, loop = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&one, k_flow_multi<TS, TC, true>, MULTI_THREADS, 0) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&loop, k_flow_multi<TS, TC, false>, MULTI_THREADS, 0) != cudaSuccess)
        return 0;
    const int64_t need = (h->flow_sp.K + MULTI_THREADS - 1) / MULTI_THREADS;
    h->flow_multi_one = need <= (int64_t)one * h->num_sms;
    if (need < 1 || h->flow_sp.K > MULTI_MAX_NODES) return 0;
    return (int)(h->flow_multi_one ? need : (int64_t)loop * h->num_sms);
}

clb_status flow_init(clb_handle* h, double delta_p) {
    h->resolve_tracer_valid = false;  // a new flow: the in-loop tracer starts empty again
    const clb_domain_desc& d = h->d;
    FlowParams& P = h->fp;
    std::memset(&P, 0, sizeof(P));
    P.g = h->g;
    const double omega = 1.0 / d.tau;
    // NSdomainSetup: IncBGK(omega) everywhere, pore codes IncBGK, bounce-back, no-dynamics,
    // biofilm IncBGK(omega_bio) or BounceBack when impermeable.
    for (int c = 0; c < MAX_CODES; ++c) { P.dyn[c] = DYN_BGK; P.omega[c] = omega; }
    if (d.bounce_back_code >= 0 && d.bounce_back_code < MAX_CODES) P.dyn[d.bounce_back_code] = DYN_BB;
    if (d.solid_code >= 0 && d.solid_code < MAX_CODES) P.dyn[d.solid_code] = DYN_NONE;
    for (int m = 0; m < d.n_microbes; ++m) {
        int c = d.bio_codes[m];
        if (c < 0 || c >= MAX_CODES) continue;
        if (d.perm_ratio[m] > 1e-14) {
            P.dyn[c] = DYN_BGK;
            P.omega[c] = 1.0 / (d.perm_ratio[m] * (1.0 / omega - 0.5) + 0.5);
        } else {
            P.dyn[c] = DYN_BB;
        }
    }
    P.rho_w = 1.0;
    P.rho_e = 1.0 - delta_p * 3.0;
    h->delta_p = delta_p;
    // the flow lattice's own map once precipitation has changed the species' one
    const std::vector<int8_t>& fmat = h->h_mat_flow.empty() ? h->h_mat : h->h_mat_flow;
    // biofilm voxels are nodes even when impermeable (bounce-back nodes are skipped by the step),
    // so that the automaton can turn them back into pore without a new layout
    int8_t cls[MAX_CODES];
    for (int c = 0; c < MAX_CODES; ++c) cls[c] = (P.dyn[c] != DYN_BB);
    for (int m = 0; m < d.n_microbes; ++m)
        if (d.bio_codes[m] >= 0 && d.bio_codes[m] < MAX_CODES) cls[d.bio_codes[m]] = 1;
    // BGK node count from a histogram of the codes (four interleaved counters, no data-dependent
    // branch), the node counts of the first and last x-planes from those planes alone
    int64_t nbgk = 0, kw = 0, ke = 0;
    {
        std::vector<int64_t> hist(4 * 128, 0);
        const uint8_t* m = reinterpret_cast<const uint8_t*>(fmat.data());
        const int64_t N = h->g.N, plane = h->g.plane;
        int64_t n = 0;
        for (; n + 4 <= N; n += 4) {
            ++hist[m[n] & 127];
            ++hist[128 + (m[n + 1] & 127)];
            ++hist[256 + (m[n + 2] & 127)];
            ++hist[384 + (m[n + 3] & 127)];
        }
        for (; n < N; ++n) ++hist[m[n] & 127];
        for (int c = 0; c < 128; ++c)
            if (P.dyn[c] == DYN_BGK) nbgk += hist[c] + hist[128 + c] + hist[256 + c] + hist[384 + c];
        for (int64_t i = 0; i < plane; ++i) {
            kw += cls[m[i] & 127];
            ke += cls[m[N - plane + i] & 127];
        }
    }
    P.n_bgk = nbgk;

    flow_free(h);
    clb_status s = sparse_build(h, cls, 19, h->flow_sp, &fmat);
    if (s != CLB_OK) return s;
    const int64_t K = h->flow_sp.K;
    h->k_west_end = kw;
    h->k_east_begin = K - ke;
    h->flow_prec = d.flow_precision;
    const size_t es = storage_size(h->flow_prec);
    cudaError_t e;
    // one buffer: the 19 population rows, then the link slots
    const size_t rows = es * 19 * (size_t)h->flow_sp.KS;
    if ((e = cudaMalloc(&h->d_f, rows + es * (size_t)std::max<int64_t>(1, h->flow_sp.L) + 16)) != cudaSuccess)
        return cuda_check(h, e, "flow populations");
    h->d_flink = (char*)h->d_f + rows;
    if ((e = cudaMalloc(&h->d_tracer, sizeof(Tracer))) != cudaSuccess) return cuda_check(h, e, "tracer");
    cudaMemsetAsync(h->d_tracer, 0, sizeof(Tracer), h->stream);
    cudaMemsetAsync(h->d_flink, 0, es * (size_t)std::max<int64_t>(1, h->flow_sp.L), h->stream);

    int grid = flow_gather_grid(h);
    h->flow_grid = grid;
    // the even step's tiled kernel: persistent CTAs, shared-memory stages sized by precision
    {
        int per_sm = 0;
        size_t sm = 0;
        switch (h->flow_prec) {
            case CLB_F64:
                sm = even_smem<double>();
                cudaFuncSetAttribute(k_flow_even_tma<double, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_flow_even_tma<double, double>, TILE, sm);
                break;
            case CLB_F32:
                sm = even_smem<float>();
                cudaFuncSetAttribute(k_flow_even_tma<float, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_flow_even_tma<float, float>, TILE, sm);
                break;
            default:
                sm = even_smem<__half>();
                cudaFuncSetAttribute(k_flow_even_tma<__half, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_flow_even_tma<__half, float>, TILE, sm);
                break;
        }
        h->flow_even_grid = h->num_sms * std::max(1, per_sm);
    }
    switch (h->flow_prec) {
        case CLB_F64: h->flow_pipe_grid = pipe_grid_of<double, double>(h); break;
        case CLB_F32: h->flow_pipe_grid = pipe_grid_of<float, float>(h); break;
        default: h->flow_pipe_grid = 0; break;
    }
    if (!h->flow_pipe_grid) h->flow_odd_pipe = 0;
    // the blocks' partials, sized for the largest grid any variant uses, then the streamed step's warp sums
    const int pcap = h->num_sms * 16;
    const int64_t warps = std::max<int64_t>(1, flow_tiles(h)) * (STREAM_FLOW_THREADS / 32);
    if ((e = cudaMalloc(&h->d_partials, sizeof(double) * (pcap + warps))) != cudaSuccess) return cuda_check(h, e, "partials");
    h->partial_cap = pcap;
    if (!h->d_flow_sync && (e = cudaMalloc(&h->d_flow_sync, sizeof(GridSync))) != cudaSuccess)
        return cuda_check(h, e, "barrier");
    h->flow_gave_up = false;
    switch (h->flow_prec) {
        case CLB_F64: h->flow_multi = flow_multi_blocks<double, double>(h); break;
        case CLB_F32: h->flow_multi = flow_multi_blocks<float, float>(h); break;
        default: h->flow_multi = flow_multi_blocks<__half, float>(h); break;
    }

    const int ig = h->num_sms * 8;
    const SparseView S = view_of(h->flow_sp);
    switch (h->flow_prec) {
        case CLB_F64: k_flow_init<double><<<ig, 256, 0, h->stream>>>((double*)h->d_f, (double*)h->d_flink, S, P, delta_p); break;
        case CLB_F32: k_flow_init<float><<<ig, 256, 0, h->stream>>>((float*)h->d_f, (float*)h->d_flink, S, P, delta_p); break;
        default: k_flow_init<__half><<<ig, 256, 0, h->stream>>>((__half*)h->d_f, (__half*)h->d_flink, S, P, delta_p); break;
    }
    h->flow_iters = 0;
    h->flow_ready = true;
    return cuda_check(h, cudaGetLastError(), "flow init");
}

// The streamed step, except where a tuning key selects the tiled and pipelined kernels or clb_autotune
// measured them faster for steps without the tracer. A traced step is two
// chained launches, the step and its energy (tiled and pipelined kernels -> streamed, us per traced step: 480 k
// nodes FP32 23.1 -> 22.4, 1.3 M 55.5 -> 54.5, 3.8 M 153.6 -> 147.4; FP64 3.8 M 261 -> 237, FP16 174 -> 124).
static bool flow_streams(const clb_handle* h, bool trace) { return !h->flow_keyed && (trace || !h->flow_tuned); }

// One step. The streamed step forms the stored energy, and counts `count` iterations, only where count is
// not 0; the kernels a tuning key selects do both at every step.
static void launch_flow(clb_handle* h, bool odd, int trace, int count, bool after) {
    ++h->launches;  // one step launch per call
    const FlowParams& P = h->fp;
    const SparseView S = view_of(h->flow_sp);
    const int grid = h->flow_grid;
    if (flow_streams(h, trace != 0)) {
        const unsigned g = (unsigned)std::max<int64_t>(1, flow_tiles(h));
        auto go = [&](auto kern, auto* ts) {
            using TS = std::remove_pointer_t<decltype(ts)>;
            launch_step(after, kern, g, STREAM_FLOW_THREADS, 0, h->stream, (TS*)h->d_f, S, P, h->d_tracer,
                        h->d_partials + h->partial_cap, trace, h->k_west_end, h->k_east_begin);
        };
#define CLB_STREAM(TS, TC)                                                                                \
    if (odd) count ? go(k_flow_stream<TS, TC, true, true>, (TS*)nullptr) : go(k_flow_stream<TS, TC, true, false>, (TS*)nullptr); \
    else count ? go(k_flow_stream<TS, TC, false, true>, (TS*)nullptr) : go(k_flow_stream<TS, TC, false, false>, (TS*)nullptr);
        switch (h->flow_prec) {
            case CLB_F64: CLB_STREAM(double, double); break;
            case CLB_F32: CLB_STREAM(float, float); break;
            default: CLB_STREAM(__half, float); break;
        }
#undef CLB_STREAM
        if (count) {
            ++h->launches;
            launch_step(true, k_flow_energy, h->num_sms, 256, 0, h->stream, h->d_partials + h->partial_cap,
                        (int64_t)g * (STREAM_FLOW_THREADS / 32), h->d_tracer, h->d_partials, P.n_bgk, trace, count);
        }
        return;
    }
    if (!odd && h->flow_even_tma) {
        const int eg = h->flow_even_grid;
#define CLB_EVEN(TS, TC)                                                                                       \
        k_flow_even_tma<TS, TC><<<eg, TILE, even_smem<TS>(), h->stream>>>((TS*)h->d_f, (TS*)h->d_flink, S, P,  \
                                                                       h->d_tracer, h->d_partials, trace,     \
                                                                       h->k_west_end, h->k_east_begin);
        switch (h->flow_prec) {
            case CLB_F64: CLB_EVEN(double, double); break;
            case CLB_F32: CLB_EVEN(float, float); break;
            default: CLB_EVEN(__half, float); break;
        }
#undef CLB_EVEN
        return;
    }
    if (odd && h->flow_odd_pipe && h->flow_pipe_grid) {
        const int pg = h->flow_pipe_grid;
#define CLB_PIPE(TS, TC)                                                                                       \
        k_flow_odd_pipe<TS, TC, 2><<<pg, PIPE_THREADS, pipe_smem<TS>(), h->stream>>>(                          \
            (TS*)h->d_f, (TS*)h->d_flink, S, P, h->d_tracer, h->d_partials, trace, h->k_west_end, h->k_east_begin);
        switch (h->flow_prec) {
            case CLB_F64: CLB_PIPE(double, double); return;
            case CLB_F32: CLB_PIPE(float, float); return;
            default: break;
        }
#undef CLB_PIPE
    }
#define CLB_LAUNCH_B(TS, TC, B)                                                                                \
    if (odd)                                                                                                   \
        k_flow_aa<TS, TC, true, B><<<grid, FLOW_THREADS, 0, h->stream>>>((TS*)h->d_f, (TS*)h->d_flink, S, P,    \
                                                                          h->d_tracer, h->d_partials, trace,   \
                                                                          h->k_west_end, h->k_east_begin);     \
    else                                                                                                       \
        k_flow_aa<TS, TC, false, B><<<grid, FLOW_THREADS, 0, h->stream>>>((TS*)h->d_f, (TS*)h->d_flink, S, P,   \
                                                                           h->d_tracer, h->d_partials, trace,  \
                                                                           h->k_west_end, h->k_east_begin);
#define CLB_LAUNCH(TS, TC) if (h->flow_minb == 2) { CLB_LAUNCH_B(TS, TC, 2) } else { CLB_LAUNCH_B(TS, TC, 3) }
    switch (h->flow_prec) {
        case CLB_F64: CLB_LAUNCH(double, double); break;
        case CLB_F32: CLB_LAUNCH(float, float); break;
        default: CLB_LAUNCH(__half, float); break;
    }
#undef CLB_LAUNCH
#undef CLB_LAUNCH_B
}

template <typename TS, typename TC>
static cudaError_t launch_flow_multi(clb_handle* h, int n) {
    GridSync* gs = (GridSync*)h->d_flow_sync;
    uint32_t polls = (uint32_t)h->barrier_polls;
    cudaError_t e = cudaMemsetAsync(gs, 0, sizeof(GridSync), h->stream);
    if (e != cudaSuccess) return e;
    TS *f = (TS*)h->d_f, *link = (TS*)h->d_flink;
    SparseView S = view_of(h->flow_sp);
    int odd = (int)(h->flow_iters & 1);
    void* args[] = {&f, &link, &S, &h->fp, &h->d_tracer, &h->d_partials, &gs, &n, &odd, &h->k_west_end, &h->k_east_begin,
                    &polls};
    ++h->launches;
    const void* kern = h->flow_multi_one
                           ? (const void*)k_flow_multi<TS, TC, true>
                           : (const void*)k_flow_multi<TS, TC, false>;
    return cudaLaunchCooperativeKernel(kern, dim3(h->flow_multi), dim3(MULTI_THREADS), args, 0, h->stream);
}

// A small lattice takes its traced steps in launches of up to MULTI_STEPS (k_flow_multi); a call of one or
// two of them, steps without the tracer, and every other lattice, a launch per step.
constexpr int MULTI_STEPS = 1024, MULTI_MIN_STEPS = 3;

clb_status flow_step(clb_handle* h, int n, bool trace, double eps) {
    (void)eps;
    const clb_status ws = waits_check(h, true, false);
    if (ws != CLB_OK) return ws;
    if (trace && h->flow_multi && !h->flow_keyed && n >= MULTI_MIN_STEPS) {
        for (int k = 0; k < n; k += MULTI_STEPS) {
            const int m = std::min(MULTI_STEPS, n - k);
            cudaError_t e;
            switch (h->flow_prec) {
                case CLB_F64: e = launch_flow_multi<double, double>(h, m); break;
                case CLB_F32: e = launch_flow_multi<float, float>(h, m); break;
                default: e = launch_flow_multi<__half, float>(h, m); break;
            }
            if (e != cudaSuccess) return cuda_check(h, e, "flow steps");
            h->flow_iters += m;
        }
        return CLB_OK;
    }
    for (int k = 0; k < n; ++k) {
        launch_flow(h, (h->flow_iters & 1) != 0, trace ? 1 : 0, trace ? 1 : (k + 1 == n ? n : 0), k > 0 && flow_streams(h, trace));
        h->flow_iters += 1;
    }
    return cuda_check(h, cudaGetLastError(), "flow step");
}

clb_status flow_solve(clb_handle* h, int max_it, double eps, int* iterations, bool keep_window) {
    // a fresh util::ValueTracer (empty window, new epsilon), or the in-loop one as the previous
    // re-solve left it
    Tracer t0;
    std::memset(&t0, 0, sizeof(t0));
    if (keep_window && h->resolve_tracer_valid) {
        std::memcpy(t0.ring, h->resolve_tracer.ring, sizeof(t0.ring));
        t0.count = h->resolve_tracer.count;
        t0.head = h->resolve_tracer.head;
    }
    Tracer cur;
    cudaError_t e = cudaMemcpyAsync(&cur, h->d_tracer, sizeof(Tracer), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return cuda_check(h, e, "tracer read");
    if (cur.gave_up) h->flow_gave_up = true;
    clb_status waited = waits_check(h, true, false);
    if (waited != CLB_OK) return waited;
    t0.eps = eps;
    t0.iterations = cur.iterations;
    t0.energy = cur.energy;
    cudaMemcpyAsync(h->d_tracer, &t0, sizeof(Tracer), cudaMemcpyHostToDevice, h->stream);
    const int64_t start = cur.iterations;
    int done = 0;
    // Steps enqueued before the host looks at the tracer. A many-step launch stops itself, so it gets as
    // many as a launch takes. A streamed step after convergence still reads the lattice (it looks at the
    // decision before its stores, which saves every other step a round trip), so the run up to a full
    // window goes at once and then few at a time: the wait costs about 15 us, a step of a lattice that
    // takes the streamed kernel 16 us and more. The other kernels return at once.
    const bool multi = h->flow_multi && !h->flow_keyed, stream = !multi && flow_streams(h, true);
    int chunk = multi ? MULTI_STEPS : stream ? std::max(4, TRACER_WINDOW - t0.count) : 64;
    bool conv = false;
    while (done < max_it) {
        int k = std::min(chunk, max_it - done);
        clb_status s = flow_step(h, k, true, eps);
        if (s != CLB_OK) return s;
        done += k;
        e = cudaMemcpyAsync(&cur, h->d_tracer, sizeof(Tracer), cudaMemcpyDeviceToHost, h->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
        if (e != cudaSuccess) return cuda_check(h, e, "tracer read");
        if (cur.gave_up) h->flow_gave_up = true;
        if ((waited = waits_check(h, true, false)) != CLB_OK) break;
        if (cur.converged) { conv = true; break; }
        if (stream) chunk = chunk >= 32 ? 32 : chunk * 2;
        else if (chunk < 1024) chunk *= 2;
    }
    h->flow_iters = cur.iterations;  // steps after convergence were no-ops
    if (iterations) *iterations = (int)(cur.iterations - start);
    if (keep_window && waited == CLB_OK) {
        h->resolve_tracer = cur;
        h->resolve_tracer_valid = true;
    }
    // leave the tracer disabled for plain steps
    int zero = 0;
    cudaMemcpyAsync(&h->d_tracer->converged, &zero, sizeof(int), cudaMemcpyHostToDevice, h->stream);
    cudaStreamSynchronize(h->stream);
    if (waited != CLB_OK) return waited;
    // a diverged solve (NaN or Inf stored energy; the tracer reads a NaN window as settled) stops
    // the run cleanly, as complab.cpp:3116-3117 does
    if (!std::isfinite(cur.energy))
        return fail(h, CLB_NONFINITE, "flow solve diverged: the stored average energy is not finite");
    if (!conv) {
        // at the cap with nothing leaving through the outlet plane the flow path is sealed: the
        // reference's percolation limit (complab.cpp:3106-3113, outlet u_x <= 1e-12)
        clb_flow_stats st;
        clb_status s = flow_stats(h, 1.0, &st);
        if (s != CLB_OK) return s;
        if (!(st.darcy_outlet_ux > THRD))
            return fail(h, CLB_PERCOLATION_LOST, "percolation lost: no flow through the outlet plane at the iteration cap");
        return CLB_NOT_CONVERGED;
    }
    return CLB_OK;
}

// Calls fn(storage type, arithmetic type, output type) for the handle's precision and dtype (0 float64,
// 1 float32), each as a null pointer of the type.
template <typename F>
static void velocity_types(clb_handle* h, int dtype, F fn) {
    double* d = nullptr;
    float* s = nullptr;
    __half* q = nullptr;
    switch (h->flow_prec) {
        case CLB_F64: if (dtype == 0) fn(d, d, d); else fn(d, d, s); break;
        case CLB_F32: if (dtype == 0) fn(s, s, d); else fn(s, s, s); break;
        default: if (dtype == 0) fn(q, s, d); else fn(q, s, s); break;
    }
}

// Velocity at the `count` voxels `nodes` into a device buffer u[3][stride] of float64 (dtype 0) or
// float32 (dtype 1).
clb_status flow_velocity_at(clb_handle* h, const int32_t* nodes, int64_t count, void* u, int64_t stride, int dtype) {
    ++h->launches;
    velocity_types(h, dtype, [&](auto* ts, auto* tc, auto* to) {
        using TS = std::remove_pointer_t<decltype(ts)>;
        using TC = std::remove_pointer_t<decltype(tc)>;
        using TO = std::remove_pointer_t<decltype(to)>;
        k_flow_velocity_at<TS, TC, TO><<<h->num_sms * 8, 256, 0, h->stream>>>(
            (const TS*)h->d_f, (const TS*)h->d_flink, view_of(h->flow_sp), flow_mat(h), h->fp, (int)(h->flow_iters & 1),
            nodes, count, (TO*)u, stride);
    });
    return cuda_check(h, cudaGetLastError(), "flow velocity");
}

// The velocity of rows [r0, r1) into a device buffer u[3][stride].
static void launch_velocity_rows(clb_handle* h, int r0, int r1, void* u, int64_t stride, int dtype) {
    ++h->launches;
    velocity_types(h, dtype, [&](auto* ts, auto* tc, auto* to) {
        using TS = std::remove_pointer_t<decltype(ts)>;
        using TC = std::remove_pointer_t<decltype(tc)>;
        using TO = std::remove_pointer_t<decltype(to)>;
        k_flow_velocity<TS, TC, TO><<<h->num_sms * 8, 256, 0, h->stream>>>(
            (const TS*)h->d_f, (const TS*)h->d_flink, view_of(h->flow_sp), flow_mat(h), h->fp, (int)(h->flow_iters & 1), r0,
            r1, (TO*)u, stride);
    });
}

// The velocity field u[3][N] into a device buffer, or to the host through the handle's staging buffer
// a run of rows at a time.
clb_status flow_velocity(clb_handle* h, void* dst, int dtype_device, bool to_host) {
    const int rows = h->g.nx * h->g.ny, nz = h->g.nz;
    if (!to_host) {
        launch_velocity_rows(h, 0, rows, dst, h->g.N, dtype_device);
        return cuda_check(h, cudaGetLastError(), "flow velocity");
    }
    const size_t es = dtype_device == 0 ? 8 : 4;
    int per = 0;
    clb_status s = stage_rows(h, 3 * es, &per);
    if (s != CLB_OK) return s;
    cudaError_t e = cudaSuccess;
    for (int r0 = 0; r0 < rows && e == cudaSuccess; r0 += per) {
        const int r1 = std::min(rows, r0 + per);
        const size_t n = (size_t)(r1 - r0) * nz, at = (size_t)r0 * nz;
        launch_velocity_rows(h, r0, r1, h->d_stage, (int64_t)n, dtype_device);
        if (r1 - r0 == rows) {  // the whole field: the three components are contiguous on both sides
            e = cudaMemcpyAsync(dst, h->d_stage, es * 3 * n, cudaMemcpyDeviceToHost, h->stream);
            break;
        }
        for (int a = 0; a < 3 && e == cudaSuccess; ++a)
            e = cudaMemcpyAsync((char*)dst + es * ((size_t)a * h->g.N + at), (char*)h->d_stage + es * a * n, es * n,
                                cudaMemcpyDeviceToHost, h->stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    return cuda_check(h, e, "velocity copy");
}

clb_status flow_populations(clb_handle* h, double* host) {
    double* buf = nullptr;
    cudaError_t e = cudaMalloc(&buf, sizeof(double) * 19 * (size_t)h->g.N);
    if (e != cudaSuccess) return cuda_check(h, e, "population buffer");
    const int odd = (int)(h->flow_iters & 1);
    const int grid = h->num_sms * 8;
    const SparseView S = view_of(h->flow_sp);
    switch (h->flow_prec) {
        case CLB_F64: k_flow_get_pops<double><<<grid, 256, 0, h->stream>>>((const double*)h->d_f, (const double*)h->d_flink, S, h->g, odd, buf); break;
        case CLB_F32: k_flow_get_pops<float><<<grid, 256, 0, h->stream>>>((const float*)h->d_f, (const float*)h->d_flink, S, h->g, odd, buf); break;
        default: k_flow_get_pops<__half><<<grid, 256, 0, h->stream>>>((const __half*)h->d_f, (const __half*)h->d_flink, S, h->g, odd, buf); break;
    }
    e = cudaMemcpyAsync(host, buf, sizeof(double) * 19 * (size_t)h->g.N, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    cudaFree(buf);
    return cuda_check(h, e, "population copy");
}

clb_status flow_set_populations(clb_handle* h, const double* host) {
    double* buf = nullptr;
    cudaError_t e = cudaMalloc(&buf, sizeof(double) * 19 * (size_t)h->g.N);
    if (e != cudaSuccess) return cuda_check(h, e, "population buffer");
    e = cudaMemcpyAsync(buf, host, sizeof(double) * 19 * (size_t)h->g.N, cudaMemcpyHostToDevice, h->stream);
    if (e != cudaSuccess) { cudaFree(buf); return cuda_check(h, e, "population copy"); }
    const int odd = (int)(h->flow_iters & 1);
    const int grid = h->num_sms * 8;
    const SparseView S = view_of(h->flow_sp);
    switch (h->flow_prec) {
        case CLB_F64: k_flow_set_pops<double><<<grid, 256, 0, h->stream>>>((double*)h->d_f, (double*)h->d_flink, S, h->g, odd, buf); break;
        case CLB_F32: k_flow_set_pops<float><<<grid, 256, 0, h->stream>>>((float*)h->d_f, (float*)h->d_flink, S, h->g, odd, buf); break;
        default: k_flow_set_pops<__half><<<grid, 256, 0, h->stream>>>((__half*)h->d_f, (__half*)h->d_flink, S, h->g, odd, buf); break;
    }
    e = cudaStreamSynchronize(h->stream);
    cudaFree(buf);
    return cuda_check(h, e, "set populations");
}

clb_status flow_stats(clb_handle* h, double char_length, clb_flow_stats* out) {
    double* u = nullptr;
    double* acc = nullptr;
    cudaError_t e = cudaMalloc(&u, sizeof(double) * 3 * (size_t)h->g.N);
    if (e != cudaSuccess) return cuda_check(h, e, "stats buffer");
    e = cudaMalloc(&acc, sizeof(double) * 3);
    if (e != cudaSuccess) { cudaFree(u); return cuda_check(h, e, "stats buffer"); }
    clb_status s = flow_velocity(h, u, 0, false);
    if (s != CLB_OK) { cudaFree(u); cudaFree(acc); return s; }
    double init[3] = {0.0, 0.0, 0.0};
    long long neg = (long long)0x8000000000000000ULL;  // below every ordered key
    std::memcpy(&init[1], &neg, sizeof(double));
    cudaMemcpyAsync(acc, init, sizeof(init), cudaMemcpyHostToDevice, h->stream);
    k_flow_vstats<<<h->num_sms * 4, 256, 0, h->stream>>>(u, h->g, acc);
    double r[3];
    Tracer t;
    cudaMemcpyAsync(r, acc, sizeof(r), cudaMemcpyDeviceToHost, h->stream);
    cudaMemcpyAsync(&t, h->d_tracer, sizeof(Tracer), cudaMemcpyDeviceToHost, h->stream);
    e = cudaStreamSynchronize(h->stream);
    cudaFree(u);
    cudaFree(acc);
    if (e != cudaSuccess) return cuda_check(h, e, "stats");
    long long key;
    std::memcpy(&key, &r[1], sizeof(key));
    long long bits = key >= 0 ? key : (key ^ 0x7fffffffffffffffLL);
    double mx;
    std::memcpy(&mx, &bits, sizeof(mx));
    const int64_t inner = (int64_t)(h->g.nx - 2) * h->g.plane;
    out->pore_mean_u = r[0] / (double)inner;
    out->pore_max_ux = mx;
    out->darcy_outlet_ux = r[2] / (double)h->g.plane;
    const double nu = (h->d.tau - 0.5) / 3.0;
    out->permeability = h->delta_p != 0 ? out->darcy_outlet_ux * nu * char_length / h->delta_p : 0.0;
    out->energy = t.energy;
    out->iterations = t.iterations;
    out->bgk_nodes = h->fp.n_bgk;
    out->active_nodes = h->flow_sp.K;
    return CLB_OK;
}

// Times the kernels of a step without the tracer (the default, the streamed step; even step through TMA tiles or
// not with the odd step compiled for 2 or 3 resident CTAs or pipelined through shared memory) over `steps`
// steps and keeps the fastest for such steps; a solve's, which are traced and on a small lattice go many to a
// launch, keep theirs. A key's choice before it lapses. The lattice state is saved before and restored
// after, so the run is unchanged. Writes a one-line report into `report`.
clb_status flow_autotune(clb_handle* h, int steps, char* report, int report_len) {
    if (steps < 2) steps = 2;
    steps += steps & 1;
    const size_t es = storage_size(h->flow_prec);
    const size_t fb = es * 19 * (size_t)h->flow_sp.KS, lb = es * (size_t)std::max<int64_t>(1, h->flow_sp.L) + 16;
    void* sf = nullptr;
    void* sl = nullptr;
    cudaError_t e = cudaMalloc(&sf, fb);
    if (e == cudaSuccess) e = cudaMalloc(&sl, lb);
    if (e != cudaSuccess) { cudaFree(sf); return cuda_check(h, e, "autotune buffers"); }
    Tracer tsave;
    cudaMemcpyAsync(sf, h->d_f, fb, cudaMemcpyDeviceToDevice, h->stream);
    cudaMemcpyAsync(sl, h->d_flink, lb, cudaMemcpyDeviceToDevice, h->stream);
    cudaMemcpyAsync(&tsave, h->d_tracer, sizeof(Tracer), cudaMemcpyDeviceToHost, h->stream);
    cudaStreamSynchronize(h->stream);
    const int64_t iters0 = h->flow_iters;
    const int save_tma = h->flow_even_tma, save_minb = h->flow_minb, save_pipe = h->flow_odd_pipe;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    float best = 1e30f;
    int best_tma = save_tma, best_minb = save_minb, best_pipe = save_pipe;
    std::string rep;
    auto timed = [&]() {
        flow_step(h, 4, false, 0.0);  // warm
        cudaEventRecord(a, h->stream);
        flow_step(h, steps, false, 0.0);
        cudaEventRecord(b, h->stream);
        cudaEventSynchronize(b);
        float ms = 0;
        cudaEventElapsedTime(&ms, a, b);
        return ms;
    };
    h->flow_keyed = h->flow_tuned = false;
    const float base = timed();
    {
        char buf[64];
        snprintf(buf, sizeof(buf), "stream:%.1fus", 1e3f * base / steps);
        rep += buf;
    }
    h->flow_tuned = true;
    for (int tma = 1; tma >= 0; --tma)
        for (int v = 0; v < 3; ++v) {  // odd step: 3 or 2 resident CTAs, or pipelined
            const int minb = v == 1 ? 2 : 3, pipe = v == 2 ? 1 : 0;
            if (pipe && !h->flow_pipe_grid) continue;
            h->flow_even_tma = tma;
            h->flow_minb = minb;
            h->flow_odd_pipe = pipe;
            h->flow_grid = flow_gather_grid(h);
            const float ms = timed();
            char buf[96];
            if (pipe) snprintf(buf, sizeof(buf), "%stma=%d,pipe:%.1fus", rep.empty() ? "" : " ", tma, 1e3f * ms / steps);
            else snprintf(buf, sizeof(buf), "%stma=%d,minb=%d:%.1fus", rep.empty() ? "" : " ", tma, minb, 1e3f * ms / steps);
            rep += buf;
            if (ms < best) { best = ms; best_tma = tma; best_minb = minb; best_pipe = pipe; }
        }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    h->flow_even_tma = best_tma;
    h->flow_minb = best_minb;
    h->flow_odd_pipe = best_pipe;
    h->flow_tuned = best < base;
    h->flow_grid = flow_gather_grid(h);
    cudaMemcpyAsync(h->d_f, sf, fb, cudaMemcpyDeviceToDevice, h->stream);
    cudaMemcpyAsync(h->d_flink, sl, lb, cudaMemcpyDeviceToDevice, h->stream);
    cudaMemcpyAsync(h->d_tracer, &tsave, sizeof(Tracer), cudaMemcpyHostToDevice, h->stream);
    e = cudaStreamSynchronize(h->stream);
    cudaFree(sf);
    cudaFree(sl);
    h->flow_iters = iters0;
    char buf[64];
    if (!h->flow_tuned) snprintf(buf, sizeof(buf), " -> stream");
    else if (best_pipe) snprintf(buf, sizeof(buf), " -> tma=%d,pipe", best_tma);
    else snprintf(buf, sizeof(buf), " -> tma=%d,minb=%d", best_tma, best_minb);
    rep += buf;
    if (report && report_len > 0) {
        std::strncpy(report, rep.c_str(), (size_t)report_len - 1);
        report[report_len - 1] = 0;
    }
    return cuda_check(h, e, "autotune");
}

}  // namespace clb
