// ade_stream.cu -- the transport step with every species streamed through registers (ade_stream.cuh):
// the launches of one domain and of a batch of domains.
//
// The step is bound by HBM, and by how its requests reach it more than by their number: one thread
// per node and one block per 128 nodes keeps the blocks in flight next to one another in every row,
// and 32 warps per SM with 7 U loads each in flight are enough. More of either is slower: 256^3 pack,
// 8 FP32 species, per step: 8 blocks per SM 0.680 ms, 9 blocks 0.746 ms, 5 blocks of 256 threads
// 0.805 ms, four species in flight 0.95 ms, a persistent grid with the next node's metadata
// prefetched 0.88 ms; the staged form 0.892 ms. Algorithmic traffic of the same step: 3.48 -> 4.57
// TB/s. Other shapes (staged -> streamed, us per step): 129x97x113 with 3 Monod species 34.0 -> 25.6;
// 200x160x160 with one decaying species 66.2 -> 38.1; 200x131x143 with 5 species, FP64 dual Monod
// 253 -> 186, FP16 Monod 172 -> 84.
#include "ade_stream.cuh"
#include "batch.cuh"
#include "grid_sync.cuh"

#include <algorithm>
#include <vector>

namespace clb {

constexpr int STREAM_THREADS = 128;

// Species in flight per thread: two 4- or 2-byte species, one 8-byte species (the same bytes; two
// spill at 64 registers: 199 us per step instead of 186).
template <typename TC>
constexpr int stream_width() { return sizeof(TC) == 8 ? 1 : 2; }

// Resident blocks the registers are budgeted for: 64 registers (8 blocks); a single 4- or 2-byte
// species fits 10 blocks (42.2 -> 38.1 us on 200x160x160).
template <typename TC, int U>
constexpr int stream_blocks() { return sizeof(TC) == 4 && U == 1 ? 10 : 8; }

template <typename TS, typename TC, bool ODD, int U, int LAW>
__global__ void __launch_bounds__(STREAM_THREADS, (stream_blocks<TC, U>()))
    k_ade_stream(TS* __restrict__ g, double* __restrict__ imm, double* __restrict__ bio, const TC* __restrict__ u,
                 const SparseView S, const double* neu, const AdeStep<TC> P, int64_t kw, int64_t ke) {
    extern __shared__ __align__(16) unsigned char stream_smem[];
    const int64_t k = (int64_t)blockIdx.x * STREAM_THREADS + threadIdx.x;
    ade_stream_node<TS, TC, ODD, U, LAW, STREAM_THREADS>(g, imm, bio, u, S, neu, P, kw, ke, stream_smem, k, k < S.K);
}

bool ade_streams(const AdeParams& P) {
    return P.law2 == CLB_LAW_NONE && !P.dis_on && !P.gate_on && P.law != CLB_LAW_SYMBOLIC;
}

template <typename TS, typename TC, bool ODD>
static void launch_stream_t(clb_handle* h, bool after) {
    const SparseView S = view_of(h->ade_sp);
    const AdeStep<TC> P = ade_step_params<TC>(h->ap, h->n_mobile);
    const unsigned grid = (unsigned)std::max<int64_t>(1, (S.K + STREAM_THREADS - 1) / STREAM_THREADS);
    const StreamLaw law = stream_law(P, sizeof(TS));
    const size_t sm = (size_t)stream_bytes<TC>(law, h->n_mobile) * STREAM_THREADS;
    auto go = [&](auto kern) {
        launch_step(after, kern, grid, STREAM_THREADS, sm, h->stream, (TS*)h->d_g, h->d_imm, h->d_bio, (const TC*)h->d_u, S,
                    h->d_neu, P, h->ade_west_end, h->ade_east_begin);
    };
    constexpr int U = stream_width<TC>();
    const bool one = h->n_mobile == 1;
    if (law == STREAM_NONE) {
        if (one) go(k_ade_stream<TS, TC, ODD, 1, STREAM_NONE>);
        else go(k_ade_stream<TS, TC, ODD, U, STREAM_NONE>);
    } else if (law == STREAM_SEPARABLE) {
        if (one) go(k_ade_stream<TS, TC, ODD, 1, STREAM_SEPARABLE>);
        else go(k_ade_stream<TS, TC, ODD, U, STREAM_SEPARABLE>);
    } else if (law == STREAM_DUAL_AHEAD) {
        go(k_ade_stream<TS, TC, ODD, U, STREAM_DUAL_AHEAD>);
    } else if constexpr (sizeof(TS) >= 4) {
        go(k_ade_stream<TS, TC, ODD, U, STREAM_DUAL_AFTER>);
    }
}

void launch_ade_stream(clb_handle* h, bool odd, bool after) {
    ++h->launches;
    switch (h->ade_prec) {
        case CLB_F64: if (odd) launch_stream_t<double, double, true>(h, after); else launch_stream_t<double, double, false>(h, after); break;
        case CLB_F32: if (odd) launch_stream_t<float, float, true>(h, after); else launch_stream_t<float, float, false>(h, after); break;
        default: if (odd) launch_stream_t<__half, float, true>(h, after); else launch_stream_t<__half, float, false>(h, after); break;
    }
}

// ------------------------------------------------------------------ Neumann planes

// The stored density of a Neumann plane node is its inner neighbour's as it stands before the step
// (FlatAdiabaticBoundaryFunctional3D after the previous stream); a node whose inner neighbour is not a
// fluid node keeps its previous value. One thread per plane pixel, side and species, the neighbour's slots
// from the step's metadata: three dependent reads (compact indices, metadata, populations), which is what
// bounds it. FP32, us per step: 8 species of 256x256 pixels 9.1, 96 uneven domains of 3 species 9.8; from
// the dense neighbour lookups (five dependent reads, 64-bit divisions, a search for the batch's
// domain) 12.7 and 13.4.
template <typename TS, typename TC, bool ODD>
__device__ __forceinline__ void neumann_pixel(const TS* g, const SparseView& S, const int8_t* dyn, int nx, int plane,
                                              int side, int p, int s, bool on, double* neu) {
    const int64_t nb = side == 0 ? p : (int64_t)(nx - 1) * plane + p, ni = side == 0 ? nb + plane : nb - plane;
    const int kb = on ? S.idx_of[nb] : -1, ki = on ? S.idx_of[ni] : -1;
    uint32_t off[7];
    on = kb >= 0 && ki >= 0;
    if (on) {
        const int db = dyn[S.code[kb]], di = dyn[S.code[ki]];
        stream_slots<ODD>(S, ki, S.meta[ki], off);
        on = (db == ADE_PORE || db == ADE_BIO) && (di == ADE_PORE || di == ADE_BIO);
    }
    step_wait();
    if (!on) return;
    const TS* f = g + (int64_t)s * S.SS;
    TC pop[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) pop[i] = ld<TS, TC>(f + off[i]);
    double r = ade_sigma<TC>();
#pragma unroll
    for (int i = 0; i < 7; ++i) r += (double)pop[i];
    neu[((int64_t)s * 2 + side) * plane + p] = r;
}

// The species with a Neumann face, by side, and what the planes need of the domain.
struct NeumannPlanes {
    int nx, plane;
    int n[2];
    int8_t s[2][CLB_MAX_SPECIES];
    int8_t dyn[MAX_CODES];
};

template <typename TS, typename TC, bool ODD>
__global__ void __launch_bounds__(STREAM_THREADS) k_neumann(const TS* g, const SparseView S, const NeumannPlanes J, double* neu) {
    const int p = blockIdx.x * STREAM_THREADS + threadIdx.x, side = blockIdx.y, j = blockIdx.z;
    const bool on = p < J.plane && j < J.n[side];
    neumann_pixel<TS, TC, ODD>(g, S, J.dyn, J.nx, J.plane, side, p, on ? J.s[side][j] : 0, on, neu);
}

bool launch_ade_neumann(clb_handle* h, bool odd, bool after) {
    NeumannPlanes J;
    J.nx = h->g.nx;
    J.plane = h->g.plane;
    J.n[0] = J.n[1] = 0;
    for (int s = 0; s < h->n_mobile; ++s) {  // internal order: the mobile species first
        if (h->ap.ltype[s] == CLB_NEUMANN) J.s[0][J.n[0]++] = (int8_t)s;
        if (h->ap.rtype[s] == CLB_NEUMANN) J.s[1][J.n[1]++] = (int8_t)s;
    }
    const int most = std::max(J.n[0], J.n[1]);
    if (most == 0) return false;
    std::memcpy(J.dyn, h->ap.dyn, sizeof(J.dyn));
    const dim3 grid((unsigned)((h->g.plane + STREAM_THREADS - 1) / STREAM_THREADS), 2, (unsigned)most);
    ++h->launches;
#define CLB_NEU(TS, TC)                                                                                                    \
    launch_step(after, odd ? k_neumann<TS, TC, true> : k_neumann<TS, TC, false>, grid, STREAM_THREADS, 0, h->stream,                 \
                (const TS*)h->d_g, view_of(h->ade_sp), J, h->d_neu);
    switch (h->ade_prec) {
        case CLB_F64: CLB_NEU(double, double); break;
        case CLB_F32: CLB_NEU(float, float); break;
        default: CLB_NEU(__half, float); break;
    }
#undef CLB_NEU
    return true;
}

// ------------------------------------------------------------------ many steps of a small lattice

// `steps` steps in one cooperative launch, for lattices small enough that a step is mostly latency (two
// launches, the Neumann planes' and the step's, their ramp-up and the metadata): every node has a resident
// thread that keeps its slots of both parities, and the blocks meet at a grid-wide barrier between steps.
//
// A Neumann face imposes the density its node's inner neighbour has before the step, which the
// neighbour's own update overwrites. So the thread of such a face node takes the inner neighbour too: the
// face node first, reading the neighbour's populations, then the neighbour; the neighbour's own thread
// leaves it out. (nx >= 4, so that no inner node belongs to two faces.)
constexpr int STREAM_MULTI_THREADS = 256;

template <typename TS, typename TC, int U, int LAW>
__global__ void __launch_bounds__(STREAM_MULTI_THREADS, 2)
    k_ade_stream_multi(TS* g, double* imm, double* bio, const TC* u, const SparseView S, const double* neu, const AdeStep<TC> P,
                       int64_t kw, int64_t ke, int neumann, int steps, int odd, GridSync* gs, uint32_t polls, int* gave_up) {
    extern __shared__ __align__(16) unsigned char stream_smem[];
    constexpr int T = STREAM_MULTI_THREADS;
    struct Node {
        StreamNode<TC> A;
        uint32_t even[7], odd[7];
    };
    auto fluid = [&](int k) {
        const int d = P.dyn[S.code[k]];
        return d == ADE_PORE || d == ADE_BIO;
    };
    // the x-face partner of node k: for a face node its inner neighbour, for a node next to a face the
    // face node, where a Neumann face couples the two (both fluid); else -1
    auto partner = [&](int64_t k) {
        const int n = S.node[k], x = n / P.plane, nx = (int)(P.N / P.plane);
        const int d = x == 0 ? 1 : x == 1 ? -1 : x == nx - 1 ? -1 : x == nx - 2 ? 1 : 0;
        if (d == 0 || !((neumann >> (x <= 1 ? 0 : 1)) & 1)) return -1;
        const int j = S.idx_of[n + (int64_t)d * P.plane];
        return j >= 0 && fluid((int)k) && fluid(j) ? j : -1;
    };
    auto load = [&](int64_t k) {
        Node N;
        const uint32_t mt = S.meta[k];
        N.A = stream_node<TC, LAW>(S, P, u, k);
        stream_slots<false>(S, k, mt, N.even);
        stream_slots<true>(S, k, mt, N.odd);
        return N;
    };
    auto step = [&](int64_t k, const Node& N, int64_t kp, const Node& I, bool odd_step) {
        auto run = [&](const uint32_t(&off)[7], const uint32_t(&in)[7]) {
            ade_stream_species<TS, TC, U, LAW, T, false>(
                g, imm, bio, S, P, kw, ke, stream_smem, k, N.A, off, true, [&](int s, bool west) {
                    if (kp < 0) return neu[((int64_t)s * 2 + (west ? 0 : 1)) * P.plane + S.node[k] % P.plane];
                    const TS* f = g + (int64_t)s * S.SS;
                    double r = ade_sigma<TC>();
#pragma unroll
                    for (int i = 0; i < 7; ++i) r += (double)ld<TS, TC>(f + in[i]);
                    return r;
                });
            if (kp >= 0)
                ade_stream_species<TS, TC, U, LAW, T, false>(g, imm, bio, S, P, kw, ke, stream_smem, kp, I.A, in, true,
                                                             [](int, bool) { return 0.0; });
        };
        if (odd_step) run(N.odd, I.odd);
        else run(N.even, I.even);
    };
    if (*(volatile unsigned*)&gs->abort) return;  // a launch of the same call before this one gave up
    const int64_t k = (int64_t)blockIdx.x * T + threadIdx.x;
    Node N = {}, I = {};
    int64_t kp = -1;
    bool mine = false;
    if (k < S.K) {
        // a node next to a face whose partner exists belongs to the partner's thread
        const bool face = k < kw || k >= ke;
        kp = partner(k);
        mine = face || kp < 0;
        if (!face) kp = -1;
        if (mine) {
            N = load(k);
            if (kp >= 0) I = load(kp);
        }
    }
    for (int t = 0; t < steps; ++t) {
        const bool odd_step = ((odd + t) & 1) != 0;
        if (mine) step(k, N, kp, I, odd_step);
        if (!grid_barrier(gs, (unsigned)t + 1, polls)) {
            if (threadIdx.x == 0) *(volatile int*)gave_up = 1;
            return;
        }
    }
}

// Lattices whose steps go many to a launch: up to two mobile species and by nodes x species, since a
// chained launch per step has the whole chip per species group where this one has a barrier. us per step, chained
// launches -> many steps per launch (FP64; FP32):
//   one species:   11 k nodes 7.4 -> 3.2; 4.9 -> 3.0    53 k 7.6 -> 3.7; 4.8 -> 3.4    76 k 7.4 -> 5.7; 4.9 -> 5.5
//   two (Monod):   11 k 7.5 -> 4.4; 4.8 -> 4.2          27 k 7.3 -> 4.6; 4.9 -> 4.2    43 k 7.4 -> 5.7; 4.9 -> 5.0
//   three (Monod): 11 k 5.8 -> 5.3; 5.3 -> 5.2          27 k 7.5 -> 6.2; 5.5 -> 5.6    43 k 6.3 -> 7.8; 5.6 -> 6.7
//   four (dual):   11 k 7.3 -> 8.7; 6.7 -> 7.7          27 k 7.9 -> 8.9; 6.7 -> 8.0
constexpr int STREAM_MULTI_SPECIES = 2;
constexpr int64_t STREAM_MULTI_VALUES = 60000;
constexpr int STREAM_MULTI_STEPS = 1024, STREAM_MULTI_MIN_STEPS = 3;

template <typename TS, typename TC>
static bool launch_stream_multi_t(clb_handle* h, int steps, cudaError_t& e) {
    SparseView S = view_of(h->ade_sp);
    if (S.K < 1 || h->n_mobile > STREAM_MULTI_SPECIES || S.K * std::max(1, h->n_mobile) > STREAM_MULTI_VALUES) return false;
    AdeStep<TC> P = ade_step_params<TC>(h->ap, h->n_mobile);
    const StreamLaw law = stream_law(P, sizeof(TS));
    const size_t sm = (size_t)stream_bytes<TC>(law, h->n_mobile) * STREAM_MULTI_THREADS;
    if (sm > 48 * 1024) return false;
    int neumann = 0;
    for (int s = 0; s < h->n_mobile; ++s) {
        if (P.ltype[s] == CLB_NEUMANN) neumann |= 1;
        if (P.rtype[s] == CLB_NEUMANN) neumann |= 2;
    }
    auto go = [&](auto kern) {
        const int64_t need = (S.K + STREAM_MULTI_THREADS - 1) / STREAM_MULTI_THREADS;
        int per = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, STREAM_MULTI_THREADS, sm) != cudaSuccess ||
            need > (int64_t)per * h->num_sms)
            return false;
        TS* g = (TS*)h->d_g;
        const TC* u = (const TC*)h->d_u;
        const double* neu = h->d_neu;
        GridSync* gs = (GridSync*)h->d_sync;
        uint32_t polls = (uint32_t)h->barrier_polls;
        int* gave_up = h->d_flags + FLAG_ADE_WAIT;
        int odd = (int)(h->ade_iters & 1);
        for (int t = 0; t < steps; t += STREAM_MULTI_STEPS, odd ^= STREAM_MULTI_STEPS & 1) {
            int n = std::min(STREAM_MULTI_STEPS, steps - t);
            void* args[] = {&g, &h->d_imm, &h->d_bio, &u, &S, &neu, &P, &h->ade_west_end, &h->ade_east_begin, &neumann, &n, &odd,
                            &gs, &polls, &gave_up};
            if ((e = cudaMemsetAsync(&gs->arrived, 0, sizeof(gs->arrived), h->stream)) != cudaSuccess) return true;
            ++h->launches;
            e = cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)need), dim3(STREAM_MULTI_THREADS), args, sm, h->stream);
            if (e != cudaSuccess) return true;
        }
        return true;
    };
    constexpr int U = stream_width<TC>();
    const bool single = h->n_mobile == 1;
    if (law == STREAM_NONE)
        return single ? go(k_ade_stream_multi<TS, TC, 1, STREAM_NONE>)
                      : go(k_ade_stream_multi<TS, TC, U, STREAM_NONE>);
    if (law == STREAM_SEPARABLE)
        return single ? go(k_ade_stream_multi<TS, TC, 1, STREAM_SEPARABLE>)
                      : go(k_ade_stream_multi<TS, TC, U, STREAM_SEPARABLE>);
    if (law == STREAM_DUAL_AHEAD)
        return go(k_ade_stream_multi<TS, TC, U, STREAM_DUAL_AHEAD>);
    if constexpr (sizeof(TS) >= 4)
        return go(k_ade_stream_multi<TS, TC, U, STREAM_DUAL_AFTER>);
    return false;
}

bool launch_ade_multi(clb_handle* h, int steps, cudaError_t& e) {
    e = cudaSuccess;
    if (steps < STREAM_MULTI_MIN_STEPS || h->g.nx < 4 || !h->d_sync) return false;
    switch (h->ade_prec) {
        case CLB_F64: return launch_stream_multi_t<double, double>(h, steps, e);
        case CLB_F32: return launch_stream_multi_t<float, float>(h, steps, e);
        default: return launch_stream_multi_t<__half, float>(h, steps, e);
    }
}

// ------------------------------------------------------------------ a batch of domains

// One block per tile of the batch's table, one thread per node of it: the tile's domain goes to shared
// memory, then the nodes are stepped. 96 uneven domains of 3 FP32 Monod species (2.9 M nodes): 138 us
// per step where the staged form (persistent blocks over runs of the table) took 198.
template <typename TS, typename TC, bool ODD, int U, int LAW>
__global__ void __launch_bounds__(STREAM_THREADS, (stream_blocks<TC, U>()))
    k_ade_stream_batch(const BatchTile* __restrict__ tiles, const StreamDomain<TC>* __restrict__ dom) {
    extern __shared__ __align__(16) unsigned char stream_smem[];
    __shared__ __align__(16) StreamDomain<TC> D;
    static_assert(sizeof(D) % 8 == 0, "copied by 8-byte words");
    const BatchTile T = tiles[blockIdx.x];
    const uint64_t* src = reinterpret_cast<const uint64_t*>(dom + T.d);
    uint64_t* dst = reinterpret_cast<uint64_t*>(&D);
    for (int q = threadIdx.x; q < (int)(sizeof(D) / 8); q += STREAM_THREADS) dst[q] = src[q];
    __syncthreads();
    for (int i = 0; i < T.count; i += STREAM_THREADS) {
        const int j = i + (int)threadIdx.x;
        ade_stream_node<TS, TC, ODD, U, LAW, STREAM_THREADS>((TS*)D.g, D.imm, D.bio, (const TC*)D.u, D.S, D.neu, D.P, D.kw,
                                                             D.ke, stream_smem, T.first + j, j < T.count);
    }
}

template <typename TS, typename TC, bool ODD>
static void launch_stream_batch_t(const BatchView& B, cudaStream_t st) {
    constexpr int U = stream_width<TC>();
    auto go = [&](auto kern, StreamLaw law) {
        const int n = B.alaw[law + 1] - B.alaw[law];
        if (n == 0) return;
        const size_t sm = (size_t)stream_bytes<TC>(law, B.max_mobile) * STREAM_THREADS;
        kern<<<n, STREAM_THREADS, sm, st>>>(B.atiles + B.alaw[law], static_cast<const StreamDomain<TC>*>(B.sdom));
    };
    if (B.max_mobile <= 1) {
        go(k_ade_stream_batch<TS, TC, ODD, 1, STREAM_NONE>, STREAM_NONE);
        go(k_ade_stream_batch<TS, TC, ODD, 1, STREAM_SEPARABLE>, STREAM_SEPARABLE);
    } else {
        go(k_ade_stream_batch<TS, TC, ODD, U, STREAM_NONE>, STREAM_NONE);
        go(k_ade_stream_batch<TS, TC, ODD, U, STREAM_SEPARABLE>, STREAM_SEPARABLE);
    }
    if constexpr (sizeof(TS) >= 4) go(k_ade_stream_batch<TS, TC, ODD, U, STREAM_DUAL_AFTER>, STREAM_DUAL_AFTER);
    go(k_ade_stream_batch<TS, TC, ODD, U, STREAM_DUAL_AHEAD>, STREAM_DUAL_AHEAD);
}

// the Neumann planes of every domain: one block per run of pixels of a face, one y-block per species
template <typename TS, typename TC, bool ODD>
__global__ void __launch_bounds__(STREAM_THREADS) k_neumann_batch(const NeumannTile* __restrict__ tiles,
                                                                  const StreamDomain<TC>* __restrict__ dom) {
    const NeumannTile T = tiles[blockIdx.x];
    const StreamDomain<TC>& D = dom[T.d];
    const int s = blockIdx.y, p = T.first + (int)threadIdx.x;
    const bool on = p < D.P.plane && s < D.P.n_mobile && (T.side == 0 ? D.P.ltype[s] : D.P.rtype[s]) == CLB_NEUMANN;
    neumann_pixel<TS, TC, ODD>((const TS*)D.g, D.S, D.P.dyn, (int)(D.P.N / D.P.plane), D.P.plane, T.side, p, s, on,
                               const_cast<double*>(D.neu));
}

void launch_neumann_batch(const BatchView& B, int prec, bool odd, cudaStream_t st) {
    if (B.nnt == 0) return;
    const dim3 grid((unsigned)B.nnt, (unsigned)std::max(1, B.max_mobile));
#define CLB_NEU(TS, TC)                                                                                                  \
    if (odd) k_neumann_batch<TS, TC, true><<<grid, STREAM_THREADS, 0, st>>>(B.ntiles, static_cast<const StreamDomain<TC>*>(B.sdom)); \
    else k_neumann_batch<TS, TC, false><<<grid, STREAM_THREADS, 0, st>>>(B.ntiles, static_cast<const StreamDomain<TC>*>(B.sdom));
    switch (prec) {
        case CLB_F64: CLB_NEU(double, double); break;
        case CLB_F32: CLB_NEU(float, float); break;
        default: CLB_NEU(__half, float); break;
    }
#undef CLB_NEU
}

void launch_ade_batch(const BatchView& B, int prec, bool odd, cudaStream_t st) {
    switch (prec) {
        case CLB_F64: if (odd) launch_stream_batch_t<double, double, true>(B, st); else launch_stream_batch_t<double, double, false>(B, st); break;
        case CLB_F32: if (odd) launch_stream_batch_t<float, float, true>(B, st); else launch_stream_batch_t<float, float, false>(B, st); break;
        default: if (odd) launch_stream_batch_t<__half, float, true>(B, st); else launch_stream_batch_t<__half, float, false>(B, st); break;
    }
}

template <typename TC>
static cudaError_t stream_domains_t(clb_handle* const* hs, int n, int storage, void** dev, std::vector<int>& form) {
    std::vector<StreamDomain<TC>> dom((size_t)n);
    form.assign((size_t)n, STREAM_NONE);
    for (int i = 0; i < n; ++i) {
        const clb_handle* h = hs[i];
        StreamDomain<TC>& D = dom[(size_t)i];
        std::memset(&D, 0, sizeof(D));
        D.g = h->d_g;
        D.imm = h->d_imm;
        D.bio = h->d_bio;
        D.u = h->d_u;
        D.neu = h->d_neu;
        D.kw = h->ade_west_end;
        D.ke = h->ade_east_begin;
        D.S = view_of(h->ade_sp);
        D.P = ade_step_params<TC>(h->ap, h->n_mobile);
        form[(size_t)i] = stream_law(D.P, storage);
    }
    cudaError_t e = cudaMalloc(dev, sizeof(StreamDomain<TC>) * (size_t)n);
    if (e == cudaSuccess) e = cudaMemcpy(*dev, dom.data(), sizeof(StreamDomain<TC>) * (size_t)n, cudaMemcpyHostToDevice);
    return e;
}

cudaError_t stream_domains(clb_handle* const* hs, int n, int prec, void** dev, std::vector<int>& form) {
    return prec == CLB_F64 ? stream_domains_t<double>(hs, n, 8, dev, form)
                           : stream_domains_t<float>(hs, n, prec == CLB_F32 ? 4 : 2, dev, form);
}

}  // namespace clb
