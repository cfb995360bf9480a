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
                 const SparseView S, const double* __restrict__ neu, const AdeStep<TC> P, int64_t kw, int64_t ke) {
    extern __shared__ __align__(16) unsigned char stream_smem[];
    const int64_t k = (int64_t)blockIdx.x * STREAM_THREADS + threadIdx.x;
    ade_stream_node<TS, TC, ODD, U, LAW, STREAM_THREADS>(g, imm, bio, u, S, neu, P, kw, ke, stream_smem, k, k < S.K);
}

bool ade_streams(const AdeParams& P) {
    return P.law2 == CLB_LAW_NONE && !P.dis_on && !P.gate_on && P.law != CLB_LAW_SYMBOLIC;
}

template <typename TS, typename TC, bool ODD>
static void launch_stream_t(clb_handle* h) {
    const SparseView S = view_of(h->ade_sp);
    const AdeStep<TC> P = ade_step_params<TC>(h->ap, h->n_mobile);
    const unsigned grid = (unsigned)std::max<int64_t>(1, (S.K + STREAM_THREADS - 1) / STREAM_THREADS);
    const StreamLaw law = stream_law(P, sizeof(TS));
    const size_t sm = (size_t)stream_bytes<TC>(law, h->n_mobile) * STREAM_THREADS;
    auto go = [&](auto kern) {
        kern<<<grid, STREAM_THREADS, sm, h->stream>>>((TS*)h->d_g, h->d_imm, h->d_bio, (const TC*)h->d_u, S, h->d_neu, P,
                                                      h->ade_west_end, h->ade_east_begin);
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

void launch_ade_stream(clb_handle* h, bool odd) {
    ++h->launches;
    switch (h->ade_prec) {
        case CLB_F64: if (odd) launch_stream_t<double, double, true>(h); else launch_stream_t<double, double, false>(h); break;
        case CLB_F32: if (odd) launch_stream_t<float, float, true>(h); else launch_stream_t<float, float, false>(h); break;
        default: if (odd) launch_stream_t<__half, float, true>(h); else launch_stream_t<__half, float, false>(h); break;
    }
}

// ------------------------------------------------------------------ a batch of domains

// One block per tile of the batch's table: the tile's domain goes to shared memory, then the block
// walks the tile 128 nodes at a time. 96 uneven domains of 3 FP32 Monod species (2.9 M nodes): 138 us
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
