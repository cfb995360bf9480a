// ade_stream.cu -- the transport step with every species streamed through registers (ade_stream.cuh):
// the single-domain launches.
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

#include <algorithm>

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

}  // namespace clb
