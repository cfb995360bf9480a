// ade_stream.cuh -- one node of the transport step for rate laws that act species by species (no
// law, decay, Monod) or only where biomass is (dual Monod), with every species streamed through
// registers: gather, collide, deposit and scatter one group of species before the next is read.
// Shared by the single-domain step and the batched step of many domains.
//
// Why streamed: a species' new populations need its own density and its own increment only, so a
// node's species have no reason to be resident together. The staged form of the step (ade.cu,
// ade_gather / ade_finish, still used where an abiotic law, a gate or a rate-law file couples the
// species) passes all 7 S populations of a node through shared memory: 1781 warp instructions per
// 32 nodes at 8 species and 16 to 20 resident warps per SM. Dual Monod couples the donor and the
// acceptors only, and only where an organism lives (the biomass flag, about 2 % of the nodes), so
// those nodes read the coupled densities once more ahead of the loop and park the increments.
#pragma once

#include "flow_node.cuh"
#include "kinetics.cuh"
#include "step_chain.cuh"
#include "tma.cuh"

#include <cstring>

namespace clb {

// What the streamed step reads of a domain's parameters, in the arithmetic type and small enough
// that a launch carries it cheaply.
template <typename TC>
struct AdeStep {
    int plane;
    int64_t N;
    int S, M, n_mobile, law;
    TC dt;
    TC mu, ks, inv_y, kd;                       // dual Monod
    int donor, acceptor[CLB_MAX_MICROBES];      // internal species, -1 none
    int8_t dyn[MAX_CODES], react[MAX_CODES];
    int8_t ltype[CLB_MAX_SPECIES], rtype[CLB_MAX_SPECIES];
    double lbc[CLB_MAX_SPECIES], rbc[CLB_MAX_SPECIES];
    TC w[2][CLB_MAX_SPECIES];                   // relaxation: pore, biofilm
    TC k1[CLB_MAX_SPECIES], k2[CLB_MAX_SPECIES];  // decay: k; Monod: k and the half-saturation
    const uint8_t* bflag;
    int* nonfinite;
};

template <typename TC>
inline AdeStep<TC> ade_step_params(const AdeParams& P, int n_mobile) {
    AdeStep<TC> Q;
    std::memset(&Q, 0, sizeof(Q));
    Q.plane = P.g.plane;
    Q.N = P.g.N;
    Q.S = P.S;
    Q.M = P.M;
    Q.n_mobile = n_mobile;
    Q.law = P.law;
    Q.dt = (TC)P.dt;
    Q.mu = (TC)P.prm[0];
    Q.ks = (TC)P.prm[1];
    Q.inv_y = (TC)(1.0 / P.prm[2]);
    Q.kd = (TC)P.prm[3];
    Q.donor = P.donor;
    for (int m = 0; m < CLB_MAX_MICROBES; ++m) Q.acceptor[m] = P.acceptor[m];
    std::memcpy(Q.dyn, P.dyn, sizeof(Q.dyn));
    std::memcpy(Q.react, P.react, sizeof(Q.react));
    for (int s = 0; s < CLB_MAX_SPECIES; ++s) {
        Q.ltype[s] = (int8_t)P.ltype[s];
        Q.rtype[s] = (int8_t)P.rtype[s];
        Q.lbc[s] = P.lbc[s];
        Q.rbc[s] = P.rbc[s];
        Q.w[0][s] = (TC)P.wpore[s];
        Q.w[1][s] = (TC)P.wbio[s];
        Q.k1[s] = (TC)P.prm[s];
        Q.k2[s] = (TC)P.prm[CLB_MAX_SPECIES + s];
    }
    Q.bflag = P.bflag;
    Q.nonfinite = P.nonfinite;
    return Q;
}

// One domain of a batch as the streamed step sees it (device copy, one per domain).
template <typename TC>
struct StreamDomain {
    void* g;
    double* imm;
    double* bio;
    const void* u;
    const double* neu;
    int64_t kw, ke;
    SparseView S;
    AdeStep<TC> P;
};

// The increment of a species from its rate, with the thresholds and the clamp dC = max(R dt, -C).
template <typename TC>
__device__ __forceinline__ TC clamped_increment(TC R, TC dt, TC C) {
    const TC thr = (TC)THRD;
    TC d = R * dt;
    if (!(d > thr || d < -thr)) return (TC)0;
    if (d + C < (TC)0) d = -C;
    return (d > thr || d < -thr) ? d : (TC)0;
}

template <typename TC>
__device__ __forceinline__ TC floored(TC c) { return c < (TC)THRD ? (TC)0 : c; }

// rate of species s under a law without coupling, from its floored concentration
template <typename TC>
__device__ __forceinline__ TC separable_rate(const AdeStep<TC>& P, int s, TC C) {
    return P.law == CLB_LAW_DECAY ? -P.k1[s] * C : -P.k1[s] * C / (P.k2[s] + C);
}

// Dual Monod's rates (biotic_rates, kinetics.cuh) at a node that may hold biomass, from conc(s), the
// floored concentration of a species, and held(m, p), microbe m's biomass as it stands at p; biomass
// advances in place and every coupled species' increment goes to deposit(s, dC).
template <typename TC, typename Held, typename Conc, typename Deposit>
__device__ __forceinline__ void dual_monod(const AdeStep<TC>& P, double* bio, int64_t nd, Held held, Conc conc,
                                           Deposit deposit) {
    const TC thr = (TC)THRD;
    const TC Cd = conc(P.donor);
    TC Rd = 0;
    for (int m = 0; m < P.M; ++m) {
        const int a = P.acceptor[m];
        if (a < 0) continue;
        double* bp = bio + (int64_t)m * P.N + nd;
        const double braw = held(m, bp);
        const TC Bm = braw < THRD ? (TC)0 : (TC)braw;
        if (Bm <= (TC)0) continue;
        const TC Ca = conc(a);
        const TC growth = P.mu * Cd * Ca * Bm / ((P.ks + Cd) * (P.ks + Ca));
        const TC rbm = growth - P.kd * Bm;
        const TC gy = growth * P.inv_y;
        Rd -= gy;
        deposit(a, clamped_increment<TC>((TC)0 - gy, P.dt, Ca));
        TC d = rbm * P.dt;
        if (d > thr || d < -thr) {
            if (d + Bm < (TC)0) d = -Bm;
            *bp = braw + (double)d;
        }
    }
    deposit(P.donor, clamped_increment<TC>(Rd, P.dt, Cd));
}

// One species group's populations in registers between its gather and its scatter.
template <typename TS, typename TC>
__device__ __forceinline__ void ade_collide_store(TS* f, const uint32_t (&off)[7], const TC (&q)[7], TC rb, TC w, TC d,
                                                  TC ux, TC uy, TC uz, bool single) {
    const TC omw = (TC)1 - w;
    const TC rho = rb + (TC)ade_sigma<TC>();
    const TC jx = rho * ux, jy = rho * uy, jz = rho * uz;
    // feq_i = t_i (rb + 4 c_i . j), in opposite-pair form (no zero products)
    const TC r8 = (TC)0.125 * rb, d8 = (TC)0.125 * d;
    TC o[7];
    // q omw + w feq with the rounding written out (which product is rounded before the sum), so every
    // form of the step gives the same bits whatever the compiler contracts: the staged kernels
    // round w feq of the rest population where the handle has several species, q omw elsewhere
    const TC x0 = (TC)0.25 * rb;
    o[0] = (single ? fma(w, x0, q[0] * omw) : fma(q[0], omw, w * x0)) + (TC)0.25 * d;
    o[1] = fma(w, r8 - (TC)0.5 * jx, q[1] * omw) + d8;
    o[4] = fma(w, r8 + (TC)0.5 * jx, q[4] * omw) + d8;
    o[2] = fma(w, r8 - (TC)0.5 * jy, q[2] * omw) + d8;
    o[5] = fma(w, r8 + (TC)0.5 * jy, q[5] * omw) + d8;
    o[3] = fma(w, r8 - (TC)0.5 * jz, q[3] * omw) + d8;
    o[6] = fma(w, r8 + (TC)0.5 * jz, q[6] * omw) + d8;
#pragma unroll
    for (int j = 0; j < 7; ++j) st<TS, TC>(f + off[j], o[q7opp(j)]);  // outgoing opp(j) back to slot j
}

// How the rate law enters the streamed step.
//   none / separable (decay, Monod): each species from its own density.
//   dual after: dual Monod of up to two microbes with mobile partners, 4- and 8-byte storage. The
//     step runs as without a law and keeps the coupled densities; where biomass is, the increments
//     are added to the stored populations afterwards. A stored 4- or 8-byte population is the
//     collision's own value, so the sum is rounded as if the deposit had been added before the
//     store, and only the nodes with biomass (a few per cent) pay for the coupling.
//   dual ahead: dual Monod otherwise (immobile partners, 2-byte storage); the coupled densities are read once
//     more ahead of the step.
enum StreamLaw { STREAM_NONE, STREAM_SEPARABLE, STREAM_DUAL_AFTER, STREAM_DUAL_AHEAD };
constexpr int STREAM_MICROBES = 2;  // of "dual after"

template <typename TC>
inline StreamLaw stream_law(const AdeStep<TC>& P, int storage) {
    if (P.law == CLB_LAW_NONE) return STREAM_NONE;
    if (P.law != CLB_LAW_DUAL_MONOD) return STREAM_SEPARABLE;
    bool after = storage >= 4 && P.M <= STREAM_MICROBES && P.donor < P.n_mobile;
    for (int m = 0; m < P.M; ++m) after = after && P.acceptor[m] < P.n_mobile;
    return after ? STREAM_DUAL_AFTER : STREAM_DUAL_AHEAD;
}

// Bytes of shared memory per thread of the step: "after" keeps the biomass of two microbes and the
// densities of the donor and their acceptors, "ahead" every mobile species' increment.
template <typename TC>
constexpr int stream_bytes(StreamLaw law, int n_mobile) {
    return law == STREAM_DUAL_AFTER ? STREAM_MICROBES * (int)sizeof(double) + (1 + STREAM_MICROBES) * (int)sizeof(TC)
         : law == STREAM_DUAL_AHEAD ? n_mobile * (int)sizeof(TC) : 0;
}

// The 7 storage slots (from a species' base) of node k in the step of parity ODD.
template <bool ODD>
__device__ __forceinline__ void stream_slots(const SparseView& S, int64_t k, uint32_t mt, uint32_t (&off)[7]) {
    const uint32_t K32 = (uint32_t)S.KS;  // row stride; SS < 2^31 is checked when the layout is built
    const uint32_t wm = mt & 0x7Fu;
    if (!ODD) {
        const uint32_t lb = 7u * K32 + (uint32_t)(S.tlb[(int)(k >> 8)] + (int)(mt >> 14));
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            const int oi = q7opp(i);
            off[i] = (i != 0 && ((wm >> oi) & 1u)) ? lb + (uint32_t)__popc(wm & ((1u << oi) - 1u))
                                                   : (uint32_t)(i * K32) + (uint32_t)k;
        }
    } else {
        const uint32_t blk = wm | ((mt >> 7) & 0x7Fu);  // wall or outside the box
        const int2 dv = *reinterpret_cast<const int2*>(S.dres + 4 * k);
        const int4 tb = *reinterpret_cast<const int4*>(S.tdb + 4 * (int)(k >> 8));
        int nb[7];  // compact index of the source node a - c_i
        nb[0] = (int)k;
        nb[1] = (int)k + tb.x + (int16_t)(dv.x & 0xFFFF);
        nb[4] = (int)k + tb.y + (int16_t)((uint32_t)dv.x >> 16);
        nb[2] = (int)k + tb.z + (int16_t)(dv.y & 0xFFFF);
        nb[5] = (int)k + tb.w + (int16_t)((uint32_t)dv.y >> 16);
        nb[3] = (int)k + 1;
        nb[6] = (int)k - 1;
        off[0] = (uint32_t)k;
#pragma unroll
        for (int i = 1; i < 7; ++i) {
            const int oi = q7opp(i);
            off[i] = ((blk >> oi) & 1u) ? (uint32_t)(i * K32) + (uint32_t)k : (uint32_t)(oi * K32) + (uint32_t)nb[i];
        }
    }
}

// What the step knows of a node besides its slots.
template <typename TC>
struct StreamNode {
    int code, nd;  // nd (dense index) only where hb
    TC ux, uy, uz;
    bool hb;       // biomass may act (dual Monod)
};

template <typename TC, int LAW>
__device__ __forceinline__ StreamNode<TC> stream_node(const SparseView& S, const AdeStep<TC>& P, const TC* __restrict__ u,
                                                      int64_t k) {
    StreamNode<TC> A;
    A.code = S.code[k];
    A.hb = LAW >= STREAM_DUAL_AFTER && (!P.bflag || P.bflag[k]);
    A.ux = u[k];
    A.uy = u[S.K + k];
    A.uz = u[2 * S.K + k];
    A.nd = A.hb ? S.node[k] : 0;
    return A;
}

// All species of one node, from its slots; every thread of the block calls it, `on` those that have a
// node. U: species whose gathers are in flight together. smem: stream_bytes() per thread.
// face(s, west): the density a Neumann face of species s imposes on the node.
//
// LOCKSTEP: the barrier before each group keeps the block's warps on the same U species: a step reads
// and writes 7 rows per species, and warps that drift apart spread their requests over all 7 S rows.
template <typename TS, typename TC, int U, int LAW, int T, bool LOCKSTEP, typename Face>
__device__ __forceinline__ void ade_stream_species(TS* g, double* imm, double* bio, const SparseView& S, const AdeStep<TC>& P,
                                                   int64_t kw, int64_t ke, unsigned char* smem, int64_t k,
                                                   const StreamNode<TC>& A, const uint32_t (&off)[7], bool on, Face face_value) {
    double* bs = reinterpret_cast<double*>(smem) + threadIdx.x;  // "after": [STREAM_MICROBES], stride T
    TC* dc = reinterpret_cast<TC*>(smem + (LAW == STREAM_DUAL_AFTER ? STREAM_MICROBES * sizeof(double) * T : 0)) + threadIdx.x;
    const int nd = A.nd;
    const int dyn = P.dyn[A.code];
    on = on && dyn != ADE_BB;  // a voxel sealed by precipitation: the identity on AA slots
    const int nm = P.n_mobile;
    const TC* wk = P.w[dyn == ADE_BIO ? 1 : 0];
    const bool west = k < kw, face = west || k >= ke;
    const bool react = LAW != STREAM_NONE && on && !face && P.react[A.code];
    const bool hb = A.hb && react;
    if (LAW == STREAM_DUAL_AFTER && hb) {
#pragma unroll
        for (int m = 0; m < STREAM_MICROBES; ++m)
            if (m < P.M) cp_async<8>(bs + m * T, bio + (int64_t)m * P.N + nd);
    }
    TC chk = 0;  // a NaN or infinite density in any species makes the sum non-finite
    for (int s0 = 0; s0 < nm; s0 += U) {
        if (LOCKSTEP && s0 > 0) __syncthreads();
        if (!on) continue;
        TC q[U][7];
#pragma unroll
        for (int v = 0; v < U; ++v) {
            if (v > 0 && s0 + v >= nm) break;
            const TS* f = g + (int64_t)(s0 + v) * S.SS;
#pragma unroll
            for (int i = 0; i < 7; ++i) q[v][i] = gather<TS, TC>(f + off[i]);
        }
        if (LAW == STREAM_DUAL_AHEAD && s0 == 0 && hb) {
            // while the first group's gathers are on their way
            for (int m = 0; m < nm; ++m) dc[m * T] = 0;
            dual_monod<TC>(
                P, bio, nd, [](int, const double* p) { return *p; },
                [&](int s) {
                    if (s >= nm) return floored<TC>((TC)imm[(int64_t)s * P.N + nd]);
                    const TS* f = g + (int64_t)s * S.SS;
                    TC r = 0;
#pragma unroll
                    for (int i = 0; i < 7; ++i) r += ld<TS, TC>(f + off[i]);
                    return floored<TC>(r + (TC)ade_sigma<TC>());
                },
                [&](int s, TC d) {
                    if (s < nm) dc[s * T] = d;
                    else if (d != (TC)0) imm[(int64_t)s * P.N + nd] += (double)d;
                });
        }
#pragma unroll
        for (int v = 0; v < U; ++v) {
            const int s = s0 + v;
            if (v > 0 && s >= nm) break;
            if (face) {
                // AdvectionDiffusionBoundaryDynamics: the one inward population makes the node's
                // density the stored value; a closed face bounces back
                const int type = west ? P.ltype[s] : P.rtype[s];
                if (type == CLB_CLOSED) continue;
                double rs;
                if (type == CLB_DIRICHLET) rs = west ? P.lbc[s] : P.rbc[s];
                else rs = face_value(s, west);
                TC sum = 0;
#pragma unroll
                for (int i = 0; i < 7; ++i)
                    if (i != (west ? 4 : 1)) sum += q[v][i];
                const TC miss = (TC)(rs - ade_sigma<TC>()) - sum;
                if (west) q[v][4] = miss;
                else q[v][1] = miss;
            }
            TC r = 0;
#pragma unroll
            for (int i = 0; i < 7; ++i) r += q[v][i];
            chk += r;
            TC d = 0;
            if (LAW == STREAM_SEPARABLE && react) {
                const TC C = floored<TC>(r + (TC)ade_sigma<TC>());
                d = clamped_increment<TC>(separable_rate<TC>(P, s, C), P.dt, C);
            }
            if (LAW == STREAM_DUAL_AHEAD && hb) d = dc[s * T];
            if (LAW == STREAM_DUAL_AFTER && hb) {
                if (s == P.donor) dc[0] = r;
#pragma unroll
                for (int m = 0; m < STREAM_MICROBES; ++m)
                    if (m < P.M && s == P.acceptor[m]) dc[(1 + m) * T] = r;
            }
            ade_collide_store<TS, TC>(g + (int64_t)s * S.SS, off, q[v], r, wk[s], d, A.ux, A.uy, A.uz, P.S == 1);
        }
    }
    if (LAW == STREAM_DUAL_AHEAD && nm == 0 && hb) {
        // no species is mobile: there was no group to take the coupled laws with
        dual_monod<TC>(
            P, bio, nd, [](int, const double* p) { return *p; },
            [&](int s) { return floored<TC>((TC)imm[(int64_t)s * P.N + nd]); },
            [&](int s, TC d) {
                if (d != (TC)0) imm[(int64_t)s * P.N + nd] += (double)d;
            });
    }
    if (LAW == STREAM_DUAL_AFTER && hb) {
        cp_async_wait_all();  // each thread reads only its own slots
        dual_monod<TC>(
            P, bio, nd, [&](int m, const double*) { return bs[m * T]; },
            [&](int s) {
                TC r = dc[0];
#pragma unroll
                for (int m = 0; m < STREAM_MICROBES; ++m)
                    if (m < P.M && s == P.acceptor[m]) r = dc[(1 + m) * T];
                return floored<TC>(r + (TC)ade_sigma<TC>());
            },
            [&](int s, TC d) {
                if (d == (TC)0) return;
                TS* f = g + (int64_t)s * S.SS;
                TC x[7];
#pragma unroll
                for (int j = 0; j < 7; ++j) x[j] = ld<TS, TC>(f + off[j]);
#pragma unroll
                for (int j = 0; j < 7; ++j) st<TS, TC>(f + off[j], x[j] + (j == 0 ? (TC)0.25 : (TC)0.125) * d);
            });
    }
    if (LAW == STREAM_SEPARABLE && react)
        for (int s = nm; s < P.S; ++s) {
            double* c = imm + (int64_t)s * P.N + S.node[k];
            const TC C = floored<TC>((TC)*c);
            const TC d = clamped_increment<TC>(separable_rate<TC>(P, s, C), P.dt, C);
            if (d != (TC)0) *c += (double)d;
        }
    if (!isfinite(chk) && P.nonfinite) *(volatile int*)P.nonfinite = 1;
}

// One node per thread of one transport step; every thread of the block calls it.
template <typename TS, typename TC, bool ODD, int U, int LAW, int T>
__device__ __forceinline__ void ade_stream_node(TS* __restrict__ g, double* __restrict__ imm, double* __restrict__ bio,
                                                const TC* __restrict__ u, const SparseView& S,
                                                const double* neu, const AdeStep<TC>& P, int64_t kw, int64_t ke,
                                                unsigned char* smem, int64_t k, bool on) {
    StreamNode<TC> A = {};
    uint32_t off[7] = {0, 0, 0, 0, 0, 0, 0};
    if (on) {
        const uint32_t mt = S.meta[k];
        A = stream_node<TC, LAW>(S, P, u, k);
        stream_slots<ODD>(S, k, mt, off);
    }
    step_wait();
    ade_stream_species<TS, TC, U, LAW, T, true>(g, imm, bio, S, P, kw, ke, smem, k, A, off, on, [&](int s, bool west) {
        return neu[((int64_t)s * 2 + (west ? 0 : 1)) * P.plane + S.node[k] % P.plane];
    });
}

}  // namespace clb
