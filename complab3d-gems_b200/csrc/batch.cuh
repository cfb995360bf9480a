// batch.cuh -- many independent domains advanced by one launch per lattice and step.
#pragma once

#include "sparse.cuh"

namespace clb {

// Everything the batched kernels need of one domain (device copy, one per domain).
struct BatchDomain {
    // flow lattice
    void* f;
    void* flink;
    SparseView fs;
    int64_t fkw, fke;  // compact index ranges of the planes x = 0, x = nx-1
    FlowParams fp;
    // species lattices
    void* g;
    void* glink;
    SparseView as;
    int64_t akw, ake;
    AdeParams ap;
    double* imm;
    double* bio;
    const void* u;
    double* neu;
    const int* mob;
    const int8_t* mat;
    int n_mobile;
};

// one Neumann plane of one mobile species of one domain
struct NeumannJob {
    int d, s, m, side;
};

// A run of consecutive compact nodes of one domain's lattice: the unit the per-lattice batched
// launches hand to a CTA, which holds the domain's description in shared memory while it works.
struct BatchTile {
    int d;
    int count;
    int64_t first;
};
// Nodes per tile; a block takes its tile 128 nodes at a time. Small tiles end together where a launch has
// few of them; larger ones save the tile and domain reads, which a flow node of 38 values notices least.
// FP32 on one B200: transport 96 domains 153.5 us per step at 128 nodes, 156.6 at 512; 16 domains 23.4 and 27.1;
// flow 96 domains 134.8 at 256 nodes, 135.4 at 512.
constexpr int BATCH_FLOW_TILE = 256;
constexpr int BATCH_ADE_TILE = 128;
// 128 pixels of an x-face of one domain that at least one mobile species treats as Neumann
struct NeumannTile {
    int d, side, first;
};
constexpr int NEUMANN_TILE = 128;

struct BatchView {
    const BatchDomain* dom;
    int ndom;
    const NeumannJob* jobs;
    int njobs;
    const BatchTile* ftiles;  // flow tiles, domain by domain
    int nft;
    const BatchTile* atiles;  // transport tiles, by the streamed form of their domain's law, then domain by domain
    int alaw[5];              // the tiles of form q are atiles[alaw[q] .. alaw[q + 1])
    const void* sdom;         // StreamDomain of every domain
    int max_mobile;
    const NeumannTile* ntiles;
    int nnt;
};

constexpr int BATCH_MAX_DOMAINS = 2048;

// One entry of the persistent schedule: a tile of one lattice of one domain at one step of the
// launch (or the Neumann planes of the domain's species at that step).
constexpr int BI_FLOW = 0, BI_NEUMANN = 1, BI_TRANSPORT = 2;
struct BatchItem {
    int d;
    int16_t kind;   // BI_FLOW, BI_NEUMANN or BI_TRANSPORT
    int16_t step;   // step within the launch
    int64_t first;  // first compact node of the tile
    int count;      // nodes in the tile
    int pad;
};
constexpr int PERSIST_MAX_STEPS = 8;

struct PersistView {
    BatchView B;
    const BatchItem* items;
    int n_items;
    const int* need;  // [3][ndom]: items of each kind per domain and step
    const int* jbeg;  // [ndom + 1]: the Neumann jobs of domain d are jobs[jbeg[d] .. jbeg[d + 1])
    int* done;        // [steps][3][ndom]: items finished, zero when the launch starts
    int* ticket;      // next item to take, zero when the launch starts
    int* status;      // nonzero: a wait gave up (the launch's remaining items were skipped)
    int fodd, aodd;   // parities of the launch's first step
    int64_t wait_ns;  // limit of one wait
};

// flow.cu
void launch_flow_batch(const BatchView& B, int prec, bool odd, cudaStream_t st);
// ade_stream.cu: the transport step of every domain; the device copies its tiles refer to (form: the
// streamed form of each handle's law)
void launch_ade_batch(const BatchView& B, int prec, bool odd, cudaStream_t st);
cudaError_t stream_domains(clb_handle* const* hs, int n, int prec, void** dev, std::vector<int>& form);
void launch_neumann_batch(const BatchView& B, int prec, bool odd, cudaStream_t st);
// ade.cu
// the persistent schedule: one launch runs the whole item table (nm: species register bucket 1, 2, 4,
// 8 or 16)
void launch_batch_persistent(const PersistView& V, int prec, int nm, int minb, int blocks_per_sm, int num_sms,
                             cudaStream_t st);
int batch_persistent_resident(int prec, int nm, int minb);  // resident CTAs per SM of that launch
int persist_minb(int prec, int nm, int minb);                // the register budget built for that request

}  // namespace clb
