// Query pipeline pieces shared by the engine's host translation units
// (engine.cu: single calls; batch.cu: captured multi-index batches, the
// autotuner and the request loop).
#pragma once

#include "common.h"
#include "index_types.h"
#include "kernels.h"
#include "stage_bodies.h"

namespace uha_engine {

bool precision_strategy(uha_strategy s);
bool fp32_rescore_strategy(uha_strategy s);
bool small_path_applies(const uha_index* index, uha_strategy strategy);
uha::LowpType lowp_type(uha_strategy s);

// The index's low-precision rows of `type` (built on first use) and the
// workspace buffers of the precision strategies.
const uha::LowpRows& lowp_rows(const uha_index* index, uha::LowpType type,
                               cudaStream_t stream);
void ensure_lowp_workspace(uha_workspace* ws, const uha_index* index,
                           cudaStream_t stream);

// Batches of n queries that the certified split scan (split_scan.cu) can serve.
bool split_shape(const uha_index* index, uha_strategy strategy, uint64_t n);

// row_forms.cu: the rows' allocation (rows x padded_dim, with a small form's place),
// and the forms, built on `stream` and synchronised before they are published; null
// while the index keeps the binary32 scan (no room, out of the form's range, or not
// worth its build yet).
struct FormCall {
    uint64_t batch;     // queries of this batch
    uint64_t upcoming;  // of this and the call's later batches
    bool now;           // built whatever it would save (captured and tuned batches)
    bool* deferred;     // set when the form is not built yet
};
// While one of these lives, the index's forms are not given back.
class FormUse {
public:
    explicit FormUse(const uha_index* index) : users_(index->form_users) { ++*users_; }
    FormUse(FormUse&& other) noexcept = default;
    FormUse& operator=(FormUse&& other) = delete;
    ~FormUse()
    {
        if (users_ != nullptr) {
            --*users_;
        }
    }

private:
    std::shared_ptr<std::atomic<int>> users_;
};
void allocate_scan_rows(uha_index* index);
// Gives the index's own form back when only the calling thread uses it and has
// nothing in flight that reads it (it is built again when it pays): a call that finds
// no room for its scan buffers needs the memory for the binary32 scan's.
void drop_form(const uha_index* index);
const uha::SplitRows* split_rows(const uha_index* index, const FormCall& call,
                                 cudaStream_t stream);
const uha::FixedRows* fixed_rows(const uha_index* index, const FormCall& call,
                                 cudaStream_t stream);
const uha::RowBits* row_bits(const uha_index* index, const FormCall& call, cudaStream_t stream);

// The workspace's query buffer (max_batch x dimension), with the place of the scan
// buffers of a largest batch where they are small and `scans` asks for it.
void allocate_raw_queries(uha_workspace* ws, const uha_index* index, bool scans);
// uha_workspace_create; without `scans` for a caller that never estimates.
uha_status create_workspace(const uha_index* index, uint64_t maximum_batch_size, bool scans,
                            uha_workspace** out);

// Whether estimates that leave `open` of n queries to the binary32 scan take less
// time than the binary32 scan of them all.
bool estimates_pay(const uha_index* index, uint64_t n, uint64_t open);

// The estimating scans' buffers of a batch of n, from the workspace's scan memory
// (false when the device has no room). Only one scan's are in use at a time.
struct SplitBuffers {
    unsigned char* queries;
    double* squares;
    uint32_t* counts;
    unsigned int* upper;
    uint32_t* done;
    uint32_t* candidates;
    unsigned long long* keys;  // filter form
    float* partials;           // else
    double* sums;              // exact and flat: the settlement's
    double* projected;         // hierarchies
};
struct FixedBuffers {
    uha::FixedParts* parts;
    uint32_t* counts;
    unsigned long long* upper;
    uint32_t* done;
    uint32_t* candidates;
    unsigned long long* least;
    uint16_t* queries;
    uint32_t* sums;
    double* settled;  // the settlement's sums
};
struct BitsBuffers {
    unsigned int* min_bits;
    uint32_t* counts;
    uint32_t* offsets;
    uint32_t* listed;
    float2* medians;
    double* projected;
};
bool split_buffers(uha_workspace* ws, const uha_index* index, uint64_t pitch, uint64_t n,
                   const uha::SplitPlan& plan, SplitBuffers* out);
bool fixed_buffers(uha_workspace* ws, const uha_index* index, uint64_t pitch, uint64_t n,
                   const uha::FixedPlan& plan, FixedBuffers* out);
bool bits_buffers(uha_workspace* ws, const uha_index* index, uint64_t n, BitsBuffers* out);

struct BatchContext {
    const uha_index* index;
    uha_workspace* ws;
    uha_strategy strategy;
    bool want_distances;
    // Pipelined calls (exact and flat indexes): this batch's prepared queries
    // and partial sums (direct / gemm) or candidate buffers (precision),
    // sized by the caller, and the stream its argmin / re-score runs on after
    // `handoff` is recorded behind the scan. Null: the workspace's own buffers
    // and stream.
    float* prepared = nullptr;
    float* partials = nullptr;
    uint32_t* candidates = nullptr;   // precision: this batch's candidate slot
    double* cand_dist = nullptr;
    uint32_t* rescore_done = nullptr;
    cudaStream_t finish_stream = nullptr;
    cudaEvent_t handoff = nullptr;
    // The precision strategies may take the fused candidate selection: the caller
    // answers the call again without it (ws->filter_disabled) when a candidate
    // list overflows (error bit uha::kCandidateOverflow).
    bool filter_candidates = false;
    // The direct strategy may take the estimating scans: the caller answers the
    // queries that they leave open (uha::kOpenQuery) by the binary32 scan.
    bool estimates = false;
    uint64_t upcoming = 0;    // queries of the call from this batch on
    bool build_forms = false;  // a row form is built whatever this call would save
    // Every reported distance in binary64, as the estimating scans that this batch's
    // binary32 scan stands in for report it.
    bool refine_every = false;
    // The batch's queries hold the sampled values alone (gathered on the host).
    bool gathered = false;
    // The fused flat query of this batch runs on stream lane `flat_lane`
    // (0: ws->stream; others: ws->flat_streams, forked and joined by the
    // caller) with that lane's scratch slots.
    int flat_lane = 0;
    bool flat_shared = false;  // other lanes' launches run beside it
};

// Allocates and clears (on ws->stream) the fused flat query's scratch of
// every stream lane, if it does not exist yet.
void ensure_flat_scratch(const uha_index* index, uha_workspace* ws);

// Enqueues one batch of n queries (`source`: device, n x dimension floats) on
// ws->stream; returns the number of kernel launches. Buffers grow (with a
// stream synchronisation) only when n needs more than an earlier call did.
uint64_t enqueue_batch(const BatchContext& c, const float* source, uint64_t n,
                       uha::Result* results, double* exact, bool time_scan,
                       cudaEvent_t scan_start, cudaEvent_t scan_stop);

// The persistent batch's description of one pair (a hierarchical index and n
// queries in ws->raw_queries, certified direct strategy), read from the
// index and from workspace buffers that a standalone run of n queries has
// sized; false when the pair has no persistent form (projection dimension
// above 256, the streaming scan of batches up to 8, oversized shared memory).
// Median bound of the L1 hierarchy: the binary32 |diff| and midpoint
// roundings (the binary64 ones are within them): 6 * 2^-24 relative, 2^-126
// absolute.
constexpr float kMedianRel = 0x1.8p-22f;
constexpr float kMedianAbs = 0x1p-126f;

// The median passes' shape for batches of n on this workspace: the tuned
// one, else the default.
uha::MedianPlan median_plan(const uha_index* index, const uha_workspace* ws, uint64_t n);
bool persistent_pair(const uha_index* index, uha_workspace* ws, uint64_t n,
                     uha::PersistentPair* d);

// Answers of a call whose queries need no device work (row 0, distance 0).
void fill_trivial(uint64_t n, uint64_t* out_indices, double* out_distances);

// Reads the status words copied to ws->host_counters and converts the host
// copies of results / exact distances into the caller's arrays.
void finish_call(const uha_index* index, uha_workspace* ws, uint64_t n,
                 const uha::Result* results, const double* exact,
                 uint64_t* out_indices, double* out_distances);

// Open queries answered at a time: enough for the binary32 scan to fill the chip, and
// its sums (of each query and row) stay small beside the estimates' that are held.
constexpr uint64_t kOpenBatch = 1024;

// A call's status and message say that an allocation found no room.
bool no_device_memory(uha_status status);

// The queries of a call that the estimating scans left open.
std::vector<uint64_t> open_queries(const uha::Result* results, uint64_t n);
// Answers them by the binary32 scans into results and exact, in batches of at most
// `batch` (and kOpenBatch) on ws (whose query buffer, status words and last stats it overwrites);
// queries: host or device, n x dimension. Returns the stats of these calls, added
// up.
uha_query_stats answer_open(const uha_index* index, uha_workspace* ws, const float* queries,
                            const std::vector<uint64_t>& open, uint64_t batch,
                            uha_strategy strategy, bool want_distances, uha::Result* results,
                            double* exact);

void validate_query_call(const uha_index* index, uha_workspace* ws,
                         const float* queries, uint64_t count, uint64_t batch,
                         uha_strategy strategy, const uint64_t* out_indices);

}  // namespace uha_engine
