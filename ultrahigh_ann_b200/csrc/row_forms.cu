// The forms of an index's rows that the estimating scans read (split BF16 parts,
// 16-bit fixed point, row bitmaps) and those scans' workspace memory.
//
// A cudaMalloc past 2 MB takes about 0.35 ms whatever its size (and now and then
// many times that), as much as a batch: 256 queries on 65,536 x 128 take 0.17 ms.
// So a form of up to kReservedForm bytes has its place in the allocation of the
// index's rows, a larger one is one allocation, made once the batches asked so far
// would have saved its cost, and a call's scan buffers are parts of one: the
// workspace's query buffer where its largest batch needs up to kReservedScan, else
// one of their own. First batch of a new index and workspace, 65,536 x 128 (L1), 256
// queries: 0.81 ms by the binary32 scan (one allocation), 1.33 ms with five, 0.27 ms
// with none.
#include "engine_internal.h"

#include <algorithm>
#include <cmath>
#include <functional>
#include <set>

namespace uha_engine {

using uha::check_cuda;
using uha::checked_mul;
using uha::IndexKind;
using uha::round_up;

namespace {

// Forms of at most this many bytes have their place beside the rows.
constexpr uint64_t kReservedForm = 64ull << 20;
// Scan buffers of at most this many bytes have theirs behind the query buffer.
constexpr uint64_t kReservedScan = 128ull << 20;

// Consecutive parts of one allocation, each on a 256-byte boundary.
struct Parts {
    uint64_t bytes = 0;
    uint64_t take(uint64_t count, uint64_t size)
    {
        const uint64_t at = bytes;
        bytes = uha::checked_add(
            bytes, round_up(checked_mul(count, size, "scan buffer"), 256), "scan buffer");
        return at;
    }
};

struct SplitLayout {
    Parts parts;
    uint64_t data, largest, norms, roots, centre;
    SplitLayout(uint64_t rows, uint64_t pitch)
        : data(parts.take(checked_mul(uha::lowp_padded_count(rows), pitch, "split rows"), 4)),
          largest(parts.take(1, sizeof(uint32_t))),  // of the roots; cleared with the data's end
          norms(parts.take(rows, sizeof(float))),
          roots(parts.take(rows, sizeof(float))),
          centre(parts.take(pitch, sizeof(float)))
    {
    }
};

struct FixedLayout {
    Parts parts;
    uint64_t ranges, summary, offsets, data;
    FixedLayout(uint64_t rows, uint64_t dim, uint64_t pitch)
        : ranges(parts.take(2 * dim, sizeof(uint32_t))),  // cleared with the summary
          // the summary, and the rows' terms right behind it
          summary(parts.take(uha::checked_add(
                                 sizeof(uha::FixedSummary) / sizeof(uha::FixedTerms), rows,
                                 "fixed-point rows"),
                             sizeof(uha::FixedTerms))),
          offsets(parts.take(pitch, sizeof(float))),
          data(parts.take(checked_mul(rows, pitch, "fixed-point rows"), sizeof(uint16_t)))
    {
    }
};

struct BitsLayout {
    Parts parts;
    uint64_t boundaries, data;
    BitsLayout(uint64_t rows, uint64_t p)
        : boundaries(parts.take(uha::bits_boundaries(p), sizeof(float))),
          data(parts.take(uha::bits_bytes(rows, p), 1))
    {
    }
};

// Bytes of the form that this index's batches read, 0 when they read none.
uint64_t form_bytes(const uha_index* index)
{
    if (index->scan_dim == 0 || index->rows < 2) {
        return 0;
    }
    if (index->kind == IndexKind::hierarchical) {
        if (index->metric == UHA_L2) {
            return SplitLayout(index->rows, uha::split_pitch(index->scan_dim)).parts.bytes;
        }
        return uha::bits_applies(index->rows, index->projection_dimension)
                   ? BitsLayout(index->rows, index->projection_dimension).parts.bytes
                   : 0;
    }
    if (small_path_applies(index, UHA_DIRECT)) {
        return 0;
    }
    if (index->metric == UHA_L2) {
        return SplitLayout(index->rows, uha::split_pitch(index->scan_dim)).parts.bytes;
    }
    return index->rows <= uha::kFixedRows
               ? FixedLayout(index->rows, index->scan_dim, uha::fixed_pitch(index->scan_dim))
                     .parts.bytes
               : 0;
}

// Memory for a form: its place beside the rows, or `own`; null without room. One of
// its own takes at most half of the free memory, so another index of that size, or
// what else the program holds on the device, still finds room.
unsigned char* form_store(const uha_index* index, uint64_t bytes,
                          uha::DeviceBuffer<unsigned char>& own)
{
    if (bytes <= index->form_space_bytes) {
        return index->form_space;
    }
    size_t free_bytes = 0;
    size_t total = 0;
    check_cuda(cudaMemGetInfo(&free_bytes, &total), "cannot query CUDA memory");
    return bytes <= free_bytes / 2 && own.try_allocate(bytes) ? own.get() : nullptr;
}

// The indexes that hold a form of their own.
struct Holders {
    std::mutex mutex;
    std::set<const uha_index*> indexes;
};

Holders& holders()
{
    static Holders* all = new Holders;  // indexes may be destroyed at exit
    return *all;
}

// After a form of its own has been published (forms_mutex held).
void note_holder(const uha_index* index)
{
    Holders& all = holders();
    std::lock_guard<std::mutex> lock(all.mutex);
    all.indexes.insert(index);
}

// A form's build has ended, one way or the other, before its memory is given back
// or written again.
struct Drain {
    cudaStream_t stream;
    ~Drain() { cudaStreamSynchronize(stream); }
};

// About the time (us) of a batch of n by the binary32 scan and by the estimating one:
// a fixed part (launches, synchronisation, delivery) and the (query, row, column)
// rates of each on a B200, within a third of what was measured from 1,000 x 300 to
// 65,536 x 1,500 values and 9 to 4,096 queries. The binary32 tile takes 64 queries'
// time at least.
struct BatchTimes {
    double binary32;
    double estimates;
};

BatchTimes batch_times(const uha_index* index, uint64_t n)
{
    const double values = static_cast<double>(index->rows) * index->scan_dim;
    const double all = values * n;
    if (index->kind == IndexKind::hierarchical) {
        return index->metric == UHA_L2 ? BatchTimes{230 + all / 4.5e6, 75 + all / 80e6}
                                       : BatchTimes{290 + all / 3.2e6, 130 + all / 25e6};
    }
    const double binary32 = 60 + values * round_up(n, 64) / 12e6;
    return index->metric == UHA_L2
               ? BatchTimes{binary32, 45 + std::max(values * 4 / 5.5e6, 6 * all / 1.4e9)}
               : BatchTimes{binary32, 45 + values * round_up(n, 32) / 24e6};
}

// Whether a form that is not there yet is built for this call. One with a place
// beside the rows is at once (50 us); a larger one, whose allocation and two passes
// over the rows cost 0.45 ms and the bytes at about 5 TB/s, once the batches so far
// and the rest of this call would have saved that. Called with forms_mutex held.
bool form_due(const uha_index* index, const FormCall& call, uint64_t bytes)
{
    if (call.now || bytes <= index->form_space_bytes) {
        return true;
    }
    auto saved = [&](uint64_t queries) {
        const BatchTimes t = batch_times(index, queries);
        return std::max(0.0, t.binary32 - t.estimates);
    };
    const double rows = static_cast<double>(index->rows) * index->scan_dim * sizeof(float);
    const double cost = 450.0 + (2.0 * rows + bytes) / 5e6;
    if (index->form_saved + saved(call.upcoming) >= cost) {
        return true;
    }
    index->form_saved += saved(call.batch);
    *call.deferred = true;
    return false;
}

// The workspace's scan memory, of at least layout(n) bytes, and where there is room
// of layout() of the next power of two of queries, so that growing batches do not
// allocate each time. Null without room.
unsigned char* scan_store(uha_workspace* ws, uint64_t n,
                          const std::function<uint64_t(uint64_t)>& layout)
{
    const uint64_t need = layout(n);
    if (need <= ws->scan_space_bytes) {
        return ws->scan_space;
    }
    if (ws->scan_store.size() < need) {
        uint64_t wide = 1;
        while (wide < n) {
            wide *= 2;
        }
        const uint64_t more = layout(std::min(wide, ws->max_batch));
        // earlier work on the stream may still use the memory
        check_cuda(cudaStreamSynchronize(ws->stream), "CUDA query failed");
        if (!ws->scan_store.try_allocate(std::max(need, more)) &&
            !ws->scan_store.try_allocate(need)) {
            return nullptr;
        }
    }
    return ws->scan_store.get();
}

template <typename T>
T* part(unsigned char* base, uint64_t at)
{
    return reinterpret_cast<T*>(base + at);
}

// Takes a batch's buffers, count elements each, from the scan memory; without a
// base only their bytes are counted.
struct Carver {
    unsigned char* base;
    Parts parts;
    template <typename T>
    void operator()(T*& to, uint64_t count)
    {
        const uint64_t at = parts.take(count, sizeof(T));
        to = base != nullptr ? part<T>(base, at) : nullptr;
    }
};

// The buffers that layout(carver, queries) takes, for a batch of n; false without
// room.
template <typename F>
bool carve(uha_workspace* ws, uint64_t n, F&& layout)
{
    unsigned char* base = scan_store(ws, n, [&](uint64_t queries) {
        Carver c{nullptr, {}};
        layout(c, queries);
        return c.parts.bytes;
    });
    if (base != nullptr) {
        Carver c{base, {}};
        layout(c, n);
    }
    return base != nullptr;
}

}  // namespace

}  // namespace uha_engine

// A form goes only while no call uses it (its index's next batches build it again
// when they pay for it and there is room). An index's lock is only tried here: the
// builder of a form holds its own while it waits for the set's.
bool uha::reclaim_device_memory() noexcept
{
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) {
        return false;
    }
    uha_engine::Holders& all = uha_engine::holders();
    std::lock_guard<std::mutex> lock(all.mutex);
    bool any = false;
    for (auto it = all.indexes.begin(); it != all.indexes.end();) {
        const uha_index* index = *it;
        std::unique_lock<std::mutex> forms(index->forms_mutex, std::try_to_lock);
        if (index->device != device || !forms.owns_lock() || index->form_users->load() != 0) {
            ++it;
            continue;
        }
        index->split = SplitRows{};
        index->bits = RowBits{};
        index->fixed = FixedRows{};
        index->form_saved = 0.0;
        it = all.indexes.erase(it);
        any = true;
    }
    return any;
}

uha_index::~uha_index()
{
    uha_engine::Holders& all = uha_engine::holders();
    std::lock_guard<std::mutex> lock(all.mutex);
    all.indexes.erase(this);
}

namespace uha_engine {

void drop_form(const uha_index* index)
{
    std::lock_guard<std::mutex> lock(index->forms_mutex);
    const uint64_t own =
        index->split.own.size() + index->bits.own.size() + index->fixed.own.size();
    if (own != 0 && index->form_users->load() <= 1) {
        index->split = uha::SplitRows{};
        index->bits = uha::RowBits{};
        index->fixed = uha::FixedRows{};
        index->form_saved = 0.0;
    }
}

bool estimates_pay(const uha_index* index, uint64_t n, uint64_t open)
{
    const BatchTimes all = batch_times(index, n);
    return all.estimates + batch_times(index, open).binary32 <= all.binary32;
}

void allocate_scan_rows(uha_index* index)
{
    // the rows end on a 256-byte boundary, where the form's place begins
    const uint64_t values = round_up(
        checked_mul(index->rows, index->padded_dim, "padded representative matrix"), 64);
    const uint64_t form = form_bytes(index);
    if (form != 0 && form <= kReservedForm &&
        index->scan_rows.try_allocate(values + form / sizeof(float))) {
        index->form_space = reinterpret_cast<unsigned char*>(index->scan_rows.get() + values);
        index->form_space_bytes = form;
        return;
    }
    index->scan_rows.allocate(values);
}

const uha::SplitRows* split_rows(const uha_index* index, const FormCall& call,
                                 cudaStream_t stream)
{
    std::lock_guard<std::mutex> lock(index->forms_mutex);
    if (!index->split.ready) {
        const uint64_t pitch = uha::split_pitch(index->scan_dim);
        const SplitLayout at(index->rows, pitch);
        if (!form_due(index, call, at.parts.bytes)) {
            return nullptr;
        }
        uha::SplitRows sp;  // published only once it is built
        Drain drain{stream};
        sp.ready = true;
        sp.pitch = pitch;
        unsigned char* base = form_store(index, at.parts.bytes, sp.own);
        if (base != nullptr) {
            sp.data = base + at.data;
            sp.norms = part<float>(base, at.norms);
            sp.roots = part<float>(base, at.roots);
            sp.centre = part<float>(base, at.centre);
            unsigned int* largest = part<unsigned int>(base, at.largest);
            const uint64_t used = index->rows * pitch * 4;
            auto split = [&] {
                // the split writes every row's whole pitch; the vectors past the rows
                // are zero
                check_cuda(cudaMemsetAsync(sp.data + used, 0, at.norms - used, stream),
                           "cannot clear split rows");
                if (index->kind == IndexKind::hierarchical) {
                    uha::launch_split_rows(index->rows64.get(), index->rows, index->scan_dim,
                                           index->scan_dim, sp.data, pitch, sp.scale, sp.centre,
                                           sp.norms, sp.roots, largest, stream);
                } else {
                    uha::launch_split_rows(index->scan_rows.get(), index->rows,
                                           index->padded_dim, index->scan_dim, sp.data, pitch,
                                           sp.scale, sp.centre, sp.norms, sp.roots, largest,
                                           stream);
                }
                float root = 0.f;
                check_cuda(cudaMemcpyAsync(&root, largest, sizeof(root), cudaMemcpyDeviceToHost,
                                           stream),
                           "cannot copy the largest norm from the CUDA device");
                check_cuda(cudaStreamSynchronize(stream), "cannot build split rows");
                return root;
            };
            float root = split();
            if (std::isfinite(root) && root > 0.f && (root < 0x1p-8f || root > 0x1p24f)) {
                sp.scale = std::ldexp(1.f, -std::clamp(std::ilogb(root), -126, 126));
                root = split();
            }
            sp.usable = root <= uha::split_largest_norm();
            if (!sp.usable) {
                sp.own.release();
            }
        }
        index->split = std::move(sp);
        if (index->split.own.size() != 0) {
            note_holder(index);
        }
    }
    return index->split.usable ? &index->split : nullptr;
}

const uha::RowBits* row_bits(const uha_index* index, const FormCall& call, cudaStream_t stream)
{
    std::lock_guard<std::mutex> lock(index->forms_mutex);
    if (!index->bits.ready) {
        const uint64_t p = index->projection_dimension;
        const BitsLayout at(index->rows, p);
        if (!form_due(index, call, at.parts.bytes)) {
            return nullptr;
        }
        uha::RowBits rb;  // published only once they are built
        Drain drain{stream};
        rb.ready = true;
        unsigned char* base = form_store(index, at.parts.bytes, rb.own);
        if (base != nullptr) {
            rb.boundaries = part<float>(base, at.boundaries);
            rb.data = base + at.data;
            uha::launch_row_bits(index->scan_rows.get(), index->rows, index->padded_dim, p,
                                 rb.boundaries, rb.data, stream);
            check_cuda(cudaStreamSynchronize(stream), "cannot build row bitmaps");
            rb.usable = true;
        }
        index->bits = std::move(rb);
        if (index->bits.own.size() != 0) {
            note_holder(index);
        }
    }
    return index->bits.usable ? &index->bits : nullptr;
}

const uha::FixedRows* fixed_rows(const uha_index* index, const FormCall& call,
                                 cudaStream_t stream)
{
    std::lock_guard<std::mutex> lock(index->forms_mutex);
    if (!index->fixed.ready) {
        const uint64_t pitch = uha::fixed_pitch(index->scan_dim);
        const FixedLayout at(index->rows, index->scan_dim, pitch);
        if (!form_due(index, call, at.parts.bytes)) {
            return nullptr;
        }
        uha::FixedRows fx;  // published only once it is built
        Drain drain{stream};
        fx.ready = true;
        fx.pitch = pitch;
        unsigned char* base = form_store(index, at.parts.bytes, fx.own);
        if (base != nullptr) {
            uha::FixedSummary* summary = part<uha::FixedSummary>(base, at.summary);
            uha::FixedTerms* terms = reinterpret_cast<uha::FixedTerms*>(summary + 1);
            float* offsets = part<float>(base, at.offsets);
            uint16_t* data = part<uint16_t>(base, at.data);
            fx.terms = terms;
            fx.offsets = offsets;
            fx.step = &summary->step;
            fx.data = data;
            check_cuda(cudaMemsetAsync(base + at.ranges, 0,
                                       at.summary + sizeof(uha::FixedSummary) - at.ranges,
                                       stream),
                       "cannot clear column ranges");
            uha::launch_fixed_rows(index->scan_rows.get(), index->rows, index->padded_dim,
                                   index->scan_dim, index->weights64.get(), data, pitch, offsets,
                                   summary, terms, part<unsigned int>(base, at.ranges), stream);
            fx.usable = uha::fixed_usable(summary, index->rows, stream);
            if (!fx.usable) {
                fx.own.release();
            }
        }
        index->fixed = std::move(fx);
        if (index->fixed.own.size() != 0) {
            note_holder(index);
        }
    }
    return index->fixed.usable ? &index->fixed : nullptr;
}

namespace {

// What each scan takes for a batch of q. Query vectors of the split scan come in
// whole tiles: the ones past the batch are read, whatever they hold, and nothing of
// them is stored.
void take_split(Carver& take, const uha_index* index, uint64_t pitch, uint64_t q,
                const uha::SplitPlan& plan, SplitBuffers* b)
{
    const bool filter = uha::split_filter_applies(plan, index->rows);
    const bool hierarchical = index->kind == IndexKind::hierarchical;
    take(b->queries,
         checked_mul(round_up(q, static_cast<uint64_t>(plan.bn)), 4 * pitch, "queries"));
    take(b->squares, q * uha::kSplitSlices);
    take(b->counts, q);
    take(b->upper, q);
    take(b->done, q);
    take(b->candidates, q * uha::kSplitCandidates);
    take(b->keys, filter ? q * uha::kSplitListKeys : 0);
    take(b->partials,
         filter ? 0
                : checked_mul(checked_mul(plan.splits, q, "partials"), index->rows, "partials"));
    take(b->sums, hierarchical ? 0 : uha::settle_sums(q, index->padded_dim));
    take(b->projected, hierarchical ? q * index->projection_dimension : 0);
}

void take_fixed(Carver& take, const uha_index* index, uint64_t pitch, uint64_t q,
                const uha::FixedPlan& plan, FixedBuffers* b)
{
    take(b->parts, q * uha::kSplitSlices);
    take(b->counts, q);
    take(b->upper, q);
    take(b->done, q);
    take(b->candidates, q * uha::kSplitCandidates);
    take(b->least, checked_mul(q, uha::fixed_tiles(index->rows), "partials"));
    take(b->queries, checked_mul(q, pitch, "queries"));
    take(b->sums, checked_mul(checked_mul(plan.splits, q, "partials"), index->rows, "partials"));
    take(b->settled, uha::settle_sums(q, index->padded_dim));
}

void take_bits(Carver& take, const uha_index* index, uint64_t q, BitsBuffers* b)
{
    const uint64_t p = index->projection_dimension;
    const uint64_t list = checked_mul(q, uha::bits_list(index->rows), "row lists");
    take(b->min_bits, q);
    take(b->counts, q);
    take(b->offsets, uha::bits_offsets(q, p));
    take(b->listed, list);
    take(b->medians, list);
    take(b->projected, q * p);
}

// Bytes of the scan buffers of batches of n, 0 when they need none.
uint64_t scan_bytes(const uha_index* index, uint64_t n)
{
    Carver take{nullptr, {}};
    if (form_bytes(index) == 0 || n > 65535) {
        return 0;
    }
    if (index->kind == IndexKind::hierarchical && index->metric == UHA_L1) {
        BitsBuffers b{};
        take_bits(take, index, n, &b);
    } else if (n <= 8) {
        return 0;
    } else if (index->metric == UHA_L2) {
        SplitBuffers b{};
        const uint64_t pitch = uha::split_pitch(index->scan_dim);
        take_split(take, index, pitch, n,
                   uha::plan_split(index->rows, pitch, n, index->sm_count), &b);
    } else {
        FixedBuffers b{};
        const uint64_t pitch = uha::fixed_pitch(index->scan_dim);
        take_fixed(take, index, pitch, n,
                   uha::plan_fixed(index->rows, pitch, n, index->sm_count), &b);
    }
    return take.parts.bytes;
}

}  // namespace

void allocate_raw_queries(uha_workspace* ws, const uha_index* index, bool scans)
{
    const uint64_t values =
        round_up(checked_mul(ws->max_batch, index->dimension, "query workspace"), 64);
    const uint64_t scan = scans ? scan_bytes(index, ws->max_batch) : 0;
    if (scan != 0 && scan <= kReservedScan &&
        ws->raw_queries.try_allocate(values + scan / sizeof(float))) {
        ws->scan_space = reinterpret_cast<unsigned char*>(ws->raw_queries.get() + values);
        ws->scan_space_bytes = scan;
        return;
    }
    ws->raw_queries.allocate(ws->max_batch * index->dimension);
}

bool split_buffers(uha_workspace* ws, const uha_index* index, uint64_t pitch, uint64_t n,
                   const uha::SplitPlan& plan, SplitBuffers* out)
{
    return carve(ws, n, [&](Carver& take, uint64_t q) {
        take_split(take, index, pitch, q, plan, out);
    });
}

bool fixed_buffers(uha_workspace* ws, const uha_index* index, uint64_t pitch, uint64_t n,
                   const uha::FixedPlan& plan, FixedBuffers* out)
{
    return carve(ws, n, [&](Carver& take, uint64_t q) {
        take_fixed(take, index, pitch, q, plan, out);
    });
}

bool bits_buffers(uha_workspace* ws, const uha_index* index, uint64_t n, BitsBuffers* out)
{
    return carve(ws, n,
                 [&](Carver& take, uint64_t q) { take_bits(take, index, q, out); });
}

}  // namespace uha_engine
