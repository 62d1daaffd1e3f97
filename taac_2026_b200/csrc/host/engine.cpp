// The packed forward of the engine (OneTransInference) as a native executor: one call prepares a batch (duplicate removal,
// statistics, row plan), one runs the tokenizers and the blocks, one the remaining blocks once no sample has a sequence
// token left, one the classifier.  A forward is about ninety launches of a few microseconds each; enqueued from Python
// they took 4 ms, more than the GPU needs for anything below a few thousand samples.
//
// The algorithm and its row layout are described at OneTransInference in onetrans.py; the comments here name the steps.
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/core/CachingHostAllocator.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <torch/csrc/autograd/python_variable.h>
#include <pybind11/stl.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "engine_ops.h"
#include "module.h"

namespace tb200_host {
namespace {

template <typename V>
V field(const py::dict& d, const char* name) { return d[name].cast<V>(); }
OptTensor optional_field(const py::dict& d, const char* name) {
    if (!d.contains(name) || d[name].is_none()) return std::nullopt;
    return d[name].cast<Tensor>();
}

// Kernels get the tensors of a record as raw pointers and row counts.  Before the first launch each one that is read has to be on the
// engine's device with the rows and columns that are read (size -1: any, columns: at least).
void require(const OptTensor& t, const char* name, const at::Device& device, at::IntArrayRef sizes) {
    TORCH_CHECK(t.has_value() && t->defined(), "OneTransInference: ", name, " is missing");
    TORCH_CHECK(t->device() == device, "OneTransInference requires all tensors of a record to live on ", device, ": ", name, " is on ", t->device());
    bool fits = t->dim() == static_cast<int64_t>(sizes.size());
    for (size_t i = 0; fits && i < sizes.size(); ++i) fits = sizes[i] < 0 || t->size(static_cast<int64_t>(i)) == sizes[i];
    TORCH_CHECK(fits, "OneTransInference: ", name, " has shape ", t->sizes(), ", expected ", sizes, " (-1: any)");
}
void require_columns(const Tensor& t, const char* name, int64_t columns) {
    TORCH_CHECK(t.size(1) >= columns, "OneTransInference: ", name, " has ", t.size(1), " columns, ", columns, " are read");
}
void check_sequence(const at::Device& device, int64_t batch, int64_t features, int64_t length, const Tensor& values, const OptTensor& lengths,
                    const OptTensor& stamps, const Tensor& request) {
    require(values, "values", device, {batch, features, length});
    if (lengths.has_value()) require(lengths, "lengths", device, {batch});
    if (stamps.has_value()) require(stamps, "timestamps", device, {batch, length});
    require(request, "request_timestamp", device, {batch});
}
// `fields` > 0: the missing flags of that many fields are read; `dense` > 0: so many dense values
void check_entity(const at::Device& device, int64_t batch, const Tensor& ids, int64_t id_columns, const OptTensor& missing, int64_t fields,
                  const OptTensor& values, const OptTensor& values_missing, int64_t dense) {
    require(ids, "int_values", device, {batch, -1});
    require_columns(ids, "int_values", id_columns);
    if (fields > 0) {
        require(missing, "int_missing_mask", device, {batch, -1});
        require_columns(*missing, "int_missing_mask", fields);
    }
    if (dense > 0) {
        require(values, "dense_values", device, {batch, dense});
        if (values_missing.has_value()) {
            require(values_missing, "dense_missing_mask", device, {batch, -1});
            require_columns(*values_missing, "dense_missing_mask", dense);
        }
    }
}

// Tensors made from weights on one stream (three-part splits, casts).  They hold for as long as their sources keep their content,
// which the sources' version counters tell, and a call on another stream is ordered behind their kernels by an event and noted
// with the allocator, so that they outlive it.
class Derived {
public:
    // the form of a weight that this library's GEMM reads
    Tensor own(const Tensor& w) { return made_from(w, own_form(w)); }
    Tensor cast(const Tensor& b, at::ScalarType type) { return made_from(b, b.to(type)); }
    void watch(const Tensor& source) {
        sources_.push_back({source, version(source), source.defined() ? source.data_ptr() : nullptr});
    }
    void keep(const Tensor& t) { made_.push_back(t); }
    // everything was enqueued on the current stream
    void seal(const at::Device& device) {
        stream_ = c10::cuda::getCurrentCUDAStream(device.index()).unwrap();
        ready_.record(c10::cuda::CUDAStream(*stream_));
    }
    bool unchanged() const {
        return std::all_of(sources_.begin(), sources_.end(), [](const Source& s) { return version(s.t) == s.version && s.t.data_ptr() == s.data; });
    }
    // before the current stream reads them
    void use(const at::Device& device) {
        const auto current = c10::cuda::getCurrentCUDAStream(device.index());
        if (current.unwrap() == *stream_ || std::find(users_.begin(), users_.end(), current.unwrap()) != users_.end()) return;
        ready_.block(current);
        for (const Tensor& t : made_) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), current);
        users_.push_back(current.unwrap());
    }

private:
    struct Source {
        Tensor t;
        int64_t version;
        const void* data;
    };
    static int64_t version(const Tensor& t) { return t.defined() && !t.is_inference() ? static_cast<int64_t>(t._version()) : 0; }
    Tensor made_from(const Tensor& source, Tensor t) {
        if (t.defined() && !t.is_same(source)) {
            watch(source);
            keep(t);
        }
        return t;
    }
    std::vector<Source> sources_;
    std::vector<Tensor> made_;
    std::vector<c10::Stream> users_;
    std::optional<c10::Stream> stream_;
    at::cuda::CUDAEvent ready_;
};

// The entries of a dict at one time.  It holds the objects, so that an equal address is the same object.
class Entries {
public:
    explicit Entries(const py::dict& d) : dict_(d) {
        for (const auto& item : d) values_.push_back(py::reinterpret_borrow<py::object>(item.second));
    }
    bool same() const {
        Py_ssize_t at = 0;
        PyObject *key, *value;
        size_t i = 0;
        while (PyDict_Next(dict_.ptr(), &at, &key, &value))
            if (i == values_.size() || values_[i++].ptr() != value) return false;
        return i == values_.size();
    }
    bool of(const py::handle& d) const { return dict_.ptr() == d.ptr(); }

private:
    py::dict dict_;
    std::vector<py::object> values_;
};

Layer layer_field(const py::dict& d, const std::string& w, const std::string& b32, Derived& derived) {
    Layer l;
    l.w = d[w.c_str()].cast<Tensor>();
    l.b32 = optional_field(d, b32.c_str());
    if (own_gemm_serves(l.w.scalar_type(), l.w.size(0), l.w.size(1))) l.own = derived.own(l.w);
    else if (l.b32.has_value()) l.b = derived.cast(*l.b32, l.w.scalar_type());
    return l;
}

// LayerNorm(SiLU(W [values, mask] + b)) of a small fp32 input, all fp32
struct SmallToken {
    Tensor w, b, gamma, beta;
    int64_t inputs;    // values of a row; the weight has as many columns again for their missing flags where there are such
    explicit SmallToken(const py::dict& d)
        : w(field<Tensor>(d, "w")), b(field<Tensor>(d, "b")), gamma(field<Tensor>(d, "gamma")), beta(field<Tensor>(d, "beta")),
          inputs(field<int64_t>(d, "inputs")) {}
    // writes [rows, d] at `out` (out_stride elements between rows)
    void run(const Tensor& values, const OptTensor& mask, void* out, int64_t out_stride, at::ScalarType type) const {
        const int64_t n = values.size(1), in_dim = w.size(0);
        check(tb200_small_token_fwd(data<float>(values), static_cast<int32_t>(n), values.stride(0),
                                    mask.has_value() ? static_cast<const uint8_t*>(mask->data_ptr()) : nullptr,
                                    mask.has_value() ? mask->stride(0) : 0, static_cast<int32_t>(in_dim), data<float>(w), data<float>(b),
                                    data<float>(gamma), data<float>(beta), out, out_stride, values.size(0), static_cast<int32_t>(w.size(1)), 1e-5f,
                                    dtype_code(type), stream_of(values)), "cuda small_token");
    }
};

// Fields of one entity -> n_tokens tokens: bag means of all fields, one projection, LayerNorm(SiLU)
struct EntityTokens {
    Tensor ptrs, rows, offsets, lengths;
    OptTensor missing_rows;
    Layer project;
    Tensor gamma, beta;
    int64_t n_fields, max_bag, dim, n_tokens, id_columns;
    EntityTokens(const py::dict& d, Derived& derived)
        : ptrs(field<Tensor>(d, "ptrs")), rows(field<Tensor>(d, "rows")), offsets(field<Tensor>(d, "offsets")), lengths(field<Tensor>(d, "lengths")),
          missing_rows(optional_field(d, "missing_rows")), project(layer_field(d, "w", "b32", derived)), gamma(field<Tensor>(d, "gamma")),
          beta(field<Tensor>(d, "beta")), n_fields(field<int64_t>(d, "n_fields")), max_bag(field<int64_t>(d, "max_bag")),
          dim(field<int64_t>(d, "dim")), n_tokens(field<int64_t>(d, "n_tokens")),
          id_columns(field<int64_t>(d, "id_columns")) {}
};

struct Block {
    Tensor attn_norm, ffn_norm, out_b;
    Layer qkv, q, kv, out, out_nobias, ffn1, ffn2;
    bool grouped_layers = false;          // the per-token layers run on this library's grouped GEMM
    Tensor ns_qkv_w, ns_qkv_b, ns_q_w, ns_q_b, ns_kv_w, ns_kv_b, ns_w1, ns_b1, ns_w2, ns_b2, ns_b2_folded, out_w_t;   // library form
    Tensor g_qkv_w, g_qkv_b, g_w1, g_b1, g_w2, g_b2, g_b2_folded, g_out_w;              // grouped form
    // e4m3 FFN: weights with their scales (fp32 blocks, or atoms of power-of-two scales)
    Tensor f_up, f_up_s, f_down, f_down_s, f_up_bf16;
    OptTensor f_b_up, f_b_down, f_b_down_folded;

    Block(const py::dict& d, Derived& derived) {
        attn_norm = field<Tensor>(d, "attn_norm");
        ffn_norm = field<Tensor>(d, "ffn_norm");
        out_b = field<Tensor>(d, "out_b");
        qkv = layer_field(d, "qkv_w", "qkv_b", derived);
        q = layer_field(d, "q_w", "q_b", derived);
        kv = layer_field(d, "kv_w", "kv_b", derived);
        out = layer_field(d, "out_w", "out_b32", derived);
        out_nobias.w = out.w;
        out_nobias.own = out.own;
        grouped_layers = d.contains("g_w1");
        auto take = [&](const char* name, Tensor& t) {
            if (d.contains(name)) t = d[name].cast<Tensor>();
        };
        take("ns_qkv_w", ns_qkv_w); take("ns_qkv_b", ns_qkv_b); take("ns_q_w", ns_q_w); take("ns_q_b", ns_q_b);
        take("ns_kv_w", ns_kv_w); take("ns_kv_b", ns_kv_b); take("ns_w1", ns_w1); take("ns_b1", ns_b1);
        take("ns_w2", ns_w2); take("ns_b2", ns_b2); take("ns_b2_folded", ns_b2_folded); take("out_w_t", out_w_t);
        take("g_qkv_w", g_qkv_w); take("g_qkv_b", g_qkv_b); 
        take("g_w1", g_w1); take("g_b1", g_b1);
        take("g_w2", g_w2); take("g_b2", g_b2); take("g_b2_folded", g_b2_folded); take("g_out_w", g_out_w);
        for (Tensor* w : {&g_qkv_w, &g_w1, &g_w2, &g_out_w}) *w = derived.own(*w);
        if (d.contains("ffn_fp8")) {
            const py::object w = d["ffn_fp8"];
            const bool mx = py::hasattr(w, "a_up");
            f_up = w.attr("w_up").cast<Tensor>();
            f_up_s = w.attr(mx ? "a_up" : "s_up").cast<Tensor>();
            f_down = w.attr("w_down").cast<Tensor>();
            f_down_s = w.attr(mx ? "a_down" : "s_down").cast<Tensor>();
            f_b_up = w.attr("b_up").cast<OptTensor>();
            f_b_down = w.attr("b_down").cast<OptTensor>();
            f_b_down_folded = d["ffn_fp8_folded"].attr("b_down").cast<OptTensor>();
            if (!mx && !w.attr("w_up_bf16").is_none()) f_up_bf16 = w.attr("w_up_bf16").cast<Tensor>();
        } else {
            ffn1 = layer_field(d, "ffn_w1", "ffn_b1", derived);
            ffn2 = layer_field(d, "ffn_w2", "ffn_b2", derived);
        }
    }
};

// The blocks as the forward reads them, with what they were made from
struct BlockSet {
    std::vector<Block> blocks;
    std::vector<Entries> entries;      // a block's dict, then those of its FFN weight objects
    std::vector<size_t> first;         // a block's place in `entries`
    Derived derived;
    explicit BlockSet(const py::list& dicts, const at::Device& device) {
        for (const auto& d : dicts) {
            const auto dict = d.cast<py::dict>();
            blocks.emplace_back(dict, derived);
            first.push_back(entries.size());
            entries.emplace_back(dict);
            for (const char* name : {"ffn_fp8", "ffn_fp8_folded"})
                if (dict.contains(name)) entries.emplace_back(dict[name].attr("__dict__").cast<py::dict>());
        }
        derived.seal(device);
    }
    bool serves(const py::list& dicts) const {
        if (dicts.size() != blocks.size()) return false;
        for (size_t i = 0; i < first.size(); ++i)
            if (!entries[first[i]].of(PyList_GET_ITEM(dicts.ptr(), static_cast<Py_ssize_t>(i)))) return false;
        return std::all_of(entries.begin(), entries.end(), [](const Entries& e) { return e.same(); }) && derived.unchanged();
    }
};

// What `prepare` leaves for the forward of the same batch
struct Prepared {
    int64_t batch = 0, length = 0;
    std::vector<int64_t> widths;
    Tensor src_map, stats, start, n0, counts, cu, cu32, ns_rows, meta;   // meta: pinned host memory
    at::cuda::CUDAEvent ready;
    std::vector<Tensor> tensors() const { return {src_map, stats, start, cu32, ns_rows}; }   // start .. share one allocation
};

enum FfnMode : int { kFfnBf16 = 0, kFfnFp8 = 1, kFfnFp8Precise = 2, kFfnMx = 3 };

class Engine {
public:
    explicit Engine(const py::dict& cfg)
        : d_(field<int64_t>(cfg, "d")), heads_(field<int64_t>(cfg, "heads")), ns_(field<int64_t>(cfg, "ns")), emb_(field<int64_t>(cfg, "emb")),
          ffn_(field<int>(cfg, "ffn")), status_(field<Tensor>(cfg, "status")), edges_(field<Tensor>(cfg, "edges")),
          final_norm_(field<Tensor>(cfg, "final_norm")), head_w_(field<Tensor>(cfg, "head_w")), head_b_(field<Tensor>(cfg, "head_b")),
          classifier_(layer_field(cfg, "classifier_w", "classifier_b", derived_)), classifier_f32_(optional_field(cfg, "classifier_w32")),
          project_(layer_field(cfg, "project_w", "project_b", derived_)), ln_w_(field<Tensor>(cfg, "ln_w")), ln_b_(field<Tensor>(cfg, "ln_b")),
          time_table_(optional_field(cfg, "time_table")), hash_buckets_(field<Tensor>(cfg, "hash_buckets")) {
        for (const auto& t : cfg["seq_tables"]) seq_tables_.push_back(t.cast<OptTensor>());
        type_ = final_norm_.scalar_type();
        device_ = final_norm_.device();
        stats_.emplace(cfg["stats"].cast<py::dict>());
        if (cfg.contains("user") && !cfg["user"].is_none()) {
            user_.emplace(cfg["user"].cast<py::dict>(), derived_);
            item_.emplace(cfg["item"].cast<py::dict>(), derived_);
            if (!cfg["user_dense"].is_none()) user_dense_.emplace(cfg["user_dense"].cast<py::dict>());
            if (!cfg["item_dense"].is_none()) item_dense_.emplace(cfg["item_dense"].cast<py::dict>());
        }
        keep_tensors(cfg);
        weights_ = cfg["weights"].cast<py::dict>();
        for (const auto& name : cfg["watched"]) {
            const py::object value = weights_[name];
            watched_.emplace_back(py::reinterpret_borrow<py::object>(name), value);
            derived_.watch(value.cast<Tensor>());
        }
        derived_.seal(device_);
    }

    // Are the weights that were cast, transposed or split for this executor still those of the model, with the same content?
    bool current() const {
        for (const auto& [name, value] : watched_)
            if (PyDict_GetItem(weights_.ptr(), name.ptr()) != value.ptr()) return false;
        return derived_.unchanged();
    }

    // The blocks of these dicts, read again where an entry, or the content of a weight that was converted, has changed.  The caller
    // holds on to the set: another thread may load the next one while this forward waits without the interpreter's lock.
    std::shared_ptr<BlockSet> load_blocks(const py::list& dicts) {
        if (loaded_ == nullptr || !loaded_->serves(dicts)) loaded_ = std::make_shared<BlockSet>(dicts, device_);
        loaded_->derived.use(device_);
        derived_.use(device_);
        return loaded_;
    }

    bool assembles_ns_tokens() const { return user_.has_value(); }

    // Duplicate removal and statistics of the behaviour sequence and the row plan of the packed layout, enqueued on the
    // current stream.  The totals that size the forward's buffers are written by the plan kernel into pinned host memory.
    std::shared_ptr<Prepared> prepare(const Tensor& values_in, const Tensor& lengths_in, const Tensor& stamps_in, const Tensor& request_in,
                                      std::vector<int64_t> widths, bool timing) {
        Timing::on() = timing;
        const c10::cuda::CUDAGuard guard(device_);
        TORCH_CHECK(values_in.dim() == 3 && values_in.size(1) >= 1 && values_in.size(2) >= 1 && values_in.size(2) <= 8192,
                    "sequence_prepare needs values [B, F, L] with at least one feature and 1 <= L <= 8192");
        check_sequence(device_, values_in.size(0), -1, values_in.size(2), values_in, lengths_in, stamps_in, request_in);
        const Tensor values = i64(values_in), lengths = i64(lengths_in), stamps = i64(stamps_in), request = i64(request_in);
        const int64_t b = values.size(0), f = values.size(1), len = values.size(2);
        const auto layers = static_cast<int64_t>(widths.size()) - 1;
        auto p = std::make_shared<Prepared>();
        p->batch = b;
        p->length = len;
        p->widths = std::move(widths);
        Tensor new_len = make({b}, at::kLong, device_);
        p->src_map = make({b, len}, at::kInt, device_);
        p->stats = make({b, 6}, at::kFloat, device_);
        void* s = stream_of(values);
        {
            TB200_TIMED("sequence_prepare", "batch"_a = b, "n_feat"_a = f, "max_len"_a = len);
            check(tb200_sequence_prepare(data<int64_t>(values), data<int64_t>(lengths), data<int64_t>(stamps), data<int64_t>(request), b,
                                         static_cast<int32_t>(f), static_cast<int32_t>(len), data<int64_t>(new_len), data<int32_t>(p->src_map),
                                         data<float>(p->stats), s), "cuda sequence_prepare");
        }
        // one allocation for the plan's int64 outputs
        const int64_t sizes[] = {b, b, (layers + 1) * b, (layers + 1) * (b + 1), b * ns_, (layers + 1) * ns_ * b};
        int64_t total = 0;
        for (int64_t n : sizes) total += n;
        Tensor flat = make({total}, at::kLong, device_);
        int64_t at = 0;
        auto part = [&](int i) {
            Tensor t = flat.narrow(0, at, sizes[i]);
            at += sizes[i];
            return t;
        };
        p->start = part(0);
        p->n0 = part(1);
        p->counts = part(2);
        p->cu = part(3);
        Tensor ns_rows0 = part(4);
        p->ns_rows = part(5).view({layers + 1, ns_ * b});
        p->cu32 = make({layers + 1, b + 1}, at::kInt, device_);
        // landing buffers are a ring of four: at most three results may be outstanding (allocating pinned memory per batch
        // can stall on the device when the host runs a batch ahead)
        const int64_t meta_size = 2 * (layers + 1);
        if (ring_.empty() || ring_[0].numel() != meta_size) {
            ring_.clear();
            for (int i = 0; i < 4; ++i) ring_.push_back(at::empty({meta_size}, at::TensorOptions().dtype(at::kLong).pinned_memory(true)));
        }
        p->meta = ring_[ring_next_++ % ring_.size()];
        std::vector<int32_t> w(p->widths.begin(), p->widths.end());
        {
            TB200_TIMED("pyramid_plan", "batch"_a = b, "layers"_a = layers);
            check(tb200_pyramid_plan_rows(data<int64_t>(new_len), static_cast<int32_t>(b), static_cast<int32_t>(len), w.data(),
                                          static_cast<int32_t>(layers), static_cast<int32_t>(ns_), data<int64_t>(p->start), data<int64_t>(p->n0),
                                          data<int64_t>(p->counts), data<int64_t>(p->cu), data<int32_t>(p->cu32), data<int64_t>(p->meta),
                                          data<int64_t>(ns_rows0), data<int64_t>(p->ns_rows), s), "cuda pyramid_plan");
        }
        const auto stream = c10::cuda::getCurrentCUDAStream(device_.index());
        // the kernel writes the landing buffer: its memory is not given out before, also when nobody waits for the result
        at::getHostAllocator(at::kCUDA)->record_event(p->meta.data_ptr(), p->meta.storage().data_ptr().get_context(), stream.unwrap());
        p->ready.record(stream);
        return p;
    }

    // Tokenizers and blocks of a prepared batch.  -> (done, tokens, layer, token_major, seq_mean, ns_mean): with `done` the two
    // pooled means; otherwise the residual stream of a batch that holds nothing but non-sequence tokens from `layer` on.
    py::tuple blocks(const std::shared_ptr<Prepared>& p, const Tensor& values_in, const OptTensor& stamps_in, const Tensor& request_in,
                     const py::tuple& entities, const OptTensor& ns_tokens_in, const Tensor& positions, const py::list& block_dicts,
                     bool select_early, bool one_kernel, int attention_kernel, bool timing);

    Tensor ns_only(const Tensor& tokens, int64_t first_layer, int64_t batch, bool token_major, const py::list& block_dicts, int attention_kernel,
                   bool timing);

    // -> (logits, embeddings, probabilities), fp32
    py::tuple classify(const OptTensor& seq_mean, const Tensor& ns_mean, bool timing);

private:
    static Tensor i64(const Tensor& t) { return t.scalar_type() == at::kLong && t.is_contiguous() ? t : t.to(at::kLong).contiguous(); }
    // act(x w^T + b) (+ residual), x [M, K]: this library's GEMM where the widths are whole tiles, the library's otherwise
    Tensor proj(const Tensor& x, const Layer& l, bool silu = false, const OptTensor& residual = std::nullopt, const OptTensor& out = std::nullopt) const {
        const int64_t n = l.w.size(0), k = l.w.size(1);
        if (l.own.defined()) return grouped(x, l.own, l.b32, silu, residual, out, status_);
        Tensor y;
        {
            TB200_TIMED("cublas_linear", "m"_a = x.numel() / k, "n"_a = n, "k"_a = k);
            y = at::linear(x, l.w, l.b);
        }
        if (silu) at::silu_(y);
        if (residual.has_value()) y.add_(*residual);
        if (!out.has_value()) return y;
        out->copy_(y);
        return *out;
    }

    void keep_tensors(const py::dict& d) {
        for (const auto& item : d) {
            if (THPVariable_Check(item.second.ptr())) derived_.keep(item.second.cast<Tensor>());
            else if (py::isinstance<py::dict>(item.second) && item.first.cast<std::string>() != "weights") keep_tensors(item.second.cast<py::dict>());
        }
    }

    Tensor native_ns_tokens(const py::tuple& entities, const Prepared& p);
    Tensor shared_ffn(const Block& blk, const Tensor& x, const Tensor& tokens, bool folded) const;

    Derived derived_;                 // before the members that are made with it
    int64_t d_, heads_, ns_, emb_;
    int ffn_;
    Tensor status_, edges_, final_norm_, head_w_, head_b_;
    Layer classifier_;
    OptTensor classifier_f32_;
    Layer project_;
    Tensor ln_w_, ln_b_;
    OptTensor time_table_;
    Tensor hash_buckets_;
    std::vector<OptTensor> seq_tables_;
    at::ScalarType type_;
    at::Device device_{at::kCUDA};
    std::optional<SmallToken> stats_, user_dense_, item_dense_;
    std::optional<EntityTokens> user_, item_;
    std::shared_ptr<BlockSet> loaded_;
    py::dict weights_;                                        // the model's weights by name
    std::vector<std::pair<py::object, py::object>> watched_;  // names and tensors of those that were converted for this executor
    std::vector<Tensor> ring_;
    size_t ring_next_ = 0;
};

// All non-sequence tokens [B, ns, d] (experiments/onetrans/model.py:240-252), every part written to its place:
// user tokens | user dense | item tokens | item dense | sequence statistics
Tensor Engine::native_ns_tokens(const py::tuple& entities, const Prepared& p) {
    const int64_t b = p.batch, es = final_norm_.element_size();
    Tensor out = make({b, ns_, d_}, type_, device_);
    int64_t slot = 0;
    auto place = [&](int64_t tokens) {
        char* at = static_cast<char*>(out.data_ptr()) + slot * d_ * es;
        slot += tokens;
        return at;
    };
    for (int who = 0; who < 2; ++who) {
        const EntityTokens& e = who == 0 ? *user_ : *item_;
        const auto& dense = who == 0 ? user_dense_ : item_dense_;
        const py::tuple parts = entities[who].cast<py::tuple>();
        const Tensor ids = parts[0].cast<Tensor>().contiguous();
        Tensor feats = make({b, e.n_fields * e.dim}, type_, device_);
        {
            TB200_TIMED("fields_bag_mean", "ids"_a = ids, "dim"_a = e.dim, "esize"_a = es, "n_fields"_a = e.n_fields);
            void* s = stream_of(feats);
            const int dt = dtype_code(type_), it = id_code(ids.scalar_type());
            int code;
            if (e.missing_rows.has_value()) {
                const Tensor miss = parts[1].cast<Tensor>().contiguous();
                code = tb200_fields_bag_mean_missing_fwd(static_cast<const void* const*>(ptr(e.ptrs)), data<int64_t>(e.rows), data<int32_t>(e.offsets),
                                                         data<int32_t>(e.lengths), static_cast<int32_t>(e.n_fields), static_cast<int32_t>(e.max_bag),
                                                         static_cast<int32_t>(e.dim), ptr(ids), it, b, static_cast<int32_t>(ids.size(1)),
                                                         data<uint8_t>(miss), static_cast<int32_t>(miss.size(1)), ptr(*e.missing_rows), ptr(feats), dt, s);
            } else {
                code = tb200_fields_bag_mean_fwd(static_cast<const void* const*>(ptr(e.ptrs)), data<int64_t>(e.rows), data<int32_t>(e.offsets),
                                                 data<int32_t>(e.lengths), static_cast<int32_t>(e.n_fields), static_cast<int32_t>(e.max_bag),
                                                 static_cast<int32_t>(e.dim), ptr(ids), it, b, static_cast<int32_t>(ids.size(1)), ptr(feats), dt, s);
            }
            check(code, "cuda fields_bag_mean");
        }
        const Tensor h = proj(feats, e.project);
        {
            const int64_t cols = e.n_tokens * d_;
            TB200_TIMED("layer_norm", "rows"_a = b, "cols"_a = cols, "esize"_a = es);
            check(tb200_layernorm_silu_strided_fwd(ptr(h), ptr(e.gamma), ptr(e.beta), place(e.n_tokens), b, static_cast<int32_t>(cols), ns_ * d_, 1e-5f,
                                                   dtype_code(type_), stream_of(h)), "cuda layer_norm");
        }
        if (dense.has_value()) {
            OptTensor miss;
            if (!parts[3].is_none()) miss = parts[3].cast<Tensor>();
            dense->run(parts[2].cast<Tensor>(), miss, place(1), ns_ * d_, type_);
        }
    }
    stats_->run(p.stats, std::nullopt, place(1), ns_ * d_, type_);
    return out;
}

// tokens + FFN(x) of the shared feed-forward; `folded`: its output bias carries the attention projection's as well
Tensor Engine::shared_ffn(const Block& blk, const Tensor& x, const Tensor& tokens, bool folded) const {
    if (ffn_ == kFfnBf16) return proj(proj(x, blk.ffn1, true), blk.ffn2, false, tokens);
    const int64_t m = x.size(0), hidden = blk.f_down.size(1);
    const auto k = static_cast<int32_t>(d_), hid = static_cast<int32_t>(hidden);
    void* s = stream_of(x);
    auto* status = data<int32_t>(status_);
    auto* b_down = data<float>(folded ? blk.f_b_down_folded : blk.f_b_down);
    Tensor h = make({m, hidden}, at::kFloat8_e4m3fn, device_), out = make_like(tokens.sizes(), tokens);
    if (ffn_ == kFfnMx) {
        const int64_t tiles = (m + 127) / 128;
        auto atoms = [&](int64_t width) {   // rows behind the end of a ragged last tile have zero scales
            Tensor t = make({tiles, width / 128, 512}, at::kByte, device_);
            if (m % 128 != 0) t.zero_();
            return t;
        };
        Tensor xq = make({m, d_}, at::kFloat8_e4m3fn, device_), xa = atoms(d_), ha = atoms(hidden);
        {
            TB200_TIMED("quant_act", "rows"_a = m, "cols"_a = d_);
            check(tb200_quant_act_mx(ptr(x), ptr(xq), data<uint8_t>(xa), m, k, s), "cuda quantize_activation_mx");
        }
        {
            TB200_TIMED("mx_gemm_silu", "m"_a = m, "n"_a = hidden, "k"_a = d_);
            check(tb200_mx_gemm(ptr(xq), data<uint8_t>(xa), ptr(blk.f_up), data<uint8_t>(blk.f_up_s), data<float>(blk.f_b_up), nullptr, ptr(h),
                                data<uint8_t>(ha), m, hid, k, 1, status, s), "cuda mx_gemm");
        }
        TB200_TIMED("mx_gemm_linear", "m"_a = m, "n"_a = d_, "k"_a = hidden);
        check(tb200_mx_gemm(ptr(h), data<uint8_t>(ha), ptr(blk.f_down), data<uint8_t>(blk.f_down_s), b_down, ptr(tokens), ptr(out), nullptr, m, k, hid,
                            2, status, s), "cuda mx_gemm");
        return out;
    }
    Tensor sh = make({m, hidden / 128}, at::kFloat, device_);
    if (ffn_ == kFfnFp8Precise) {
        Tensor hb = make({m, hidden}, at::kBFloat16, device_);
        {
            TB200_TIMED("gemm_bf16", "groups"_a = 1, "m"_a = m, "n"_a = hidden, "k"_a = d_, "silu"_a = true, "residual"_a = false);
            check(tb200_gemm_bf16_grouped(ptr(x), ptr(blk.f_up_bf16), data<float>(blk.f_b_up), nullptr, ptr(hb), 1, m, hid, k, 1, status, s),
                  "cuda grouped_linear");
        }
        TB200_TIMED("quant_act", "rows"_a = m, "cols"_a = hidden);
        check(tb200_quant_act_1x128(ptr(hb), ptr(h), data<float>(sh), m, hid, s), "cuda quantize_activation_1x128");
    } else {
        Tensor xq = make({m, d_}, at::kFloat8_e4m3fn, device_), sx = make({m, d_ / 128}, at::kFloat, device_);
        {
            TB200_TIMED("quant_act", "rows"_a = m, "cols"_a = d_);
            check(tb200_quant_act_1x128(ptr(x), ptr(xq), data<float>(sx), m, k, s), "cuda quantize_activation_1x128");
        }
        TB200_TIMED("fp8_gemm_silu", "m"_a = m, "n"_a = hidden, "k"_a = d_);
        check(tb200_fp8_gemm(ptr(xq), data<float>(sx), ptr(blk.f_up), data<float>(blk.f_up_s), data<float>(blk.f_b_up), nullptr, ptr(h),
                             data<float>(sh), m, hid, k, 1, status, s), "cuda fp8_gemm");
    }
    TB200_TIMED("fp8_gemm_linear", "m"_a = m, "n"_a = d_, "k"_a = hidden);
    check(tb200_fp8_gemm(ptr(h), data<float>(sh), ptr(blk.f_down), data<float>(blk.f_down_s), b_down, ptr(tokens), ptr(out), nullptr, m, k, hid, 2,
                         status, s), "cuda fp8_gemm");
    return out;
}

py::tuple Engine::blocks(const std::shared_ptr<Prepared>& p, const Tensor& values_in, const OptTensor& stamps_in, const Tensor& request_in,
                         const py::tuple& entities, const OptTensor& ns_tokens_in, const Tensor& positions, const py::list& block_dicts,
                         bool select_early, bool one_kernel, int attention_kernel, bool timing) {
    Timing::on() = timing;
    const c10::cuda::CUDAGuard guard(device_);
    derived_.use(device_);
    const int64_t b = p->batch, n_feat = static_cast<int64_t>(seq_tables_.size()), max_len = p->length;
    check_sequence(device_, b, n_feat, max_len, values_in, std::nullopt, std::nullopt, request_in);
    if (time_table_.has_value()) require(stamps_in, "timestamps", device_, {b, max_len});
    if (ns_tokens_in.has_value()) {
        require(ns_tokens_in, "ns_tokens", device_, {b, ns_, d_});
    } else {
        for (int who = 0; who < 2; ++who) {
            const EntityTokens& e = who == 0 ? *user_ : *item_;
            const auto& dense = who == 0 ? user_dense_ : item_dense_;
            const py::tuple parts = entities[who].cast<py::tuple>();
            const auto optional = [&](int i) { return parts[i].is_none() ? OptTensor() : OptTensor(parts[i].cast<Tensor>()); };
            check_entity(device_, b, parts[0].cast<Tensor>(), e.id_columns, optional(1), e.missing_rows.has_value() ? e.n_fields : 0, optional(2),
                         optional(3), dense.has_value() ? dense->inputs : 0);
        }
    }
    const Tensor values = i64(values_in), request = i64(request_in);
    // the non-sequence tokens need nothing the host has to wait for
    const Tensor ns_tokens = (ns_tokens_in.has_value() ? *ns_tokens_in : native_ns_tokens(entities, *p)).contiguous();
    const auto loaded = load_blocks(block_dicts);
    const std::vector<Block>& stack = loaded->blocks;
    const auto& widths = p->widths;
    const auto layers = static_cast<int64_t>(stack.size());
    TORCH_CHECK(static_cast<int64_t>(widths.size()) == layers + 1, "OneTransInference: prepared for ", widths.size() - 1, " blocks, the model has ", layers);
    {   // the one host read of a forward; already there when the serving loop prepared the batch ahead of time
        py::gil_scoped_release nogil;
        p->ready.synchronize();
    }
    const int64_t* meta = p->meta.data_ptr<int64_t>();
    std::vector<int64_t> totals(layers + 1), max_rows(layers + 1);
    for (int64_t l = 0; l <= layers; ++l) {
        totals[l] = meta[2 * l];
        max_rows[l] = meta[2 * l + 1];
    }
    auto cu = [&](int64_t l) { return data<int64_t>(p->cu) + l * (b + 1); };
    auto cu32 = [&](int64_t l) { return p->cu32.select(0, l); };
    auto counts = [&](int64_t l) { return data<int64_t>(p->counts) + l * b; };
    auto ns_ids = [&](int64_t l) { return p->ns_rows.select(0, l); };   // token-major row ids [ns * B]
    void* s = stream_of(values);

    // ---- sequence tokenizer on the valid events only, in the packed layout of layer 0: the rows reserved for the
    // non-sequence tokens go through it as padding ids and are overwritten afterwards
    const int64_t total0 = totals[0];
    const bool has_time = time_table_.has_value();
    Tensor ids = make({n_feat, total0}, at::kLong, device_), pos = make({total0}, at::kLong, device_);
    OptTensor buckets, stamps;
    if (has_time) {
        buckets = make({total0}, at::kLong, device_);
        stamps = i64(*stamps_in);
    }
    {
        TB200_TIMED("packed_token_index", "batch"_a = b, "n_feat"_a = n_feat, "rows"_a = total0);
        check(tb200_packed_token_index(data<int64_t>(values), data<int64_t>(stamps), data<int64_t>(request), data<int32_t>(p->src_map), cu(0),
                                       data<int64_t>(p->n0), data<int64_t>(p->start), has_time ? data<int64_t>(edges_) : nullptr,
                                       has_time ? static_cast<int32_t>(edges_.numel()) : 0, data<int64_t>(hash_buckets_), b,
                                       static_cast<int32_t>(n_feat), static_cast<int32_t>(max_len), total0, data<int64_t>(ids), data<int64_t>(pos),
                                       data<int64_t>(buckets), s), "cuda packed_token_index");
    }
    // rows of a layer that the pyramid keeps for the next one, in the next layer's order; on request the destination of every row
    auto kept_rows = [&](int64_t l, OptTensor* row_dst) {
        Tensor src = make({std::max<int64_t>(totals[l + 1], 1)}, at::kLong, device_), unused = make({b, ns_}, at::kLong, device_);
        if (row_dst != nullptr) *row_dst = make({std::max<int64_t>(totals[l], 1)}, at::kInt, device_);
        TB200_TIMED("pyramid_kept_rows", "batch"_a = b);
        check(tb200_pyramid_kept_rows(cu(l), cu(l + 1), counts(l), counts(l + 1), static_cast<int32_t>(b), static_cast<int32_t>(ns_),
                                      data<int64_t>(src), data<int64_t>(unused), row_dst != nullptr ? data<int32_t>(*row_dst) : nullptr, s),
              "cuda pyramid_kept_rows");
        return src.narrow(0, 0, totals[l + 1]);
    };
    // When the first block is evaluated for the kept rows only, its residual stream is needed for those rows alone: the
    // tokenizer's last kernel then writes `tokens` already compacted and only the normalised rows at full height.
    bool first_kept = select_early && widths[1] < widths[0] && max_rows[0] != ns_ && totals[1] < (1ll << 31);
    OptTensor row_dst;
    Tensor first_src;
    if (first_kept) first_src = kept_rows(0, &row_dst);
    const int64_t rows_out = first_kept ? totals[1] : total0;
    const Tensor& first_norm = stack[0].attn_norm;
    const Tensor& table_a = has_time ? *time_table_ : positions;
    const int64_t* ids_a = has_time ? data<int64_t>(buckets) : data<int64_t>(pos);
    Tensor tokens = make({rows_out, d_}, type_, device_), x = make({total0, d_}, type_, device_);
    if (one_kernel) {
        std::vector<const void*> tables;
        std::vector<int64_t> table_rows;
        for (int64_t f = 0; f < n_feat; ++f) {
            tables.push_back(ptr(seq_tables_[f]));
            table_rows.push_back(seq_tables_[f].has_value() ? seq_tables_[f]->size(0) : 1);
        }
        TB200_TIMED("token_project", "rows"_a = total0, "cols"_a = d_, "k"_a = n_feat * emb_, "rows_out"_a = rows_out, "ids"_a = ids, "bytes"_a = 0);
        check(tb200_token_project_fwd(tables.data(), table_rows.data(), static_cast<int32_t>(n_feat), static_cast<int32_t>(emb_), data<int64_t>(ids),
                                      ptr(project_.w), data<float>(project_.b32), ptr(ln_w_), ptr(ln_b_), ptr(table_a), table_a.size(0), ids_a,
                                      has_time ? ptr(positions) : nullptr, has_time ? positions.size(0) : 0, has_time ? data<int64_t>(pos) : nullptr,
                                      ptr(first_norm), data<int32_t>(row_dst), rows_out, ptr(tokens), ptr(x), total0, static_cast<int32_t>(d_), 1e-5f,
                                      1e-6f, data<int32_t>(status_), s), "cuda token_project");
    } else {
        bool all_tables = true, any_table = false;
        for (const auto& t : seq_tables_) {
            all_tables &= t.has_value();
            any_table |= t.has_value();
        }
        Tensor features = make({total0, any_table ? n_feat * emb_ : project_.w.size(1)}, type_, device_);
        if (!all_tables) features.zero_();
        for (int64_t f = 0; f < n_feat; ++f)
            if (seq_tables_[f].has_value())
                gather_rows_into(*seq_tables_[f], data<int64_t>(ids) + f * total0, Timing::on() ? ids.select(0, f) : Tensor(), features, f * emb_);
        const Tensor projected = proj(features, project_);
        TB200_TIMED("token_tail", "rows"_a = total0, "cols"_a = d_, "esize"_a = x.element_size(), "tables"_a = has_time ? 2 : 1, "rows_out"_a = rows_out);
        check(tb200_token_tail_select_fwd(ptr(projected), ptr(ln_w_), ptr(ln_b_), ptr(table_a), table_a.size(0), ids_a,
                                          has_time ? ptr(positions) : nullptr, has_time ? positions.size(0) : 0, has_time ? data<int64_t>(pos) : nullptr,
                                          ptr(first_norm), data<int32_t>(row_dst), rows_out, ptr(tokens), ptr(x), total0, static_cast<int32_t>(d_), 1e-5f,
                                          1e-6f, dtype_code(type_), s), "cuda token_tail");
    }

    // ---- the non-sequence tokens take the rows left for them
    Tensor x_ns = make({ns_, b, d_}, type_, device_);
    {
        const Tensor token_ids = ns_ids(first_kept ? 1 : 0), normed_ids = ns_ids(0);
        TB200_TIMED("scatter_rows", "rows"_a = 2 * ns_ * b, "dim"_a = d_, "esize"_a = x.element_size());
        check(tb200_ns_rows_fwd(ptr(ns_tokens), b, static_cast<int32_t>(ns_), static_cast<int32_t>(d_), ptr(first_norm), 1e-6f, data<int64_t>(token_ids),
                                ptr(tokens), data<int64_t>(normed_ids), ptr(x), ptr(x_ns), dtype_code(type_), s), "cuda ns_rows");
    }

    const int64_t hd = d_ / heads_;
    auto heads_view = [&](const Tensor& m, int64_t part) {   // columns [part d, part d + d) of a [rows, parts d] matrix as [rows, H, hd]
        return m.as_strided({m.size(0), heads_, hd}, {m.size(1), hd, 1}, m.storage_offset() + part * d_);
    };
    for (int64_t l = 0; l < layers; ++l) {
        const Block& blk = stack[l];
        const bool g = blk.grouped_layers;
        if (max_rows[l] == ns_)   // no sample has a sequence token left from here on
            return py::make_tuple(false, tokens, l, false, py::none(), py::none());
        const Tensor ids_here = ns_ids(l);
        if (l > 0) {
            x = rms_norm(tokens, blk.attn_norm);
            x_ns = gather_rows(x, ids_here).view({ns_, b, d_});
        }
        const bool selected = select_early && widths[l + 1] < widths[l];
        // every row the pyramid keeps is a non-sequence row: the rest of the block runs token-major on those alone
        const bool only_ns_kept = selected && max_rows[l + 1] == ns_ && g && hd == 64 && type_ == at::kBFloat16 && (attention_kernel == 0 || attention_kernel == 4);
        const Tensor ids_next = selected ? ns_ids(l + 1) : ids_here;
        Tensor attn;
        if (only_ns_kept) {
            // keys and values for every row; queries, attention rows and everything behind them for the non-sequence tokens, token-major
            // as the blocks behind this one want them.  The projection's bias is added by the norm on the fly and rides on the
            // feed-forward's output bias into the next residual.
            const Tensor kv = proj(x, blk.kv);
            const Tensor qkv = grouped(x_ns, blk.g_qkv_w, blk.g_qkv_b, false, std::nullopt, std::nullopt, status_);
            scatter_rows(kv, ids_here, qkv.narrow(2, d_, 2 * d_));
            attn = make({ns_, b, d_}, type_, device_);
            {
                const int64_t st[12] = {3 * d_, hd, b * 3 * d_, 0, hd, 2 * d_, 0, hd, 2 * d_, d_, hd, b * d_};
                const Tensor cu_here = cu32(l);
                TB200_TIMED("attention_fewq", "seq_len"_a = py::none(), "cu_rows"_a = cu_here, "cu_rows_q"_a = cu32(l + 1), "key_valid"_a = py::none(),
                            "batch"_a = b, "heads"_a = heads_, "lq"_a = ns_, "lk"_a = max_rows[l], "dim"_a = hd, "ns_start"_a = max_rows[l],
                            "causal"_a = true, "self_rows"_a = false, "esize"_a = qkv.element_size());
                check(tb200_attn_last_rows_fwd(ptr(qkv), ptr(kv), static_cast<char*>(kv.data_ptr()) + d_ * kv.element_size(), ptr(attn),
                                               static_cast<int32_t>(b), static_cast<int32_t>(heads_), static_cast<int32_t>(ns_),
                                               static_cast<int32_t>(max_rows[l]), st, data<int32_t>(cu_here),
                                               static_cast<float>(1.0 / std::sqrt(static_cast<double>(hd))), dtype_code(type_), s), "cuda varlen_attention");
            }
            const Tensor tok = gather_rows(tokens, l == 0 && first_kept ? ids_next : ids_here).view({ns_, b, d_});
            add_shared_linear(tok, attn, blk.g_out_w, status_);
            const Tensor h = norm_grouped(tok, blk.ffn_norm, blk.out_b, blk.g_w1, blk.g_b1, true, status_);
            grouped(h, blk.g_w2, blk.g_b2_folded, false, tok, tok, status_);
            return py::make_tuple(false, tok, l + 1, true, py::none(), py::none());
        }
        if (selected) {
            // The pyramid keeps only the last rows of every sample after this block, and a row of the block's output depends
            // on the other rows through its keys and values alone: keys and values are projected for every row, the rest
            // runs for the rows that survive.
            const Tensor src = l == 0 && first_kept ? first_src : kept_rows(l, nullptr);
            const Tensor kv = proj(x, blk.kv);
            const Tensor qm = proj(gather_rows(x, src), blk.q);
            if (g) {
                const Tensor qkv = grouped(x_ns, blk.g_qkv_w, blk.g_qkv_b, false, std::nullopt, std::nullopt, status_);
                scatter_rows(kv, ids_here, qkv.narrow(2, d_, 2 * d_));
                scatter_rows(qm, ids_next, qkv.narrow(2, 0, d_));
            } else {
                scatter_rows(kv, ids_here, at::bmm(x_ns, blk.ns_kv_w), blk.ns_kv_b);
                scatter_rows(qm, ids_next, at::bmm(x_ns, blk.ns_q_w), blk.ns_q_b);
            }
            const int kernel = attention_kernel == 1 || attention_kernel == 4 ? attention_kernel : 0;
            attn = packed_attention(heads_view(qm, 0), heads_view(kv, 0), heads_view(kv, 1), cu32(l), max_rows[l], cu32(l + 1), max_rows[l + 1], kernel,
                                    status_);
            if (!(l == 0 && first_kept)) tokens = gather_rows(tokens, src);
        } else {
            const Tensor qkv = proj(x, blk.qkv);
            if (g) scatter_rows(qkv, ids_here, grouped(x_ns, blk.g_qkv_w, blk.g_qkv_b, false, std::nullopt, std::nullopt, status_));
            else scatter_rows(qkv, ids_here, at::bmm(x_ns, blk.ns_qkv_w), blk.ns_qkv_b);
            attn = packed_attention(heads_view(qkv, 0), heads_view(qkv, 1), heads_view(qkv, 2), cu32(l), max_rows[l], std::nullopt, 0, attention_kernel,
                                    status_);
        }
        const Tensor attn2d = attn.view({-1, d_});
        const bool folded = ffn_ != kFfnBf16;
        if (folded) {
            proj(attn2d, blk.out_nobias, false, tokens, tokens);
            x = rms_norm(tokens, blk.ffn_norm, blk.out_b);
        } else {
            tokens = proj(attn2d, blk.out, false, tokens);
            x = rms_norm(tokens, blk.ffn_norm);
        }
        const Tensor out = shared_ffn(blk, x, tokens, folded);
        x_ns = gather_rows(x, ids_next).view({ns_, b, d_});
        if (g) {
            const Tensor h = grouped(x_ns, blk.g_w1, blk.g_b1, true, std::nullopt, std::nullopt, status_);
            scatter_rows(out, ids_next, grouped(h, blk.g_w2, folded ? blk.g_b2_folded : blk.g_b2, false, std::nullopt, std::nullopt, status_),
                         std::nullopt, tokens);
        } else {
            const Tensor h = bias_act_rows(at::bmm(x_ns, blk.ns_w1), blk.ns_b1, true);
            scatter_rows(out, ids_next, at::bmm(h, blk.ns_w2), folded ? blk.ns_b2_folded : blk.ns_b2, tokens);
        }
        tokens = out;
        if (!selected && widths[l + 1] < widths[l]) tokens = gather_rows(tokens, kept_rows(l, nullptr));
    }
    Tensor seq_mean = make({b, d_}, at::kFloat, device_), ns_mean = make({b, d_}, at::kFloat, device_);
    {
        TB200_TIMED("pool_rows", "rows"_a = totals[layers], "cols"_a = d_, "esize"_a = x.element_size());
        check(tb200_pool_rows_fwd(ptr(tokens), cu(layers), counts(layers), b, static_cast<int32_t>(ns_), static_cast<int32_t>(d_), ptr(final_norm_),
                                  1e-6f, data<float>(seq_mean), data<float>(ns_mean), dtype_code(type_), s), "cuda pool_rows");
    }
    return py::make_tuple(true, py::none(), layers, false, seq_mean, ns_mean);
}

// Blocks first_layer .. end for a batch whose samples hold nothing but their non-sequence tokens, then the final norm and
// their mean -> [B, d] fp32.  Every row takes the per-token projections and feed-forward and every sample attends causally
// over its ns tokens: six batched or shared matrix products per block on a token-major [ns, B, d] tensor.
Tensor Engine::ns_only(const Tensor& tokens, int64_t first_layer, int64_t batch, bool token_major, const py::list& block_dicts, int attention_kernel,
                       bool timing) {
    Timing::on() = timing;
    const c10::cuda::CUDAGuard guard(device_);
    const auto loaded = loaded_ != nullptr ? loaded_ : load_blocks(block_dicts);   // `blocks` has looked at them in this forward
    loaded->derived.use(device_);
    const std::vector<Block>& stack = loaded->blocks;
    const int64_t hd = d_ / heads_;
    Tensor tok = (token_major ? tokens : tokens.view({batch, ns_, d_}).transpose(0, 1)).contiguous().view({ns_, batch, d_});
    for (size_t l = static_cast<size_t>(first_layer); l < stack.size(); ++l) {
        const Block& blk = stack[l];
        const bool g = blk.grouped_layers;
        const Tensor qkv = g ? norm_grouped(tok, blk.attn_norm, std::nullopt, blk.g_qkv_w, blk.g_qkv_b, false, status_)
                             : bias_act_rows(at::bmm(rms_norm(tok, blk.attn_norm), blk.ns_qkv_w), blk.ns_qkv_b, false);
        Tensor attn = make({ns_, batch, d_}, type_, device_);
        {
            // sample-major views of the token-major tensors: (B, H, L = ns, hd)
            int64_t st[12];
            for (int i = 0; i < 3; ++i) {
                st[3 * i] = 3 * d_;
                st[3 * i + 1] = hd;
                st[3 * i + 2] = batch * 3 * d_;
            }
            st[9] = d_;
            st[10] = hd;
            st[11] = batch * d_;
            const char* q = static_cast<const char*>(qkv.data_ptr());
            const int64_t part = d_ * qkv.element_size();
            TB200_TIMED(ns_ <= 32 && hd == 64 ? "attention_small" : "attention_mma", "seq_len"_a = py::none(), "cu_rows"_a = py::none(),
                        "cu_rows_q"_a = py::none(), "key_valid"_a = py::none(), "batch"_a = batch, "heads"_a = heads_, "lq"_a = ns_, "lk"_a = ns_,
                        "dim"_a = hd, "ns_start"_a = ns_, "causal"_a = true, "self_rows"_a = false, "esize"_a = qkv.element_size());
            check(tb200_attn_fwd(q, q + part, q + 2 * part, ptr(attn), static_cast<int32_t>(batch), static_cast<int32_t>(heads_),
                                 static_cast<int32_t>(ns_), static_cast<int32_t>(ns_), static_cast<int32_t>(hd), st, nullptr, nullptr, nullptr, nullptr,
                                 static_cast<int32_t>(ns_), 1, 0, static_cast<float>(1.0 / std::sqrt(static_cast<double>(hd))), dtype_code(type_),
                                 attention_kernel, 0, data<int32_t>(status_), stream_of(qkv)), "cuda varlen_attention");
        }
        // the output projection onto the residual stream; its bias is added by the norm on the fly and rides on the
        // feed-forward's output bias into the next residual
        if (g) {
            add_shared_linear(tok, attn, blk.g_out_w, status_);
            const Tensor h = norm_grouped(tok, blk.ffn_norm, blk.out_b, blk.g_w1, blk.g_b1, true, status_);
            grouped(h, blk.g_w2, blk.g_b2_folded, false, tok, tok, status_);
        } else {
            tok.view({ns_ * batch, d_}).addmm_(attn.view({ns_ * batch, d_}), blk.out_w_t);
            const Tensor h = bias_act_rows(at::bmm(rms_norm(tok, blk.ffn_norm, blk.out_b), blk.ns_w1), blk.ns_b1, true);
            tok = bias_act_rows(at::baddbmm(tok, h, blk.ns_w2), blk.ns_b2_folded, false);
        }
    }
    Tensor mean = make({batch, d_}, at::kFloat, device_);
    TB200_TIMED("pool_rows", "rows"_a = ns_ * batch, "cols"_a = d_, "esize"_a = tok.element_size());
    check(tb200_pool_rows_fwd(ptr(tok), nullptr, nullptr, batch, static_cast<int32_t>(ns_), static_cast<int32_t>(d_), ptr(final_norm_), 1e-6f, nullptr,
                              data<float>(mean), dtype_code(type_), stream_of(tok)), "cuda pool_rows");
    return mean;
}

py::tuple Engine::classify(const OptTensor& seq_mean, const Tensor& ns_mean, bool timing) {
    Timing::on() = timing;
    const c10::cuda::CUDAGuard guard(device_);
    const int64_t b = ns_mean.size(0), actions = head_w_.size(0);
    derived_.use(device_);
    const bool own = classifier_.own.defined();
    Tensor joined = make({b, 2 * d_}, at::kFloat, device_), h;
    OptTensor joined_cast;
    if (own && type_ != at::kFloat) joined_cast = make({b, 2 * d_}, type_, device_);
    void* s = stream_of(ns_mean);
    check(tb200_join_summaries(data<float>(seq_mean), data<float>(ns_mean), data<float>(joined), ptr(joined_cast), b, static_cast<int32_t>(d_),
                               dtype_code(type_), s), "cuda join_summaries");
    if (own) {
        // serving mode: the wide layer on the tcgen05 GEMM; its inputs come out of a 16-bit network, so 16-bit operands with
        // fp32 accumulation lose nothing that was still there
        h = proj(joined_cast.value_or(joined), classifier_, true);
    } else {
        TB200_TIMED("cublas_linear", "m"_a = b, "n"_a = d_, "k"_a = 2 * d_);
        h = at::silu(at::linear(joined, *classifier_f32_, classifier_.b32));
    }
    Tensor logits = make({b, actions}, at::kFloat, device_), probs = make({b, actions}, at::kFloat, device_);
    check(tb200_head_fwd(ptr(h), data<float>(head_w_), data<float>(head_b_), data<float>(logits), data<float>(probs), b, static_cast<int32_t>(d_),
                         static_cast<int32_t>(actions), dtype_code(h.scalar_type()), s), "cuda head");
    return py::make_tuple(logits, joined, probs);
}

}  // namespace

void bind_engine(PyObject* module) {
    auto m = py::reinterpret_borrow<py::module_>(module);
    m.def("check_sequence", &check_sequence);
    m.def("check_entity", &check_entity);
    py::class_<Prepared, std::shared_ptr<Prepared>>(m, "Prepared")
        .def_readonly("batch", &Prepared::batch)
        .def_readonly("widths", &Prepared::widths)
        .def_readonly("stats", &Prepared::stats)
        .def("tensors", &Prepared::tensors);
    py::class_<Engine>(m, "Engine")
        .def(py::init<py::dict>())
        .def("current", &Engine::current)
        .def("load_blocks", [](Engine& e, const py::list& dicts) { e.load_blocks(dicts); })
        .def("assembles_ns_tokens", &Engine::assembles_ns_tokens)
        .def("prepare", &Engine::prepare)
        .def("blocks", &Engine::blocks)
        .def("ns_only", &Engine::ns_only)
        .def("classify", &Engine::classify);
}

}  // namespace tb200_host
