// Native host path of the calls a decode step makes once per layer: descriptor checks, workspace and decode-table
// look-ups, output allocation and the launch, in one call from Python instead of some fifty interpreted steps and two
// ctypes conversions.  Same checks and messages as the Python layer, which stays the owner of workspaces: one that has to
// grow is asked for by calling back into comp_inference_b200._lib.
//
// Measured, RansLinear.forward of a 512 x 4096 shard, one row, back to back: 25.5 us in Python, 7.0 to 7.5 here, of which
// 0.47 is finding that the module's buffers are still the same; the kernel itself takes 5.6.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <mutex>
#include <optional>
#include <unordered_map>

#include "../../include/comp_inference_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = c10::optional<Tensor>;

namespace {

void check(int rc) {
    if (rc != 0) throw std::runtime_error("comp_inference_b200: " + std::string(ci_last_error()) + " (code " + std::to_string(rc) + ")");
}

void require_cuda(const Tensor &t, const char *name) {
    TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor: this package has no CPU path");
}

py::object lib_attr(const char *name) { return py::module_::import("comp_inference_b200._lib").attr(name); }

// Launches go to the current stream of the current device, as everywhere in this package.
ci_stream_t stream() { return reinterpret_cast<ci_stream_t>(c10::cuda::getCurrentCUDAStream().stream()); }

// While a stream captures, nothing can be read back, and what a kernel writes exists only once the graph has run.
bool capturing() { return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }

struct StreamKey {
    int device;
    void *stream;
    bool operator==(const StreamKey &o) const { return device == o.device && stream == o.stream; }
};
struct StreamKeyHash {
    size_t operator()(const StreamKey &k) const { return std::hash<void *>()(k.stream) * 31 + k.device; }
};

// Buffers owned by the Python layer, one per (device, stream), remembered here; a larger one is asked for when needed.
// A remembered buffer stays valid: the Python layer never frees one it handed out.
struct BufferCache {
    std::mutex mutex;
    std::unordered_map<StreamKey, Tensor, StreamKeyHash> map;

    template <class Ask>
    Tensor get(const Tensor &like, size_t bytes, Ask ask) {
        const StreamKey key{(int)like.get_device(), stream()};
        {
            std::lock_guard<std::mutex> lock(mutex);
            auto it = map.find(key);
            if (it != map.end() && (size_t)it->second.nbytes() >= bytes) return it->second;
        }
        Tensor t = ask();
        if (capturing()) return t;                              // a graph's own memory
        std::lock_guard<std::mutex> lock(mutex);
        map[key] = t;
        return t;
    }
};
// never destroyed: at exit the allocator behind the tensors may be gone before them
BufferCache &g_workspaces = *new BufferCache, &g_scratch = *new BufferCache;

Tensor workspace(const Tensor &like, size_t bytes) {
    return g_workspaces.get(like, bytes, [&] { return lib_attr("workspace")(like.device(), bytes).cast<Tensor>(); });
}

Tensor decode_scratch(const Tensor &like, int64_t K, int64_t N) {
    Tensor t = g_scratch.get(like, (size_t)(K * N * 2), [&] {
        return py::module_::import("comp_inference_b200.pytorch_runtime").attr("_decode_scratch")(like.device(), K, N).cast<Tensor>().view({-1});
    });
    return t.narrow(0, 0, K * N).view({K, N});
}

// Entry points into the streams of tall tiles (ci_build_entry_points): every kEntryStep rows, the length of a half tile of
// the heights the kernels run best at.
constexpr int64_t kEntryStep = 64;
struct Entries {
    Tensor states, rows, spans;
    uint32_t cap = 0;
};

// Inference tensors have no version.
uint32_t version_of(const Tensor &t) {
    return t.is_inference() ? 0 : t.unsafeGetTensorImpl()->version_counter().current_version();
}

// The arrays of one compressed weight and its descriptor.
struct Weight {
    Tensor stream, states, tables, slot_map, offsets, lens, mantissa, lut;
    Entries entries;
    bool lasting = true;       // false: made under stream capture without what has to be derived first; not to be kept
    ci_tiled_weight w;
    // What it was made from: the tensors as they were given, where their data lay and which version it was.
    static constexpr int kArrays = 7;
    Tensor given[kArrays];
    const void *data[kArrays];
    uint32_t version[kArrays];

    void remember(std::initializer_list<Tensor> arrays) {
        int i = 0;
        for (const Tensor &t : arrays) {
            given[i] = t;
            data[i] = t.defined() ? t.data_ptr() : nullptr;
            version[i++] = t.defined() ? version_of(t) : 0;
        }
    }
    // Whether it still describes a module's buffers: none replaced, none moved, none written to.
    bool matches(const py::dict &buffers, int64_t th, int64_t tw) const {
        static PyObject *const names[kArrays] = {
            PyUnicode_InternFromString("rans_exp_stream"), PyUnicode_InternFromString("rans_exp_states"),
            PyUnicode_InternFromString("rans_exp_tables"), PyUnicode_InternFromString("rans_exp_slot_map"),
            PyUnicode_InternFromString("rans_exp_tile_offsets"), PyUnicode_InternFromString("rans_exp_tile_max_lens"),
            PyUnicode_InternFromString("rans_man_raw")};
        if ((uint32_t)th != w.tile_h || (uint32_t)tw != w.tile_w) return false;
        for (int i = 0; i < kArrays; ++i) {
            PyObject *o = PyDict_GetItem(buffers.ptr(), names[i]);
            if (o == nullptr || !THPVariable_Check(o)) return false;
            const Tensor &t = THPVariable_Unpack(o);
            if (!t.is_same(given[i]) || t.data_ptr() != data[i] || version_of(t) != version[i]) return false;
        }
        return true;
    }
};

Tensor as_u32(const Tensor &t, const char *name) {
    require_cuda(t, name);
    TORCH_CHECK(t.scalar_type() == at::kUInt32 || t.scalar_type() == at::kInt, name, " must be uint32 or int32, got torch.",
                t.scalar_type());
    return t.contiguous();
}
Tensor as_u8(const Tensor &t, const char *name) {
    require_cuda(t, name);
    TORCH_CHECK(t.scalar_type() == at::kByte, name, " must be uint8, got torch.", t.scalar_type());
    return t.contiguous();
}

void fill(Weight &h, int64_t K, int64_t N, int64_t th, int64_t tw, uint32_t max_len) {
    memset(&h.w, 0, sizeof h.w);
    h.w.stream = (const uint8_t *)h.stream.data_ptr();
    h.w.states = (const uint32_t *)h.states.data_ptr();
    h.w.tables = (const uint32_t *)h.tables.data_ptr();
    h.w.slot_map = (const uint8_t *)h.slot_map.data_ptr();
    h.w.tile_offsets = (const uint32_t *)h.offsets.data_ptr();
    h.w.tile_max_lens = (const uint32_t *)h.lens.data_ptr();
    h.w.mantissa = h.mantissa.defined() ? (const uint8_t *)h.mantissa.data_ptr() : nullptr;
    h.w.lut = h.lut.defined() ? (const uint32_t *)h.lut.data_ptr() : nullptr;
    h.w.stream_len = (uint64_t)h.stream.numel();
    h.w.K = (uint32_t)K;
    h.w.N = (uint32_t)N;
    h.w.tile_h = (uint32_t)th;
    h.w.tile_w = (uint32_t)tw;
    h.w.max_tile_len = max_len;
}

// What is derived from a weight's arrays is kept per tensor objects, as in the Python layer, and holds only for what it was made
// of: weak references, data pointers and versions tell.  A write that torch's version counter does not see (through .data, by
// another library, by a replayed graph) is not seen here either.  An entry stays until its tensors are gone or have changed: a
// captured graph may refer to it.
struct Ref {
    c10::weak_intrusive_ptr<c10::TensorImpl> impl;
    const void *data;
    uint32_t version;
    explicit Ref(const Tensor &t) : impl(t.getIntrusivePtr()), data(t.data_ptr()), version(version_of(t)) {}
    bool is(const Tensor &t) const {
        return !impl.expired() && impl._unsafe_get_target() == t.unsafeGetTensorImpl() && data == t.data_ptr() &&
               !t.is_inference() && version == version_of(t);
    }
};
// The decode table of tables and slot_map, the depth of the deepest tile, and the other arrays that came with them last.
struct Tables {
    Ref lens, tables, slot_map;
    Tensor lut;
    uint32_t max_len;
    std::optional<Ref> last[4] = {};
    // Whether all of h's arrays have come before as they are now.
    bool seen(const Weight &h) {
        const Tensor *arrays[4] = {&h.stream, &h.states, &h.offsets, &h.mantissa};
        bool all = true;
        for (int i = 0; i < 4; ++i) {
            if (!arrays[i]->defined() || (last[i] && last[i]->is(*arrays[i]))) continue;
            last[i].emplace(*arrays[i]);
            all = false;
        }
        return all;
    }
    bool is(const Weight &h) const { return lens.is(h.lens) && tables.is(h.tables) && slot_map.is(h.slot_map); }
    bool expired() const { return lens.impl.expired() || tables.impl.expired() || slot_map.impl.expired(); }
};
// The entry points of all of a weight's streams.
struct Index {
    Ref stream, states, tables, slot_map, offsets, lens;
    int64_t K, N, th;
    Entries entries;
    bool is(const Weight &h) const {
        return stream.is(h.stream) && states.is(h.states) && tables.is(h.tables) && slot_map.is(h.slot_map) &&
               offsets.is(h.offsets) && lens.is(h.lens) && K == h.w.K && N == h.w.N && th == h.w.tile_h;
    }
    bool expired() const {
        return stream.impl.expired() || states.impl.expired() || tables.impl.expired() || slot_map.impl.expired() ||
               offsets.impl.expired() || lens.impl.expired();
    }
};
// By the tensor that an entry begins with.
template <class T>
struct Derived {
    std::mutex mutex;
    std::unordered_map<const void *, T> map;

    // Calls use(entry) if there is one that holds for h.
    template <class Use>
    bool find(const Tensor &first, const Weight &h, Use use) {
        std::lock_guard<std::mutex> lock(mutex);
        auto it = map.find(first.unsafeGetTensorImpl());
        if (it == map.end() || !it->second.is(h)) return false;
        use(it->second);
        return true;
    }
    void keep(const Tensor &first, T entry) {
        std::lock_guard<std::mutex> lock(mutex);
        // what belongs to weights that are gone goes with the next new one
        for (auto it = map.begin(); it != map.end();) it = it->second.expired() ? map.erase(it) : std::next(it);
        map.insert_or_assign(first.unsafeGetTensorImpl(), std::move(entry));
    }
};
Derived<Tables> &g_tables = *new Derived<Tables>;               // by tile_max_lens
Derived<Index> &g_indexes = *new Derived<Index>;                // by the stream

Weight tiled(const Tensor &stream_t, const Tensor &states, const Tensor &tables, const Tensor &slot_map, const Tensor &offsets,
             const Tensor &lens, const OptTensor &mantissa, int64_t K, int64_t N, int64_t th, int64_t tw, bool entries) {
    Weight h;
    h.stream = as_u8(stream_t, "compressed stream");
    h.states = as_u32(states, "states");
    h.tables = as_u32(tables, "tables");
    h.slot_map = as_u8(slot_map, "slot_map");
    h.offsets = as_u32(offsets, "tile_offsets");
    h.lens = as_u32(lens, "tile_max_lens");
    if (mantissa.has_value()) h.mantissa = as_u8(*mantissa, "mantissas");
    h.remember({stream_t, states, tables, slot_map, offsets, lens, mantissa.has_value() ? *mantissa : Tensor()});
    if (th <= 0 || tw <= 0) throw py::value_error("tile sizes must be positive");
    const int64_t tiles = ((K + th - 1) / th) * ((N + tw - 1) / tw);
    if (h.states.numel() != tiles * 2 * tw)
        throw py::value_error("Initial states size mismatch. Expected " + std::to_string(tiles * 2 * tw));
    if (h.offsets.numel() != tiles || h.lens.numel() != tiles)
        throw py::value_error("tile_offsets / tile_max_lens must have " + std::to_string(tiles) + " entries");
    if (h.mantissa.defined() && h.mantissa.numel() < tiles * th * tw)
        throw py::value_error("mantissa plane has " + std::to_string(h.mantissa.numel()) + " bytes, " +
                              std::to_string(tiles * th * tw) + " expected");
    uint32_t max_len = 0;
    // a contiguous copy made above is a new object on every call: nothing to remember
    if (h.tables.is_same(tables) && h.slot_map.is_same(slot_map) && h.lens.is_same(lens)) {
        bool seen = false;
        const bool known = g_tables.find(lens, h, [&](Tables &t) {
            h.lut = t.lut;
            max_len = t.max_len;
            seen = t.seen(h);
        });
        if (known) {
            if (!seen) check(ci_weight_written(stream()));      // they may be the previous kernel's product
        } else if (capturing()) {
            h.lasting = false;                                  // the kernels that build the table themselves and need no depth
        } else {
            (void)tables._version(), (void)slot_map._version();  // inference tensors are refused: nobody counts their versions
            h.lut = at::empty({4096}, tables.options().dtype(at::kInt));
            check(ci_prepare_lut((const uint32_t *)tables.data_ptr(), (const uint8_t *)slot_map.data_ptr(),
                                 (uint32_t *)h.lut.data_ptr(), stream()));
            max_len = lib_attr("max_tile_len")(lens).cast<uint32_t>();
            c10::cuda::stream_synchronize(c10::cuda::getCurrentCUDAStream().stream());   // the next call may come on another one
            Tables t{Ref(lens), Ref(tables), Ref(slot_map), h.lut, max_len};
            t.seen(h);
            g_tables.keep(lens, std::move(t));
        }
    }
    fill(h, K, N, th, tw, max_len);
    // Entry points are worth their making only where they can be kept: not for copies, nor for inference tensors, whose
    // versions nobody counts.
    auto kept = [](const Tensor &mine, const Tensor &given) { return mine.is_same(given) && !given.is_inference(); };
    const bool tall = entries && h.lut.defined() && max_len != 0 && tw == 32 && th > 2 * kEntryStep && th % (2 * kEntryStep) == 0 &&
                      th <= 65536 && kept(h.stream, stream_t) && kept(h.states, states) && kept(h.offsets, offsets) &&
                      kept(h.lens, lens) && (reinterpret_cast<uintptr_t>(h.w.stream) & 15u) == 0 &&
                      (reinterpret_cast<uintptr_t>(h.w.states) & 15u) == 0;
    if (tall) {
        if (g_indexes.find(h.stream, h, [&](const Index &i) { h.entries = i.entries; })) {
        } else if (capturing()) {
            h.lasting = false;
        } else {
            Entries e;
            const int64_t n = tiles * (th / 2 / kEntryStep);
            e.states = at::empty({n * 64}, h.states.options());
            e.rows = at::empty({n * 64}, h.states.options().dtype(at::kShort));
            e.spans = at::empty({n}, h.states.options());
            Tensor cap = at::empty({1}, h.states.options().dtype(at::kInt));
            const int rc = ci_build_entry_points(&h.w, kEntryStep, (uint32_t *)e.states.data_ptr(), (uint16_t *)e.rows.data_ptr(),
                                                 (uint32_t *)e.spans.data_ptr(), (uint32_t *)cap.data_ptr(), stream());
            if (rc == CI_E_INVALID) {
                e = Entries();                                  // tiles too deep for the staged decoder's window: none
            } else {
                check(rc);
                e.cap = std::max<uint32_t>(1, (uint32_t)cap.item<int32_t>());
            }
            h.entries = e;
            g_indexes.keep(h.stream, Index{Ref(h.stream), Ref(h.states), Ref(h.tables), Ref(h.slot_map), Ref(h.offsets),
                                           Ref(h.lens), K, N, th, e});
        }
    }
    if (h.entries.states.defined()) {
        h.w.entry_step = kEntryStep;
        h.w.entry_states = (const uint32_t *)h.entries.states.data_ptr();
        h.w.entry_rows = (const uint16_t *)h.entries.rows.data_ptr();
        h.w.entry_spans = (const uint32_t *)h.entries.spans.data_ptr();
        h.w.entry_cap = h.entries.cap;
    }
    return h;
}

// Activations as rows of K bf16 with unit stride, without touching a tensor that already is that.
struct Rows {
    Tensor keep;
    const uint16_t *ptr;
    int64_t ld, M;
};
Rows rows_of(const Tensor &x, int64_t K) {
    TORCH_CHECK(x.scalar_type() == at::kBFloat16, "activations must be bfloat16, got torch.", x.scalar_type());
    require_cuda(x, "x");
    Rows r;
    if (x.dim() >= 1 && x.size(-1) == K && x.is_contiguous()) {
        r.keep = x;
        r.ld = K;
        r.M = x.numel() / K;
    } else {
        r.keep = x.reshape({-1, K});
        if (r.keep.stride(1) != 1) r.keep = r.keep.contiguous();
        r.ld = r.keep.stride(0);
        r.M = r.keep.size(0);
        if (r.M <= 1) r.ld = K;                                 // the stride of a single row means nothing
    }
    r.ptr = (const uint16_t *)r.keep.data_ptr();
    return r;
}

std::vector<int64_t> out_shape(const Tensor &x, int64_t n) {
    std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
    if (s.empty()) s.push_back(n); else s.back() = n;
    return s;
}

Tensor linear_call(const Weight &h, const Tensor &x, const OptTensor &bias, const OptTensor &out, int64_t split_k, bool transposed,
                   int64_t prefill_rows) {
    const int64_t K = transposed ? h.w.N : h.w.K, n_out = transposed ? h.w.K : h.w.N;
    const Rows r = rows_of(x, K);
    if (prefill_rows > 0 && r.M >= prefill_rows && !out.has_value()) {
        // many rows: one stand-alone decode into a reused buffer, then a library GEMM (see RansLinear)
        Tensor x2 = r.keep.dim() == 2 ? r.keep : r.keep.view({r.M, K});
        Tensor y;
        const int64_t rows = (h.w.K + 7) / 8 * 8, cols = (h.w.N + 7) / 8 * 8;
        if ((rows != h.w.K || cols != h.w.N) && h.w.tile_w == 32 && h.w.max_tile_len != 0) {
            // Odd sizes: the library has only slow kernels for operands whose rows are not 16-byte aligned (3.5 times
            // slower at 748 x 4873 x 13236), so the weight is decoded into padded rows and the activations are copied.
            Tensor w = decode_scratch(x, rows, cols);
            check(ci_decode_bf16_ld(&h.w, (uint16_t *)w.data_ptr(), cols, stream()));
            if (rows != h.w.K) w.narrow(0, h.w.K, rows - h.w.K).zero_();
            const int64_t Kp = transposed ? cols : rows;
            if (transposed && cols != K) w.narrow(1, K, cols - K).zero_();
            if (Kp != K || r.ld % 8) {
                Tensor xp = at::empty({r.M, Kp}, x.options());
                xp.narrow(1, 0, K).copy_(x2);
                if (Kp != K) xp.narrow(1, K, Kp - K).zero_();
                x2 = xp;
            }
            y = at::matmul(x2, transposed ? w.t() : w);
            if (y.size(1) != n_out) y = y.narrow(1, 0, n_out).contiguous();
        } else {
            Tensor w = decode_scratch(x, h.w.K, h.w.N);
            check(ci_decode_bf16(&h.w, (uint16_t *)w.data_ptr(), stream()));
            y = at::matmul(x2, transposed ? w.t() : w);
        }
        if (bias.has_value()) y.add_(*bias);
        return y.view(out_shape(x, n_out));
    }
    Tensor y;
    if (out.has_value()) {
        y = out->view({r.M, n_out});
        TORCH_CHECK(y.scalar_type() == at::kBFloat16 && y.stride(1) == 1, "out must be a bfloat16 tensor with unit inner stride");
    } else {
        y = at::empty(out_shape(x, n_out), x.options());
        TORCH_CHECK(y.numel() == r.M * n_out, "activations of ", x.sizes(), " do not have ", K, " columns");
    }
    const uint16_t *b = nullptr;
    Tensor keep_bias;
    if (bias.has_value()) {
        TORCH_CHECK(bias->scalar_type() == at::kBFloat16 && bias->numel() == n_out,
                    "bias must be bfloat16 with one entry per output feature");
        keep_bias = bias->contiguous();
        b = (const uint16_t *)keep_bias.data_ptr();
    }
    size_t bytes = ci_linear_workspace_bytes((uint32_t)r.M, (uint32_t)n_out, transposed ? 0 : h.w.K, h.w.tile_h);
    if (r.M > 16 && !transposed && split_k > 1)                 // an explicit split-K of the prefill GEMM: room for its partials
        bytes = std::max(bytes, (size_t)(1 << 14) + (size_t)std::min<int64_t>(split_k, 8) * r.M * n_out * 4);
    const Tensor ws = workspace(x, bytes);
    const int64_t ldy = out.has_value() ? y.stride(0) : n_out;
    check(transposed ? ci_linear_transposed(&h.w, r.ptr, r.ld, (uint32_t)r.M, b, (uint16_t *)y.data_ptr(), ldy, ws.data_ptr(),
                                            ws.nbytes(), stream())
                     : ci_linear(&h.w, r.ptr, r.ld, (uint32_t)r.M, b, (uint16_t *)y.data_ptr(), ldy, ws.data_ptr(), ws.nbytes(),
                                 (uint32_t)split_k, stream()));
    return out.has_value() ? *out : y;
}

Tensor embedding_call(const Weight &h, const Tensor &x, const OptTensor &out) {
    require_cuda(x, "x");
    const Tensor ids = x.to(at::kLong).contiguous();
    const int64_t n = ids.numel(), N = h.w.N;
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.push_back(N);
    Tensor o;
    int64_t ld = N;
    if (out.has_value()) {
        o = out->view({n, N});
        TORCH_CHECK(o.scalar_type() == at::kBFloat16 && (n == 0 || o.stride(1) == 1),
                    "out must be a bfloat16 tensor with unit inner stride");
        if (n > 0) ld = o.stride(0);
    } else {
        o = at::empty(shape, x.options().dtype(at::kBFloat16));
    }
    check(ci_embedding(&h.w, (const int64_t *)ids.data_ptr(), (uint64_t)n, (uint16_t *)o.data_ptr(), ld, stream()));
    return o.view(shape);
}

Tensor decode_call(const Weight &h, bool bf16) {
    Tensor o = at::empty({h.w.K, h.w.N}, h.stream.options().dtype(bf16 ? at::kBFloat16 : at::kByte));
    check(bf16 ? ci_decode_bf16(&h.w, (uint16_t *)o.data_ptr(), stream()) : ci_decode_plane(&h.w, (uint8_t *)o.data_ptr(), stream()));
    return o;
}

// bf16 [K,N] -> the package arrays of the one-pass encoder (32-wide tiles).  Returns (stream, states, sizes, tables,
// slot_map, offsets, max_lens, mantissas, freqs, cdf, man_hist or None); freqs, cdf, man_hist on the host.
py::tuple compress(const Tensor &w, int64_t th, int64_t tw, bool want_man_hist) {
    require_cuda(w, "weight");
    TORCH_CHECK(w.scalar_type() == at::kBFloat16 && w.dim() == 2 && w.is_contiguous(), "expected a contiguous 2-D bfloat16 tensor");
    const int64_t K = w.size(0), N = w.size(1), tiles = ((K + th - 1) / th) * ((N + tw - 1) / tw);
    const auto u8 = w.options().dtype(at::kByte), u32 = w.options().dtype(at::kUInt32);
    const auto u16 = at::TensorOptions().dtype(at::kUInt16);
    Tensor states = at::empty({tiles * 2 * tw}, u32), sizes = at::empty({tiles * 2 * tw}, u32), offsets = at::empty({tiles}, u32);
    Tensor lens = at::empty({tiles}, u32), tables = at::empty({256}, u32), slot_map = at::empty({4096}, u8);
    Tensor man = at::empty({tiles * th * tw}, u8), freqs = at::empty({256}, u16), cdf = at::empty({256}, u16), man_hist;
    if (want_man_hist) man_hist = at::empty({256}, at::TensorOptions().dtype(at::kLong));
    const size_t bytes = ci_compress_scratch_bytes((uint32_t)K, (uint32_t)N, (uint32_t)th, (uint32_t)tw);
    Tensor scratch = at::empty({(int64_t)bytes}, u8), stream_t;
    uint64_t n = 0;
    int rc;
    {
        py::gil_scoped_release release;                         // waits for the device
        rc = ci_compress_bf16((const uint16_t *)w.data_ptr(), (uint32_t)K, (uint32_t)N, (uint32_t)th, (uint32_t)tw,
                              (uint8_t *)man.data_ptr(), (uint32_t *)states.data_ptr(), (uint32_t *)sizes.data_ptr(),
                              (uint32_t *)offsets.data_ptr(), (uint32_t *)lens.data_ptr(), (uint32_t *)tables.data_ptr(),
                              (uint8_t *)slot_map.data_ptr(), scratch.data_ptr(), bytes, (uint16_t *)freqs.data_ptr(),
                              (uint16_t *)cdf.data_ptr(), want_man_hist ? (uint64_t *)man_hist.data_ptr() : nullptr, &n, stream());
    }
    check(rc);
    stream_t = at::empty({(int64_t)n}, u8);
    check(ci_compress_pack((uint32_t)K, (uint32_t)N, (uint32_t)th, (uint32_t)tw, (const uint32_t *)sizes.data_ptr(),
                           (const uint32_t *)offsets.data_ptr(), (const uint32_t *)lens.data_ptr(), scratch.data_ptr(), bytes,
                           (uint8_t *)stream_t.data_ptr(), n, stream()));
    return py::make_tuple(stream_t, states, sizes, tables, slot_map, offsets, lens, man, freqs, cdf,
                          want_man_hist ? py::cast(man_hist) : py::none());
}

// linear_of(weight, buffers, tile_h, tile_w, x, bias, split_k, prefill_rows): a module's call in one step, None where `buffers`
// are no longer what the descriptor was made from.  A plain C function: the binding layer's own argument handling costs a call as
// much as the allocation of its result.
PyObject *linear_of(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8) throw py::type_error("linear_of takes 8 arguments");
    const Weight &h = *py::cast<const Weight *>(py::handle(args[0]));
    TORCH_CHECK_TYPE(PyDict_Check(args[1]) && THPVariable_Check(args[4]), "linear_of needs a module's buffers and a tensor");
    long long v[4];
    for (int i = 0; i < 4; ++i) {
        v[i] = PyLong_AsLongLong(args[i < 2 ? 2 + i : 4 + i]);
        if (v[i] == -1 && PyErr_Occurred()) throw py::error_already_set();
    }
    if (!h.matches(py::reinterpret_borrow<py::dict>(args[1]), v[0], v[1])) Py_RETURN_NONE;
    OptTensor bias;
    if (args[5] != Py_None) {
        TORCH_CHECK_TYPE(THPVariable_Check(args[5]), "bias must be a tensor");
        bias = THPVariable_Unpack(args[5]);
    }
    return THPVariable_Wrap(linear_call(h, THPVariable_Unpack(args[4]), bias, std::nullopt, v[2], false, v[3]));
    END_HANDLE_TH_ERRORS
}
PyMethodDef fast_calls[] = {{"linear_of", (PyCFunction)(void (*)(void))linear_of, METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};

}  // namespace

PYBIND11_MODULE(_ci_host, m) {
    if (PyModule_AddFunctions(m.ptr(), fast_calls) != 0) throw py::error_already_set();
    py::class_<Weight>(m, "Weight", "Descriptor of a compressed weight and the tensors it points into")
        .def(py::init(&tiled), py::arg("stream"), py::arg("states"), py::arg("tables"), py::arg("slot_map"), py::arg("tile_offsets"),
             py::arg("tile_max_lens"), py::arg("mantissas"), py::arg("K"), py::arg("N"), py::arg("tile_h"), py::arg("tile_w"), py::arg("entries") = false)
        .def("matches", &Weight::matches)
        .def_readonly("lasting", &Weight::lasting)
        .def("route", [](const Weight &h, int64_t rows) {           // the kernel that linear runs (ci_linear_route), entry points included
            const int route = ci_linear_route(&h.w, (uint32_t)rows);
            if (route < 0) check(route);
            return route;
        })
        .def("linear", &linear_call, py::arg("x"), py::arg("bias") = py::none(), py::arg("out") = py::none(), py::arg("split_k") = 0,
             py::arg("transposed") = false, py::arg("prefill_rows") = 0)
        .def("embedding", &embedding_call, py::arg("x"), py::arg("out") = py::none())
        .def("decode", &decode_call, py::arg("bf16"));
    m.def("compress", &compress, py::arg("weight"), py::arg("tile_h"), py::arg("tile_w"), py::arg("want_man_hist"));
}
