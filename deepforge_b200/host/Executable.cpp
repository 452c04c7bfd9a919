// Runtime: variant-pack validation, then the kernel plan's launches through the dfgpu ABI.
//
// Validation order and error codes follow the reference's execute_variant
// (lib/Runtime/Executable.cpp:1023-1223): every argument UID present, non-null and
// aligned; no two argument byte ranges overlap when either is written; workspace
// non-null (when needed), 64-byte aligned and disjoint from every argument. All of these
// are DFE_INVALID_VARIANT_PACK. Extra UIDs in the pack and the handle are ignored.
// Pointers are device pointers: they are compared and offset, never dereferenced here.
#include "Internal.h"

#include <mutex>

namespace deepforge::runtime {

using compiler::KernelOp;
using compiler::KernelStep;
using compiler::TensorAccess;
using compiler::TensorBinding;
using import::ErrorCode;
using import::Status;

namespace {
// Where a launch finds one of its pointers: in the argument table, in the workspace, or nowhere (null).
struct Source {
    TensorBinding::Kind kind = TensorBinding::Kind::kAbsent;
    std::size_t at = 0;   // index into the argument table, or byte offset in the workspace
};
struct StepSources {
    std::vector<Source> tensors;
    Source scratch;
};

// A few values on the stack, more on the heap: a call binds fewer than ten pointers as a rule.
template <class T>
class Few {
public:
    explicit Few(std::size_t count) : data_(few_) {
        if (count > kFew) {
            many_.resize(count);
            data_ = many_.data();
        }
    }
    T& operator[](std::size_t i) { return data_[i]; }
    T* data() { return data_; }

private:
    static constexpr std::size_t kFew = 32;
    T few_[kFew];
    std::vector<T> many_;
    T* data_;
};
}  // namespace

struct Executable::Impl {
    compiler::GraphCompileMetadata metadata;
    compiler::WorkspacePlan workspace;
    compiler::KernelPlan plan;
    void* stream = nullptr;
    std::int64_t launches = 0;
    mutable std::mutex mutex;
    std::vector<StepSources> sources;   // of the plan's steps
};

std::string_view cpu_variant_name(CpuVariant variant) noexcept {
    switch (variant) {
        case CpuVariant::kScalar: return "scalar";
        case CpuVariant::kAvx2: return "avx2";
        case CpuVariant::kAvx512: return "avx512";
    }
    return "unknown";
}

Executable::Executable(std::unique_ptr<Impl> impl) : impl_(std::move(impl)) {}
Executable::~Executable() = default;
Executable::Executable(Executable&&) noexcept = default;
Executable& Executable::operator=(Executable&&) noexcept = default;

std::unique_ptr<Executable> ExecutableFactory::create(compiler::GraphCompileMetadata metadata, compiler::WorkspacePlan workspace,
                                                      compiler::KernelPlan plan) {
    auto impl = std::make_unique<Executable::Impl>();
    impl->metadata = std::move(metadata);
    impl->workspace = std::move(workspace);
    impl->plan = std::move(plan);
    auto const& arguments = impl->metadata.arguments;
    auto source = [&](TensorBinding const& binding) {
        Source out;
        if (binding.kind == TensorBinding::Kind::kWorkspace) out = {binding.kind, static_cast<std::size_t>(binding.offset)};
        if (binding.kind == TensorBinding::Kind::kArgument)
            for (std::size_t i = 0; i < arguments.size(); ++i)
                if (arguments[i].uid == binding.uid) out = {binding.kind, i};
        return out;
    };
    for (auto const& step : impl->plan.steps) {
        impl->launches += step.launches;
        StepSources sources;
        for (auto const& binding : step.tensors) sources.tensors.push_back(source(binding));
        sources.scratch = source(step.scratch);
        impl->sources.push_back(std::move(sources));
    }
    return std::unique_ptr<Executable>(new Executable(std::move(impl)));
}

std::int64_t Executable::get_workspace_size() const noexcept { return static_cast<std::int64_t>(impl_->workspace.size_bytes); }

Status Executable::get_workspace_size(std::int64_t& workspace_size) const {
    workspace_size = get_workspace_size();
    return Status::ok();
}

namespace {
Status reject_overrides(OverrideUids const& uids, OverrideShapes const& shapes, OverrideStrides const& strides) {
    if (uids.empty() && shapes.empty() && strides.empty()) return Status::ok();
    return Status::failure(ErrorCode::kInvalidVariantPack, "override", "the graph was compiled without shape overrides");
}
}  // namespace

Status Executable::get_workspace_size(FrontendHandle, std::int64_t& workspace_size, OverrideUids const& uids, OverrideShapes const& shapes,
                                      OverrideStrides const& strides) const {
    auto status = reject_overrides(uids, shapes, strides);
    if (status.is_bad()) return status;
    return get_workspace_size(workspace_size);
}

std::int64_t Executable::get_workspace_size(FrontendHandle, OverrideUids const& uids, OverrideShapes const& shapes, OverrideStrides const& strides) const {
    return reject_overrides(uids, shapes, strides).is_good() ? get_workspace_size() : -1;
}

bool Executable::supports_variant(CpuVariant variant) const noexcept { return variant == CpuVariant::kScalar; }
CpuVariant Executable::selected_variant() const noexcept { return CpuVariant::kScalar; }
void Executable::set_stream(void* stream) noexcept {
    std::lock_guard<std::mutex> lock(impl_->mutex);
    impl_->stream = stream;
}

Status Executable::execute_on(void* stream, VariantPack& pack, void* workspace) const {
    return run_steps(0, static_cast<std::int64_t>(impl_->plan.steps.size()), pack, workspace, stream, true);
}
std::int64_t Executable::launch_count() const noexcept { return impl_->launches; }
std::string Executable::plan_text() const { return impl_->plan.to_text(); }

Status Executable::execute(FrontendHandle handle, VariantPack& pack, void* workspace) const {
    return execute_variant(CpuVariant::kScalar, handle, pack, workspace);
}

Status Executable::execute(FrontendHandle handle, VariantPack& pack, void* workspace, OverrideUids const& uids, OverrideShapes const& shapes,
                           OverrideStrides const& strides) const {
    return execute_variant(CpuVariant::kScalar, handle, pack, workspace, uids, shapes, strides);
}

Status Executable::execute_variant(CpuVariant variant, FrontendHandle handle, VariantPack& pack, void* workspace, OverrideUids const& uids,
                                   OverrideShapes const& shapes, OverrideStrides const& strides) const {
    auto status = reject_overrides(uids, shapes, strides);
    if (status.is_bad()) return status;
    return execute_variant(variant, handle, pack, workspace);
}

Status Executable::execute_variant(CpuVariant variant, FrontendHandle, VariantPack& pack, void* workspace) const {
    if (!supports_variant(variant))
        return Status::failure(ErrorCode::kUnsupportedCpuFeature, cpu_variant_name(variant), "this executable carries one sm_100a kernel plan; use the scalar variant name");
    return execute_steps(0, static_cast<std::int64_t>(impl_->plan.steps.size()), pack, workspace);
}

Status Executable::execute_steps(std::int64_t first, std::int64_t last, VariantPack& pack, void* workspace) const {
    return run_steps(first, last, pack, workspace, nullptr, false);
}

Status Executable::run_steps(std::int64_t first, std::int64_t last, VariantPack& pack, void* workspace, void* call_stream, bool own_stream) const {
    auto find = [&](std::int64_t uid, void*& pointer) {
        auto it = pack.find(uid);
        if (it == pack.end()) return false;
        pointer = it->second;
        return true;
    };
    return run(first, last, find, workspace, call_stream, own_stream);
}

Status Executable::execute_list(std::int64_t const* uids, void* const* list, std::size_t count, void* workspace, void* call_stream, bool own_stream) const {
    auto const steps = static_cast<std::int64_t>(impl_->plan.steps.size());
    constexpr std::size_t kFewEntries = 32;   // (above, a map beats the scan)
    if (count > kFewEntries) {
        VariantPack pack;
        pack.reserve(count);
        for (std::size_t i = 0; i < count; ++i) pack[uids[i]] = list[i];
        return run_steps(0, steps, pack, workspace, call_stream, own_stream);
    }
    auto find = [&](std::int64_t uid, void*& pointer) {
        for (std::size_t at = count; at > 0; --at)   // from the end: the last entry of a UID counts, as in a map
            if (uids[at - 1] == uid) {
                pointer = list[at - 1];
                return true;
            }
        return false;
    };
    return run(0, steps, find, workspace, call_stream, own_stream);
}

template <class Find>
Status Executable::run(std::int64_t first, std::int64_t last, Find const& find, void* workspace, void* call_stream, bool own_stream) const {
    auto const& impl = *impl_;
    if (first < 0 || last > static_cast<std::int64_t>(impl.plan.steps.size()) || first > last)
        return Status::failure(ErrorCode::kInvalidArgument, "steps", "step range is outside the kernel plan");

    struct Range {
        std::uintptr_t begin, end;
        bool written;
    };
    auto const& arguments = impl.metadata.arguments;
    auto const count = arguments.size();
    Few<void*> bound(count);
    Few<Range> ranges(count);
    for (std::size_t i = 0; i < count; ++i) {
        auto const& argument = arguments[i];
        if (!find(argument.uid, bound[i]))
            return Status::failure(ErrorCode::kInvalidVariantPack, argument.name, "UID " + std::to_string(argument.uid) + " is missing from the variant pack");
        if (bound[i] == nullptr) return Status::failure(ErrorCode::kInvalidVariantPack, argument.name, "pointer is null");
        auto address = reinterpret_cast<std::uintptr_t>(bound[i]);
        if (address % argument.alignment != 0) return Status::failure(ErrorCode::kInvalidVariantPack, argument.name, "pointer is not aligned to " + std::to_string(argument.alignment) + " bytes");
        ranges[i] = {address, address + argument.size_bytes, argument.access != TensorAccess::kRead};
    }
    for (std::size_t i = 0; i < count; ++i)
        for (std::size_t j = i + 1; j < count; ++j)
            if ((ranges[i].written || ranges[j].written) && ranges[i].begin < ranges[j].end && ranges[j].begin < ranges[i].end)
                return Status::failure(ErrorCode::kInvalidVariantPack, arguments[i].name, "storage overlaps '" + arguments[j].name + "' and at least one of them is written");
    auto const workspace_bytes = impl.workspace.size_bytes;
    if (workspace_bytes != 0) {
        if (workspace == nullptr) return Status::failure(ErrorCode::kInvalidVariantPack, "workspace", "pointer is null but " + std::to_string(workspace_bytes) + " bytes are required");
        auto address = reinterpret_cast<std::uintptr_t>(workspace);
        if (address % compiler::kWorkspaceAlignment != 0) return Status::failure(ErrorCode::kInvalidVariantPack, "workspace", "pointer is not aligned to 64 bytes");
        for (std::size_t i = 0; i < count; ++i)
            if (address < ranges[i].end && ranges[i].begin < address + workspace_bytes)
                return Status::failure(ErrorCode::kInvalidVariantPack, "workspace", "storage overlaps '" + arguments[i].name + "'");
    }

    // The plan is immutable and the launchers keep no state between calls, so a call with its own stream needs no
    // lock; calls on the shared stream take it, so that the launches of one plan stay together on that stream.
    std::unique_lock<std::mutex> lock(impl.mutex, std::defer_lock);
    void* stream = call_stream;
    if (!own_stream) {
        lock.lock();
        stream = impl.stream;
    }
    auto resolve = [&](Source const& source) -> void* {
        switch (source.kind) {
            case TensorBinding::Kind::kArgument: return bound[source.at];
            case TensorBinding::Kind::kWorkspace: return static_cast<char*>(workspace) + source.at;
            default: return nullptr;
        }
    };
    for (std::int64_t index = first; index < last; ++index) {
        auto const& step = impl.plan.steps[static_cast<std::size_t>(index)];
        auto const& sources = impl.sources[static_cast<std::size_t>(index)];
        Few<void*> pointers(sources.tensors.size());
        for (std::size_t i = 0; i < sources.tensors.size(); ++i) pointers[i] = resolve(sources.tensors[i]);
        void* scratch = resolve(sources.scratch);
        int code = 0;
        switch (step.op) {
            case KernelOp::kBlockScaleQuantize: code = dfgpu_block_scale_quantize(&std::get<dfgpu_bsq_params>(step.params), pointers.data(), scratch, stream); break;
            case KernelOp::kBlockScaleDequantize: code = dfgpu_block_scale_dequantize(&std::get<dfgpu_bsd_params>(step.params), pointers.data(), scratch, stream); break;
            case KernelOp::kConstants: code = dfgpu_constants(&std::get<dfgpu_constants_params>(step.params), pointers.data(), scratch, stream); break;
            case KernelOp::kPointwise: code = dfgpu_pointwise(&std::get<dfgpu_pointwise_params>(step.params), pointers.data(), scratch, stream); break;
            case KernelOp::kConvFprop: {
                // bit 1 of `reserved` (set by the lowering) promises that the kernel launched just before this one is the
                // plan's previous step; that does not hold for the first launch of a call
                dfgpu_conv_params params = std::get<dfgpu_conv_params>(step.params);
                if (index == first) params.reserved &= ~2;
                code = dfgpu_conv_fprop(&params, pointers.data(), scratch, stream);
                break;
            }
            case KernelOp::kMatmul: code = dfgpu_matmul(&std::get<dfgpu_matmul_params>(step.params), pointers.data(), scratch, stream); break;
            case KernelOp::kSdpaForward: code = dfgpu_sdpa_forward(&std::get<dfgpu_sdpa_params>(step.params), pointers.data(), scratch, stream); break;
            case KernelOp::kMatmulFp8: code = dfgpu_matmul_fp8(&std::get<dfgpu_matmul_fp8_params>(step.params), pointers.data(), scratch, stream); break;
            case KernelOp::kBlockScaleQuantizePair: code = dfgpu_block_scale_quantize_pair(&std::get<dfgpu_bsq_pair_params>(step.params), pointers.data(), scratch, stream); break;
            case KernelOp::kConvFpropPair: {
                dfgpu_conv_pair_params params = std::get<dfgpu_conv_pair_params>(step.params);
                if (index == first) params.first.reserved &= ~2;  // see kConvFprop above
                code = dfgpu_conv_fprop_pair(&params, pointers.data(), scratch, stream);
                break;
            }
        }
        if (code != 0) {
            auto mapped = code == 19 ? ErrorCode::kGraphExecutionFailed : static_cast<ErrorCode>(code);
            return Status::failure(mapped, step.label, dfgpu_last_error());
        }
    }
    return Status::ok();
}

}  // namespace deepforge::runtime
