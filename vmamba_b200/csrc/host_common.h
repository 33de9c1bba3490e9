// Shared parts of the host extension (_host.so): the torch side of libss2d_b200.so.
// Every function here only prepares arguments and launches; the kernels are behind the C interface of ss2d_b200.h.
#pragma once
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include "ss2d_b200.h"

namespace host {

using at::Tensor;
using OptT = std::optional<Tensor>;

// A status of the library, raised in Python as vmamba_b200._lib.Ss2dError(status, where).
struct LibError {
    int status;
    const char* where;
};
inline void check(int status, const char* where) {
    if (status != SS2D_OK) throw LibError{status, where};
}

inline int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return SS2D_F32;
        case at::kHalf: return SS2D_F16;
        case at::kBFloat16: return SS2D_BF16;
        default: TORCH_CHECK_TYPE(false, "unsupported dtype ", t, ": expected float32, float16 or bfloat16");
    }
}
inline int dtype_code(const Tensor& t) { return dtype_code(t.scalar_type()); }

inline void require_cuda(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        TORCH_CHECK(!t->defined() || t->is_cuda(),
                    "vmamba_b200 operators run on CUDA tensors only (no CPU fallback); use the oracle under oracle/ for CPU reference values");
}
// what library products between raw-pointer calls would have checked
inline void require_on(const Tensor& x, std::initializer_list<const Tensor*> ts) {
    require_cuda({&x});
    for (const Tensor* t : ts)
        TORCH_CHECK(!t->defined() || t->device() == x.device(), "expected all tensors on ", x.device(), ", got one on ", t->device());
}
inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
inline Tensor opt(const OptT& t) { return t.has_value() ? *t : Tensor(); }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline Tensor f32(const Tensor& t) {
    if (!t.defined() || (t.scalar_type() == at::kFloat && t.is_contiguous())) return t;
    return t.contiguous().to(at::kFloat);
}
inline Tensor rows(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
inline Tensor bytes(int64_t n, const Tensor& like) { return at::empty({n}, like.options().dtype(at::kByte)); }

// The caller's state as a call on raw pointers needs it: x's device, no autocast (a library product inside would return another
// type than the one whose code goes to the kernels behind it).
struct CallGuard {
    explicit CallGuard(const Tensor& x) : device(x.device()), no_autocast(c10::autocast_dispatch_keyset) {}
    c10::cuda::OptionalCUDAGuard device;
    c10::impl::ExcludeDispatchKeyGuard no_autocast;
};

// host_ops.cpp
std::pair<Tensor, Tensor> scan_fwd(Tensor u, Tensor delta, Tensor A, Tensor B, Tensor C, Tensor D, Tensor bias, bool softplus, bool out_float,
                                   int64_t every, Tensor out);
std::vector<Tensor> scan_bwd(Tensor u, Tensor delta, Tensor A, Tensor B, Tensor C, Tensor D, Tensor bias, Tensor dout, bool softplus, Tensor ckpt);
// the same with dB and dC (B, K, N, L) written into views of a larger tensor whose (image, group) blocks are evenly spaced
std::vector<Tensor> scan_bwd_into(Tensor u, Tensor delta, Tensor A, Tensor B, Tensor C, Tensor D, Tensor bias, Tensor dout, bool softplus, Tensor ckpt,
                                  Tensor dB, Tensor dC);
Tensor cross_scan(const Tensor& x, int64_t scans);       // (B, C, H, W) -> (B, 4, C, L)
Tensor cross_merge(const Tensor& ys, int64_t scans);     // (B, 4, C, H, W) -> (B, C, L)
int64_t scan_ratio(const Tensor& u, const Tensor& delta);

// host_core.cpp: CrossScan (op 0), CrossMerge (1), rows into (2) and out of (3) route order, rows of a route `stride` apart
Tensor cross(const Tensor& in, Tensor out, int64_t B, int64_t C, int64_t H, int64_t W, int64_t stride, int op);
int64_t padded_row(int64_t B, int64_t C, int64_t H, int64_t W);
bool rows_fit(int64_t H, int64_t W, int64_t esize);
// step sizes (B, 4, D, S) of rows in route order (B, 4, R + 2N, S); returns the B / C rows (B, 4, 2N, S)
Tensor expand_rows(const Tensor& xd, const Tensor& wdt, Tensor dts, int64_t B, int64_t D, int64_t R, int64_t N, int64_t S);

}  // namespace host
