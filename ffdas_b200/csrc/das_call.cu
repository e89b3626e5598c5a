// das_call.cu -- ffdas_das_call / ffdas_das_backward_call: a whole call from one
// packed argument array (the Python binding spends about a microsecond per
// separate native call and descriptor; a small frame takes 3 us on the GPU).
#include <cstring>

#include "core.h"
#include "das_problem.h"

namespace {

// Reads the packed values in order; `ok` turns false past the end.
struct reader {
    const int64_t *q;
    int64_t n, i = 0;
    bool ok = true;
    int64_t next() {
        if (i >= n) {
            ok = false;
            return 0;
        }
        return q[i++];
    }
    template <typename T> T *ptr() { return reinterpret_cast<T *>(static_cast<uintptr_t>(next())); }
    float real() {
        const int64_t bits = next();
        double d;
        std::memcpy(&d, &bits, sizeof(d));
        return (float)d;
    }
};

// x: ndim and four padded dims and strides.
ffdas_error_t read_x(reader &r, ffdas_tensor_desc &d) {
    d.dtype = (ffdas_datatype_t)r.next();
    d.ndim = r.next();
    for (int k = 0; k < 4; k++) d.dims[k] = r.next();
    for (int k = 0; k < 4; k++) d.strides[k] = r.next();
    if (!r.ok || d.ndim < 1 || d.ndim > 4) return FFDAS_ERROR_INVALID_ARGUMENT;
    return ffdas_type_size(d.dtype) ? FFDAS_SUCCESS : FFDAS_ERROR_UNSUPPORTED_TYPE;
}

// an image: ndim, dims, strides at the end of the array
ffdas_error_t read_image(reader &r, ffdas_tensor_desc &d) {
    d.ndim = r.next();
    if (!r.ok || d.ndim < 1) return FFDAS_ERROR_INVALID_ARGUMENT;
    if (d.ndim > FFDAS_MAX_DIMS) return FFDAS_ERROR_DIMS_TOO_LARGE;
    for (int64_t k = 0; k < d.ndim; k++) d.dims[k] = r.next();
    for (int64_t k = 0; k < d.ndim; k++) d.strides[k] = r.next();
    if (!r.ok) return FFDAS_ERROR_INVALID_ARGUMENT;
    return ffdas_type_size(d.dtype) ? FFDAS_SUCCESS : FFDAS_ERROR_UNSUPPORTED_TYPE;
}

// A forward call unpacked; its descriptors stay here.
struct forward_args {
    ffdas_handle_t h = nullptr;
    uintptr_t stream = 0;
    ffdas_tensor_desc xd, od;
    ffdas::das_call a;
    const float *scale = nullptr;
    int64_t scale_count = 0;
    void *pairs = nullptr;
    size_t pair_bytes = 0;

    ffdas_error_t read(const int64_t *q, int64_t n) {
        if (!q) return FFDAS_ERROR_NULL_POINTER;
        reader r{q, n};
        h = r.ptr<ffdas_context>();
        if (!h) return FFDAS_ERROR_INVALID_HANDLE;
        stream = (uintptr_t)r.next();
        a.srcpos = r.ptr<const float>();
        a.srcdir = r.ptr<const float>();
        a.wavenum = r.real();
        a.x = r.ptr<const void>();
        FFDAS_TRY(read_x(r, xd));
        a.dstpos = r.ptr<const float>();
        a.offsets = r.ptr<const float>();
        a.weights = r.ptr<const float>();
        a.sparse_count = (int)r.next();
        a.sparse_indices = r.ptr<const int>();
        a.out = r.ptr<void>();
        od.dtype = (ffdas_datatype_t)r.next();
        a.compute_type = (ffdas_compute_type_t)r.next();
        a.alg = (ffdas_alg_t)r.next();
        scale = r.ptr<const float>();
        scale_count = r.next();
        pairs = r.ptr<void>();
        pair_bytes = (size_t)r.next();
        a.sparse = r.next() != 0;
        FFDAS_TRY(read_image(r, od));
        a.x_desc = &xd;
        a.out_desc = &od;
        return FFDAS_SUCCESS;
    }
};

}  // namespace

extern "C" {

ffdas_error_t ffdas_das_call(const int64_t *q, int64_t n) {
    forward_args f;
    FFDAS_TRY(f.read(q, n));
    const ffdas::das_call &a = f.a;
    FFDAS_TRY(ffdas_set_stream(f.h, f.stream));
    if (f.scale) FFDAS_TRY(ffdas_set_channel_scale(f.h, f.scale, f.scale_count));
    ffdas_error_t e = f.pairs ? ffdas_set_pair_buffer(f.h, f.pairs, f.pair_bytes) : FFDAS_SUCCESS;
    if (e == FFDAS_SUCCESS)
        e = a.sparse ? ffdas_das_sparse(f.h, a.srcpos, a.srcdir, a.wavenum, &f.xd, a.x, a.dstpos, a.offsets, a.weights,
                                        a.sparse_count, a.sparse_indices, nullptr, &f.od, a.out, a.compute_type, a.alg)
                     : ffdas_das(f.h, a.srcpos, a.srcdir, a.wavenum, &f.xd, a.x, a.dstpos, a.offsets, a.weights, nullptr,
                                 &f.od, a.out, a.compute_type, a.alg);
    if (f.pairs) ffdas_set_pair_buffer(f.h, nullptr, 0);
    if (f.scale) ffdas_set_channel_scale(f.h, nullptr, 0);
    return e;
}

ffdas_error_t ffdas_das_call_pair_bytes(const int64_t *q, int64_t n, size_t *bytes) {
    if (!bytes) return FFDAS_ERROR_NULL_POINTER;
    forward_args f;
    FFDAS_TRY(f.read(q, n));
    return ffdas::kept_pair_bytes(*f.h, f.a, f.scale || f.h->chan_scale, bytes);
}

ffdas_error_t ffdas_das_backward_call(const int64_t *q, int64_t n) {
    if (!q) return FFDAS_ERROR_NULL_POINTER;
    reader r{q, n};
    ffdas_handle_t h = r.ptr<ffdas_context>();
    if (!h) return FFDAS_ERROR_INVALID_HANDLE;
    const uintptr_t stream = (uintptr_t)r.next();
    const float *srcpos = r.ptr<const float>(), *srcdir = r.ptr<const float>();
    const float wavenum = r.real();
    const void *x = r.ptr<const void>();
    ffdas_tensor_desc xd, gd;
    FFDAS_TRY(read_x(r, xd));
    const float *dstpos = r.ptr<const float>(), *offsets = r.ptr<const float>(), *weights = r.ptr<const float>();
    const int count = (int)r.next();
    const int *idx = r.ptr<const int>();
    const void *gout = r.ptr<const void>();
    gd.dtype = (ffdas_datatype_t)r.next();
    float *gx = r.ptr<float>(), *goff = r.ptr<float>(), *gw = r.ptr<float>(), *gdst = r.ptr<float>(), *gsrc = r.ptr<float>();
    void *pairs = r.ptr<void>();
    const size_t pair_bytes = (size_t)r.next();
    FFDAS_TRY(read_image(r, gd));
    FFDAS_TRY(ffdas_set_stream(h, stream));
    if (pairs) FFDAS_TRY(ffdas_set_pair_buffer(h, pairs, pair_bytes));
    const ffdas_error_t e = ffdas_das_backward(h, srcpos, srcdir, wavenum, &xd, x, dstpos, offsets, weights, count, idx, &gd,
                                               gout, gx, goff, gw, gdst, gsrc);
    if (pairs) ffdas_set_pair_buffer(h, nullptr, 0);
    return e;
}

}  // extern "C"
