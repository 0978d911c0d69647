// A whole forward and a whole backward call as one entry point each: the stages of ssd_b200.h in order, with their
// internal buffers carved out of one caller-allocated workspace.  A small call is bound by the host, not by the GPU (one
// tile forward: 22 us of kernels in 48 us; with backward 50 in 235), and a foreign call with a score of arguments per stage, an
// allocation per buffer and a stream look-up were a good part of that: one tile forward 48 -> 33 us, with backward
// 235 -> 216 us (most of the rest is the framework's autograd engine).
#include "ssd_host.h"
#include "ssd_tile.cuh"

namespace ssd {

namespace {

// Workspace layout: buffers one after the other, each on a 256-byte boundary.
struct Carver {
    unsigned char* base;
    size_t used = 0;
    template <class T>
    T* take(size_t count) {
        T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
        used += (count * sizeof(T) + 255) & ~size_t(255);
        return p;
    }
};

struct ForwardWork {
    float *q, *cs, *states;
    size_t bytes;
    ForwardWork(const SsdShape& s, void* base) {
        Carver c{static_cast<unsigned char*>(base)};
        const size_t rows = static_cast<size_t>(s.batch) * s.nheads;
        q = c.take<float>(rows * s.seqlen);
        cs = c.take<float>(rows * s.seqlen);
        states = c.take<float>(rows * (s.seqlen / kTile) * kStateRows * state_cols(s));
        bytes = c.used;
    }
};

struct BackwardWork {
    float *dstates, *g_last, *ddt_t, *dy, *gate_part, *dbc_part;
    double* dA_part;
    int split;
    size_t bytes;
    BackwardWork(const SsdShape& s, bool has_d, bool has_z, void* base) {
        Carver c{static_cast<unsigned char*>(base)};
        const size_t rows = static_cast<size_t>(s.batch) * s.nheads, tiles = rows * (s.seqlen / kTile);
        const size_t tokens = static_cast<size_t>(s.batch) * row_tokens(s);
        dstates = c.take<float>(tiles * kStateRows * state_cols(s));
        g_last = c.take<float>(tiles * (state_cols(s) / 64));
        ddt_t = c.take<float>(rows * s.seqlen);
        dA_part = c.take<double>(tiles);
        dy = has_z ? c.take<float>(tokens * s.nheads * s.headdim) : nullptr;
        gate_part = has_d ? c.take<float>(ssd_gate_partial_floats(&s)) : nullptr;
        split = ssd_dbc_split(&s);
        dbc_part = split > 1 ? c.take<float>(2 * tokens * s.ngroups * s.dstate * split) : nullptr;
        bytes = c.used;
    }
};

int run_states(const SsdShape& s, const float* x, const float* m, const float* q, const float* cs, const float* start,
               float* states, float* end, int mode, int route, int* status, ssd_stream_t st) {
    if (ssd_use_state_scan(&s, route)) return ssd_chunk_state_scan(&s, x, m, q, cs, start, states, end, mode, status, st);
    const int rc = ssd_chunk_state(&s, x, m, q, cs, states, mode, status, st);
    if (rc != SSD_OK) return rc;
    return mode == 0 ? ssd_state_passing_fwd(&s, states, cs, start, end, st)
                     : ssd_state_passing_bwd(&s, states, nullptr, cs, start, nullptr, end, st);
}

}  // namespace

}  // namespace ssd

// The fused state kernel has batch * ngroups CTAs and takes the place of two launches where that is at least 1.5 x the SM
// count ([8,4096,256,64], 512 chains: 0.80 ms against 1.03 ms for the pair; [8,4096,32,64], 64 chains: the pair is
// faster, 0.13 against 0.19 ms).
extern "C" int ssd_use_state_scan(const SsdShape* shape, int state_route) {
    if (state_route == 2 || !ssd_chunk_state_scan_supported(shape)) return 0;
    return state_route == 1 || 2ll * shape->batch * shape->ngroups >= 3ll * ssd::sm_count() ? 1 : 0;
}

extern "C" size_t ssd_forward_work_bytes(const SsdShape* shape) {
    if (ssd_check_shape(shape) != SSD_OK) return 0;
    return ssd::ForwardWork(*shape, nullptr).bytes;
}

extern "C" size_t ssd_backward_work_bytes(const SsdShape* shape, int has_d, int has_z) {
    if (ssd_check_shape(shape) != SSD_OK) return 0;
    return ssd::BackwardWork(*shape, has_d != 0, has_z != 0, nullptr).bytes;
}

extern "C" int ssd_forward(const SsdShape* shape, const SsdForwardArgs* a, int state_route, ssd_stream_t stream) {
    using namespace ssd;
    int rc = ssd_check_shape(shape);
    if (rc != SSD_OK) return rc;
    if (!a || !a->x || !a->dt || !a->A || !a->bm || !a->cm || !a->y || !a->work || !a->status) return SSD_ERR_NULL;
    const bool gated = a->D != nullptr || a->z != nullptr;
    if (gated && !a->out) return SSD_ERR_NULL;
    const SsdShape& s = *shape;
    const ForwardWork w(s, a->work);
    rc = ssd_dt_cumsum(&s, a->dt, a->dt_bias, a->A, w.q, w.cs, stream);
    if (rc == SSD_OK)
        rc = run_states(s, a->x, a->bm, w.q, w.cs, a->initial_state, w.states, a->final_state, 0, state_route, a->status,
                        stream);
    if (rc == SSD_OK)
        rc = ssd_chunk_scan_copy_fwd(&s, a->x, a->bm, a->cm, w.states, w.q, w.cs, a->y, gated ? nullptr : a->out, a->status,
                                     stream);
    if (rc != SSD_OK || !gated) return rc;
    return ssd_gate_skip_fwd(&s, a->y, a->x, a->D, a->D ? a->d_mode : 0, a->z, a->out, stream);
}

extern "C" int ssd_backward(const SsdShape* shape, const SsdBackwardArgs* a, int state_route, ssd_stream_t stream) {
    using namespace ssd;
    int rc = ssd_check_shape(shape);
    if (rc != SSD_OK) return rc;
    if (!a || !a->x || !a->dt || !a->A || !a->bm || !a->cm || !a->y || !a->dout || !a->forward_work || !a->work ||
        !a->dx || !a->ddt || !a->dA || !a->dB || !a->dC || !a->status)
        return SSD_ERR_NULL;
    const SsdShape& s = *shape;
    const ForwardWork f(s, const_cast<void*>(a->forward_work));
    const BackwardWork w(s, a->D != nullptr, a->z != nullptr, a->work);
    const int d_mode = a->D ? a->d_mode : 0;
    const float* dy = a->dout;
    if (a->D != nullptr || a->z != nullptr) {
        rc = ssd_gate_skip_bwd(&s, a->dout, a->y, a->x, a->D, d_mode, a->z, w.dy, a->dz, w.gate_part, a->dD, stream);
        if (rc != SSD_OK) return rc;
        if (a->z != nullptr) dy = w.dy;
    }
    rc = run_states(s, dy, a->cm, f.q, f.cs, a->dfinal, w.dstates, a->d_initial, 1, state_route, a->status, stream);
    if (rc == SSD_OK)
        rc = ssd_chunk_dbc_split_bwd(&s, a->x, a->bm, a->cm, dy, f.states, w.dstates, f.q, f.cs, a->dB, a->dC, w.g_last,
                                     w.split, w.dbc_part, a->status, stream);
    if (rc == SSD_OK)
        rc = ssd_chunk_dx_bwd(&s, a->x, a->bm, a->cm, dy, a->y, w.dstates, f.q, f.cs, a->dt, a->dt_bias, a->A, w.g_last,
                              a->dx, w.ddt_t, w.dA_part, a->D, d_mode, a->status, stream);
    if (rc == SSD_OK) rc = ssd_dt_finalize_bias_bwd(&s, w.ddt_t, w.dA_part, a->ddt, a->dA, a->d_dt_bias, stream);
    return rc;
}
