// One MoE MLP layer call on one GPU: bucketing, local scatter, the two expert products with the activation
// between them, and the score-weighted gather -- and the backward of the whole -- as ONE host call each.
//
// The device work is that of the single operators (fmoe_count_and_pos, fmoe_local_scatter, fmoe_linear_*,
// fmoe_combine_*, fmoe_local_gather_sum), queued in the same order on the same stream.  What this saves is
// host time: a layer of a few hundred tokens was bound by the Python between its launches.  The buffers come
// from the caller in two pieces per direction, laid out here.
#include "common.cuh"
#include <algorithm>

using namespace fmoe;

namespace {

constexpr size_t kAlign = 256;
size_t up(size_t n) { return (n + kAlign - 1) / kAlign * kAlign; }

// Piece of a caller-provided buffer.
struct Carver {
    char* base;
    size_t at = 0;
    void* take(size_t bytes) {
        void* p = base ? base + at : nullptr;
        at += up(bytes);
        return p;
    }
};

struct Layout {
    int64_t rows, d, h;
    size_t row_d, row_h;
    explicit Layout(const fmoe_moe_mlp_t& a)
        : rows(a.n_tokens * a.top_k), d(a.d_model), h(a.d_hidden), row_d((size_t)(a.d_model * dtype_size(a.dtype))),
          row_h((size_t)(a.d_hidden * dtype_size(a.dtype))) {}
};

struct Index {   // what the backward needs of the routing
    int64_t *offsets, *pos, *inv;
    size_t bytes;
    Index(const fmoe_moe_mlp_t& a, void* base) {
        Carver c{(char*)base};
        const size_t n = (size_t)(a.n_tokens * a.top_k) * 8;
        offsets = (int64_t*)c.take((size_t)(a.n_expert + 1) * 8);
        pos = (int64_t*)c.take(n);
        inv = (int64_t*)c.take(n);
        bytes = c.at;
    }
};

// Forward buffers.  keep: they are read again by the backward; otherwise the experts' output reuses the rows
// of their input, and no activation derivative is stored.
struct Rows {
    void *x, *h, *pre, *y;
    size_t bytes;
    Rows(const fmoe_moe_mlp_t& a, void* base) {
        const Layout l(a);
        Carver c{(char*)base};
        x = c.take(l.rows * l.row_d);
        h = c.take(l.rows * l.row_h);
        pre = a.keep && saves_derivative(a.activation) ? c.take(l.rows * l.row_h) : nullptr;
        y = a.keep ? c.take(l.rows * l.row_d) : x;
        bytes = c.at;
    }
};

// Backward buffers: gradients of the experts' output (then, once nothing reads it any more, of their input) and
// of their hidden activations, and the scratch of the products.
struct Grads {
    void *y, *h, *scratch;
    size_t bytes;
    Grads(const fmoe_moe_mlp_t& a, void* base) {
        const Layout l(a);
        Carver c{(char*)base};
        y = c.take(l.rows * l.row_d);
        h = c.take(l.rows * l.row_h);
        scratch = c.take(std::max(fmoe_linear_scratch_bytes(l.rows, l.h, l.d, a.n_expert, a.dtype),
                                  fmoe_linear_scratch_bytes(l.rows, l.d, l.h, a.n_expert, a.dtype)));
        bytes = c.at;
    }
};

int check_args(const fmoe_moe_mlp_t* a) {
    FMOE_REQUIRE(a != nullptr, "moe_mlp: null argument block");
    FMOE_REQUIRE(a->n_tokens > 0 && a->top_k > 0 && a->d_model > 0 && a->d_hidden > 0 && a->n_expert > 0,
                 "moe_mlp: bad sizes tokens=%lld top_k=%d d_model=%lld d_hidden=%lld experts=%d", (long long)a->n_tokens,
                 a->top_k, (long long)a->d_model, (long long)a->d_hidden, a->n_expert);
    FMOE_REQUIRE(dtype_size(a->dtype) != 0, "moe_mlp: unknown dtype %d", a->dtype);
    FMOE_REQUIRE(a->w1 && a->w2 && a->score && a->index && a->rows, "moe_mlp: null pointer");
    return 0;
}

}  // namespace

extern "C" int fmoe_moe_mlp_bytes(const fmoe_moe_mlp_t* a, int64_t* index_bytes, int64_t* row_bytes, int64_t* grad_bytes) {
    FMOE_REQUIRE(a && index_bytes && row_bytes && grad_bytes, "moe_mlp_bytes: null pointer");
    FMOE_REQUIRE(a->n_tokens > 0 && a->top_k > 0 && a->d_model > 0 && a->d_hidden > 0 && a->n_expert > 0 &&
                 dtype_size(a->dtype) != 0, "moe_mlp_bytes: bad sizes");
    // the routing scratch is dead once the experts run: it shares the row buffers
    const size_t scratch = fmoe_routing_scratch_bytes(a->n_tokens * a->top_k, a->n_expert);
    *index_bytes = (int64_t)Index(*a, nullptr).bytes;
    *row_bytes = (int64_t)std::max(Rows(*a, nullptr).bytes, scratch);
    *grad_bytes = (int64_t)Grads(*a, nullptr).bytes;
    return 0;
}

extern "C" int fmoe_moe_mlp_forward(const fmoe_moe_mlp_t* a, fmoe_stream_t st) {
    if (int rc = check_args(a)) return rc;
    FMOE_REQUIRE(a->inp && a->gate_idx && a->out, "moe_mlp_forward: null pointer");
    const Layout l(*a);
    const Index ix(*a, a->index);
    const Rows r(*a, a->rows);
    if (int rc = fmoe_count_and_pos(a->gate_idx, l.rows, a->n_expert, nullptr, ix.offsets, ix.pos, ix.inv, a->rows, st)) return rc;
    if (int rc = fmoe_local_scatter(a->inp, ix.pos, r.x, l.rows, a->n_tokens, (int64_t)l.row_d, a->top_k, st)) return rc;
    if (int rc = fmoe_linear_forward(r.x, a->w1, a->b1, ix.offsets, r.h, r.pre, l.rows, l.d, l.h, a->n_expert, a->dtype,
                                     a->activation, st)) return rc;
    if (int rc = fmoe_linear_forward(r.h, a->w2, a->b2, ix.offsets, r.y, nullptr, l.rows, l.h, l.d, a->n_expert, a->dtype,
                                     FMOE_ACT_NONE, st)) return rc;
    return fmoe_combine_forward(r.y, ix.inv, a->score, a->out, a->n_tokens, a->top_k, l.d, a->dtype, st);
}

extern "C" int fmoe_moe_mlp_backward(const fmoe_moe_mlp_t* a, fmoe_stream_t st) {
    if (int rc = check_args(a)) return rc;
    FMOE_REQUIRE(a->keep, "moe_mlp_backward: the forward kept nothing");
    FMOE_REQUIRE(a->grad_out && (!a->gw1 || (a->gw2 && a->grads)), "moe_mlp_backward: null pointer");
    FMOE_REQUIRE(!a->grad_inp || a->gw1, "moe_mlp_backward: the input gradient comes with the weight gradients");
    const Layout l(*a);
    const Index ix(*a, a->index);
    const Rows r(*a, a->rows);
    const Grads g(*a, a->grads);
    void* grad_y = a->gw1 ? g.y : nullptr;
    if (grad_y || a->grad_score) {
        if (int rc = fmoe_combine_backward(a->grad_out, r.y, ix.inv, a->score, grad_y, a->grad_score, a->n_tokens, a->top_k,
                                           l.d, a->dtype, st)) return rc;
    }
    if (!grad_y) return 0;
    const void* act_pre = a->activation == FMOE_ACT_NONE ? nullptr : r.pre ? r.pre : r.h;
    // the first layer's bias gradient is the column sum of the hidden gradient, which that product returns
    if (int rc = fmoe_linear_backward_colsum(g.y, r.h, a->w2, ix.offsets, act_pre, g.h, a->gw2, a->gb2, a->gb1, l.rows, l.h, l.d,
                                             a->n_expert, a->dtype, a->activation, 0, g.scratch, st)) return rc;
    if (int rc = fmoe_linear_backward(g.h, r.x, a->w1, ix.offsets, nullptr, a->grad_inp ? g.y : nullptr, a->gw1, nullptr, l.rows,
                                      l.d, l.h, a->n_expert, a->dtype, FMOE_ACT_NONE, 0, g.scratch, st)) return rc;
    if (!a->grad_inp) return 0;
    return fmoe_local_gather_sum(g.y, ix.inv, a->grad_inp, a->n_tokens, a->top_k, l.d, a->dtype, st);
}
