// One decode step of a DeepSeek attention layer (archive/ktransformers/operators/attention.py:349-478, decode branch) as one host call: the projections on GGUF blocks, the
// norms, rotations and the cache write, the absorb products and the attention over the latent cache.  The launches are those of the calls it makes; what it saves is the
// host work between them, which bound the layer: called one by one from Python a token took 200 us.
#include "handles.cuh"

using namespace ktb;

static size_t step_up(size_t n) { return (n + 255) / 256 * 256; }

extern "C" {

size_t ktb200_latent_step_bytes(int batch, int heads, int nope_dim, int v_dim, int q_rank) {
    if (batch <= 0 || heads <= 0 || nope_dim <= 0 || v_dim <= 0 || q_rank < 0) return 0;
    const size_t B = batch, H = heads;
    return 2 * step_up(B * q_rank * 2) + step_up(B * H * (nope_dim + 64) * 2) + step_up(B * 576 * 2) + step_up(B * H * 64 * 2) + 2 * step_up(B * H * 512 * 2) + step_up(B * H * v_dim * 2);
}

int ktb200_latent_step(const ktb200_latent_step_params* p, void* stream) {
    if (!p || !p->x || !p->out || !p->scratch || !p->q_a || !p->kv_a || !p->o || (p->q_rank > 0 && (!p->q_b || !p->q_norm))) { set_error("latent_step: null pointer"); return KTB200_EINVAL; }
    if (p->batch <= 0) return KTB200_OK;
    if (p->heads <= 0 || p->nope_dim <= 0 || p->v_dim <= 0 || p->q_rank < 0 || p->scratch_bytes < ktb200_latent_step_bytes(p->batch, p->heads, p->nope_dim, p->v_dim, p->q_rank) ||
        ((uintptr_t)p->scratch & 255)) {
        set_error("latent_step: bad shape, scratch too small or not aligned to 256 bytes");
        return KTB200_EINVAL;
    }
    // a linear writes rows of its own size and type: they have to be the scratch's
    const int q_out = p->heads * (p->nope_dim + 64), hidden = p->kv_a->in_size, device = p->kv_a->device;
    auto suits = [&](const char* name, const ktb200_linear* l, int in, int out) -> int {
        if (!l->loaded) { set_error("latent_step: %s: Not Loaded", name); return KTB200_ESTATE; }
        if (l->in_size == in && (l->out_size == out || out == 0) && l->hidden_type == KTB200_TYPE_BF16 && l->device == device) return KTB200_OK;
        set_error("latent_step: %s is %d -> %d, type %d, device %d; expected %d -> %d in bf16 on device %d", name, l->in_size, l->out_size, l->hidden_type, l->device, in, out, device);
        return KTB200_EINVAL;
    };
    int rc = suits("q_a", p->q_a, hidden, p->q_rank > 0 ? p->q_rank : q_out);
    if (rc == KTB200_OK && p->q_rank > 0) rc = suits("q_b", p->q_b, p->q_rank, q_out);
    if (rc == KTB200_OK) rc = suits("kv_a", p->kv_a, hidden, 576);
    if (rc == KTB200_OK) rc = suits("o", p->o, p->heads * p->v_dim, 0);      // (its rows go to `out`)
    if (rc != KTB200_OK) return rc;
    const size_t B = p->batch, H = p->heads;
    uint8_t* at = reinterpret_cast<uint8_t*>(p->scratch);
    auto take = [&](size_t n) { uint8_t* q = at; at += step_up(n); return q; };
    void *qa = take(B * p->q_rank * 2), *qn = take(B * p->q_rank * 2), *q = take(B * H * (p->nope_dim + 64) * 2), *kva = take(B * 576 * 2), *q_pe = take(B * H * 64 * 2);
    void *q_abs = take(B * H * 512 * 2), *lat = take(B * H * 512 * 2), *o = take(B * H * p->v_dim * 2);
    if (p->q_rank > 0) {
        rc = ktb200_linear_forward(p->q_a, p->batch, p->x, qa, p->q_a_bias, nullptr, stream);
        if (rc == KTB200_OK) rc = ktb200_add_rmsnorm(qa, nullptr, p->q_norm, p->q_eps, qn, p->batch, p->q_rank, stream);
        if (rc == KTB200_OK) rc = ktb200_linear_forward(p->q_b, p->batch, qn, q, p->q_b_bias, nullptr, stream);
    } else {
        rc = ktb200_linear_forward(p->q_a, p->batch, p->x, q, p->q_a_bias, nullptr, stream);
    }
    if (rc == KTB200_OK) rc = ktb200_linear_forward(p->kv_a, p->batch, p->x, kva, p->kv_a_bias, nullptr, stream);
    if (rc == KTB200_OK)
        rc = ktb200_mla_step_prep(q, p->heads, p->nope_dim, kva, p->kv_norm, p->kv_eps, p->inv_freq, p->positions, p->position_stride, p->cache_position, p->kv_cache, p->page_size,
                                  p->max_pages, q_pe, p->kv_len, p->batch, stream);
    if (rc == KTB200_OK) rc = ktb200_mla_absorb_q(q, p->nope_dim + 64, (long)p->heads * (p->nope_dim + 64), p->w_uk, p->heads, p->nope_dim, 512, q_abs, p->batch, stream);
    if (rc == KTB200_OK) {
        ktb200_mla_params m{};
        m.batch = p->batch; m.num_heads = p->heads; m.page_size = p->page_size; m.max_pages_per_seq = p->table_pages; m.sm_scale = p->sm_scale;
        m.q_nope = q_abs; m.q_pe = q_pe; m.kv_cache = p->kv_cache; m.page_table = p->page_table; m.kv_len = p->kv_len; m.out = lat;
        m.workspace = p->workspace; m.workspace_bytes = p->workspace_bytes;
        rc = ktb200_mla_decode(&m, stream);
    }
    if (rc == KTB200_OK) rc = ktb200_mla_absorb_o(lat, p->w_uv, p->heads, p->v_dim, 512, o, p->batch, stream);
    if (rc == KTB200_OK) rc = ktb200_linear_forward(p->o, p->batch, o, p->out, p->o_bias, nullptr, stream);
    return rc;
}

}  // extern "C"
