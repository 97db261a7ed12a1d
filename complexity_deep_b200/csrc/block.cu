// One decoder block of a prompt as one call: the launches of cd_complexity_block in order, each through its own entry
// point, whose checks and choice of kernel stay where they are.
//
// Host code only. A block is nine or ten launches, and a caller that makes them one by one from Python spends 19 us on
// each (arguments, checks, an output tensor), more than the kernels of a small model take: 150M-class, a prompt of 37
// tokens, 12 layers: kernels 0.54 ms, pass 2.31 ms; through this call the pass takes 1.32 ms, 4 us a launch of them the driver's.
#include "../../include/cdeep.h"

extern "C" int cd_complexity_block(const cd_block* p, void* stream) {
  if (!p || p->B < 1 || p->S < 1 || p->H < 8 || p->hq < 1 || p->hkv < 1 || p->E < 1 || p->I < 8 || p->I_s < 8) return CD_ERR_INVALID;
  if (static_cast<long long>(p->B) * p->S > 0x7fffffffLL) return CD_ERR_INVALID;
  if (!cd_attention_prefill_supported(p->B, p->S, p->hq, p->hkv, p->D)) return CD_ERR_UNSUPPORTED;
  const int T = p->B * p->S, N = (p->hq + 2 * p->hkv) * p->D;
  int e = cd_rmsnorm_split(p->x, p->x_lo, p->ln1, p->eps1, p->normed, nullptr, T, p->H, stream);
  if (e != CD_OK) return e;
  if (cd_mu_qkv_rope_supported(T, N, p->hq, p->hkv, p->D)) {
    e = cd_mu_qkv_rope(p->normed, p->mu, p->w_qkv, p->w_mu, p->qkv, T, p->H, N, p->q_norm, p->k_norm, p->cos_t, p->sin_t,
                       p->eps_qk, p->S, 0, p->hq, p->hkv, p->D, stream);
  } else {
    e = cd_mu_qkv(p->normed, p->mu, p->w_qkv, p->w_mu, p->qkv, T, p->H, N, stream);
    if (e == CD_OK)
      e = cd_qk_norm_rope(p->qkv, p->q_norm, p->k_norm, p->cos_t, p->sin_t, p->eps_qk, T, p->S, 0, p->hq, p->hkv, p->D, stream);
  }
  if (e == CD_OK) e = cd_attention_prefill(p->qkv, p->attn, p->B, p->S, p->hq, p->hkv, p->D, p->scale, stream);
  if (e == CD_OK) e = cd_linear(p->attn, p->w_o, p->x, p->x_lo, p->h1, p->h1_lo, T, p->hq * p->D, p->H, stream);
  if (e == CD_OK) e = cd_rmsnorm_split(p->h1, p->h1_lo, p->ln2, p->eps2, p->x_sorted, p->inv_perm, T, p->H, stream);
  if (e != CD_OK) return e;
  if (p->bn == p->bn_s || T <= 64) {   // one launch for both; up to 64 rows stream the weights whatever the layouts
    e = cd_moe_up_pair_layouts(p->x_sorted, p->offsets, p->E, p->w_up, p->h_r, p->I, p->bn, p->w_up_s, p->h_s, p->I_s, p->bn_s, T,
                               p->H, stream);
  } else {
    e = cd_moe_up(p->x_sorted, p->offsets, p->E, p->w_up, p->h_r, T, p->H, p->I, p->bn, stream);
    if (e == CD_OK) e = cd_moe_up(p->x_sorted, nullptr, 1, p->w_up_s, p->h_s, T, p->H, p->I_s, p->bn_s, stream);
  }
  if (e == CD_OK)
    e = cd_moe_down(p->h_r, p->I, p->w_down, p->h_s, p->I_s, p->w_down_s, p->offsets, p->E, p->perm, p->h1, p->h1_lo, p->out,
                    p->out_lo, T, p->H, stream);
  if (e == CD_OK)
    e = cd_mu_proj(p->out, p->w_mu_proj, p->mu_param, p->mu_min, p->mu_max, 1, p->clamp_lo, p->clamp_hi, p->mu_out, T, p->H, stream);
  return e;
}
