// Launches of the decode kernel for five to eight query heads per KV head (tq_decode_g4.cuh, NH = 8).
#include "tq_decode_g4.cuh"

bool tq_decode_g8_try(const tqatt::AttnParams& P, const tqatt::SplitPlan& plan, const TqFast& fk, const TqFast& fv, cudaStream_t st, int* rc) {
  const int kf = P.L.k_format, vf = P.L.v_format;
  if (P.group > 8) return false;
  const bool w4 = four_warps(P, plan);
#define TQ_ATT_G8S(K, V)                                                                                   \
  if (P.sparse_v && kf == K && vf == V) {                                                                  \
    if (!layout_matches<K, V>(P.L)) return false;                                                          \
    if (w4) *rc = launch_attn_g4<K, V, true, false, 4, false, 8>(P, plan, fk, fv, st);                           \
    else *rc = launch_attn_g4<K, V, true, false, ATT_WARPS, false, 8>(P, plan, fk, fv, st);                      \
    return true;                                                                                           \
  }
  TQ_ATT_G8S(2, 2) TQ_ATT_G8S(2, 3) TQ_ATT_G8S(2, 4) TQ_ATT_G8S(3, 2) TQ_ATT_G8S(3, 3) TQ_ATT_G8S(3, 4) TQ_ATT_G8S(4, 2)
  TQ_ATT_G8S(4, 3) TQ_ATT_G8S(4, 4)
#undef TQ_ATT_G8S
  if (P.sparse_v) return false;   // q8_0 and PROD keys: the general kernel
#define TQ_ATT_G8(K, V)                                                                                    \
  if (kf == K && vf == V) {                                                                                \
    if (!layout_matches<K, V>(P.L)) return false;                                                          \
    /* where four CTAs with two page records each fit an SM */                                            \
    if constexpr (4 * (G4<K, V, 4, 8>::SMEM + 1024) <= 228 * 1024) {                                       \
      if (w4) {                                                                                            \
        if (P.tail_late) *rc = launch_attn_g4<K, V, false, false, 4, true, 8>(P, plan, fk, fv, st);              \
        else *rc = launch_attn_g4<K, V, false, false, 4, false, 8>(P, plan, fk, fv, st);                         \
        return true;                                                                                       \
      }                                                                                                    \
    }                                                                                                      \
    if (P.tail_late) *rc = launch_attn_g4<K, V, false, false, ATT_WARPS, true, 8>(P, plan, fk, fv, st);          \
    else *rc = launch_attn_g4<K, V, false, false, ATT_WARPS, false, 8>(P, plan, fk, fv, st);                     \
    return true;                                                                                           \
  }
  TQ_ATT_G8(2, 2) TQ_ATT_G8(2, 3) TQ_ATT_G8(2, 4) TQ_ATT_G8(3, 2) TQ_ATT_G8(3, 3) TQ_ATT_G8(3, 4) TQ_ATT_G8(4, 2)
  TQ_ATT_G8(4, 3) TQ_ATT_G8(4, 4)
  TQ_ATT_G8(8, 2) TQ_ATT_G8(8, 3) TQ_ATT_G8(8, 4) TQ_ATT_G8(8, 8)
  TQ_ATT_G8(18, 2) TQ_ATT_G8(18, 3) TQ_ATT_G8(19, 2) TQ_ATT_G8(19, 3) TQ_ATT_G8(19, 4) TQ_ATT_G8(20, 3) TQ_ATT_G8(20, 4)
#undef TQ_ATT_G8
  return false;
}
