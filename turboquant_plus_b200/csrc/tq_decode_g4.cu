// Launches of the decode kernel for at most four query heads per KV head (tq_decode_g4.cuh).
#include "tq_decode_g4.cuh"

bool tq_decode_g4_try(const tqatt::AttnParams& P, const tqatt::SplitPlan& plan, const TqFast& fk, const TqFast& fv, cudaStream_t st, int* rc) {
  const int kf = P.L.k_format, vf = P.L.v_format;
  const bool w4 = four_warps(P, plan);
  // PolarQuant K and V: every pair of widths, with the sparse-V and the measurement variants
#define TQ_ATT_G4(K, V)                                                                                              \
  if (kf == K && vf == V) {                                                                                          \
    if (!layout_matches<K, V>(P.L)) return false;                                                                    \
    if (P.nodeq && K == 3 && V == 3) *rc = launch_attn_g4<3, 3, false, true>(P, plan, fk, fv, st);                         \
    else if (P.sparse_v && w4) *rc = launch_attn_g4<K, V, true, false, 4>(P, plan, fk, fv, st);                         \
    else if (P.sparse_v) *rc = launch_attn_g4<K, V, true, false>(P, plan, fk, fv, st);                                     \
    else if (P.tail_late && w4) *rc = launch_attn_g4<K, V, false, false, 4, true>(P, plan, fk, fv, st);                   \
    else if (P.tail_late) *rc = launch_attn_g4<K, V, false, false, ATT_WARPS, true>(P, plan, fk, fv, st);                  \
    else if (w4) *rc = launch_attn_g4<K, V, false, false, 4>(P, plan, fk, fv, st);                                      \
    else *rc = launch_attn_g4<K, V, false, false>(P, plan, fk, fv, st);                                                    \
    return true;                                                                                                     \
  }
  TQ_ATT_G4(2, 2) TQ_ATT_G4(2, 3) TQ_ATT_G4(2, 4) TQ_ATT_G4(3, 2) TQ_ATT_G4(3, 3) TQ_ATT_G4(3, 4) TQ_ATT_G4(4, 2)
  TQ_ATT_G4(4, 3) TQ_ATT_G4(4, 4)
#undef TQ_ATT_G4
  // q8_0 and PROD keys (the sparse-V option of these pairs runs the general kernel)
  if (P.sparse_v) return false;
#define TQ_ATT_G4X(K, V)                                                                                   \
  if (kf == K && vf == V) {                                                                                \
    if (!layout_matches<K, V>(P.L)) return false;                                                          \
    /* the four-warp form where four CTAs with two page records each fit an SM */                         \
    if constexpr (4 * (G4<K, V, 4>::SMEM + 1024) <= 228 * 1024) {                                          \
      if (w4) {                                                                                            \
        if (P.tail_late) *rc = launch_attn_g4<K, V, false, false, 4, true>(P, plan, fk, fv, st);                 \
        else *rc = launch_attn_g4<K, V, false, false, 4>(P, plan, fk, fv, st);                                   \
        return true;                                                                                       \
      }                                                                                                    \
    }                                                                                                      \
    if (P.tail_late) *rc = launch_attn_g4<K, V, false, false, ATT_WARPS, true>(P, plan, fk, fv, st);             \
    else *rc = launch_attn_g4<K, V, false, false>(P, plan, fk, fv, st);                                          \
    return true;                                                                                           \
  }
  TQ_ATT_G4X(8, 2) TQ_ATT_G4X(8, 3) TQ_ATT_G4X(8, 4) TQ_ATT_G4X(8, 8)
  TQ_ATT_G4X(18, 2) TQ_ATT_G4X(18, 3) TQ_ATT_G4X(19, 2) TQ_ATT_G4X(19, 3) TQ_ATT_G4X(19, 4) TQ_ATT_G4X(20, 3) TQ_ATT_G4X(20, 4)
#undef TQ_ATT_G4X
  return false;
}
