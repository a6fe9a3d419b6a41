// ws_sor_tags.h — the exchange tags of the region solve (ws_sor_tb.cu), as
// plain C so that the rule can be checked on the host.
#pragma once
#ifdef __CUDACC__
#define WS_TAG_FN static __host__ __device__ __forceinline__
#else
#define WS_TAG_FN static inline
#endif
// The tag base after a solve that started from tag0, as CTA 0 leaves it: no
// word of that solve may carry a tag that a later one waits for. A solve that
// ended ran the same epochs in every CTA. In one that a timed-out wait ended,
// CTAs far from the stuck one are ahead of CTA 0 by an unknown number of
// epochs, and an epoch holds one iteration at least.
WS_TAG_FN unsigned tb_next_tag_base(unsigned tag0, unsigned epochs, int aborted, int iters) {
  return tag0 + 1u + (aborted ? (unsigned)(iters > 0 ? iters : 0) : epochs);
}
