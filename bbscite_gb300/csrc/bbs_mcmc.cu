// Persistent chain kernels of one dataset for one row width BBS_W (trees of
// up to 32 BBS_W nodes), with (BBS_REC 1) or without recorded moves and step
// traces.  The build compiles this unit once per row width and kind.
#include "bbs_launch.cuh"

namespace bbs {

template <int W, bool REC>
int launch_mcmc_w(const RunArgs &a, int q, bool sum, int cpb, int n_sms,
                  cudaStream_t s) {
#define BBS_CASE(QQ)                                                  \
  case QQ:                                                            \
    return sum ? launch_mcmc_t<W, QQ, true, REC>(a, cpb, n_sms, s)    \
               : launch_mcmc_t<W, QQ, false, REC>(a, cpb, n_sms, s);
  switch (q) {
    BBS_CASE(1)
    BBS_CASE(2)
#if BBS_W <= 4
    BBS_CASE(3)
    BBS_CASE(4)
#endif
    default: return (int)cudaErrorInvalidValue;
  }
#undef BBS_CASE
}

template int launch_mcmc_w<BBS_W, BBS_REC != 0>(const RunArgs &, int, bool,
                                                int, int, cudaStream_t);

}  // namespace bbs
