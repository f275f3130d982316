// Work-list kernels for many datasets in one launch, for one row width BBS_W
// (trees of up to 32 BBS_W nodes), with one-warp chains or (BBS_MULTI 1)
// chains of several warps.  The build compiles this unit once per row width
// and kind.
#include "bbs_launch.cuh"

namespace bbs {

template <int W, bool MULTI>
int launch_batch_w(const BatchArgs &b, int q, bool sum, int wpb, int n_sms,
                   cudaStream_t s) {
#define BBS_CASE(QQ)                                                   \
  case QQ:                                                             \
    return sum ? launch_batch_t<W, QQ, true, MULTI>(b, wpb, n_sms, s)  \
               : launch_batch_t<W, QQ, false, MULTI>(b, wpb, n_sms, s);
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

template int launch_batch_w<BBS_W, BBS_MULTI != 0>(const BatchArgs &, int,
                                                   bool, int, int,
                                                   cudaStream_t);

}  // namespace bbs
