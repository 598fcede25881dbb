// The channel-wise prepare kernels with 128 value channels (the source is gdn_cw_fwd.cu's).
#define LETHE_CW_FWD_V128
#include "gdn_cw_fwd.cu"
