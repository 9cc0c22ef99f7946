#include "lbgb_march.cuh"

namespace lbgb {
template int launch_march<LBGB_BF16DEV>(const MarchCall &c, cudaStream_t s);
}
