#include "lbgb_march.cuh"

namespace lbgb {
template int launch_march<LBGB_F32>(const MarchCall &c, cudaStream_t s);
}
