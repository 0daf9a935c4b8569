// The matrix kernel's instances for Q4_0 weights.
#include "jq_matmul_launch.cuh"

namespace jq {
namespace mm {

int launch_q4_0(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s) { return launch_format<JQ_TYPE_Q4_0>(plan, args, map, s); }

}  // namespace mm
}  // namespace jq
