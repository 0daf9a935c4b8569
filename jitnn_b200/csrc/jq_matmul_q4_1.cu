// The matrix kernel's instances for Q4_1 weights.
#include "jq_matmul_launch.cuh"

namespace jq {
namespace mm {

int launch_q4_1(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s) { return launch_format<JQ_TYPE_Q4_1>(plan, args, map, s); }

}  // namespace mm
}  // namespace jq
