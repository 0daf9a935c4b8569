// The matrix kernel's instances for Q6_K weights.
#include "jq_matmul_launch.cuh"

namespace jq {
namespace mm {

int launch_q6_k(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s) { return launch_format<JQ_TYPE_Q6_K>(plan, args, map, s); }

}  // namespace mm
}  // namespace jq
