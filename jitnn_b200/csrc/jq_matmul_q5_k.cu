// The matrix kernel's instances for Q5_K weights.
#include "jq_matmul_launch.cuh"

namespace jq {
namespace mm {

int launch_q5_k(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s) { return launch_format<JQ_TYPE_Q5_K>(plan, args, map, s); }

}  // namespace mm
}  // namespace jq
