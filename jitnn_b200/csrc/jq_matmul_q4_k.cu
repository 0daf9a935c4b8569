// The matrix kernel's instances for Q4_K weights.
#include "jq_matmul_launch.cuh"

namespace jq {
namespace mm {

int launch_q4_k(const Plan& plan, const Args& args, const CUtensorMap& map, cudaStream_t s) { return launch_format<JQ_TYPE_Q4_K>(plan, args, map, s); }

}  // namespace mm
}  // namespace jq
