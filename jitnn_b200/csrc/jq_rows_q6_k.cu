// The rows kernel's instances for Q6_K weights.
#include "jq_rows_launch.cuh"

namespace jq {
namespace rows {

int launch_q6_k(Args& a, int ctas, bool after, cudaStream_t s) { return launch_format<JQ_TYPE_Q6_K>(a, ctas, after, s); }

}  // namespace rows
}  // namespace jq
