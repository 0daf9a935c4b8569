// The rows kernel's instance for Q5_K weights.
#include "jq_rows_launch.cuh"

namespace jq {
namespace rows {

int launch_q5_k(Args& a, int ctas, cudaStream_t s) { return launch_format<JQ_TYPE_Q5_K>(a, ctas, s); }

}  // namespace rows
}  // namespace jq
