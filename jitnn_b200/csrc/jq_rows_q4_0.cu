// The rows kernel's instances for Q4_0 weights.
#include "jq_rows_launch.cuh"

namespace jq {
namespace rows {

int launch_q4_0(Args& a, int ctas, bool after, cudaStream_t s) { return launch_format<JQ_TYPE_Q4_0>(a, ctas, after, s); }

}  // namespace rows
}  // namespace jq
