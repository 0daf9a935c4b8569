// The rows kernel's instances for Q4_1 weights.
#include "jq_rows_launch.cuh"

namespace jq {
namespace rows {

int launch_q4_1(Args& a, int ctas, bool after, cudaStream_t s) { return launch_format<JQ_TYPE_Q4_1>(a, ctas, after, s); }

}  // namespace rows
}  // namespace jq
