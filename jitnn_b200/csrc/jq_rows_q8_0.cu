// The rows kernel's instances for Q8_0 weights.
#include "jq_rows_launch.cuh"

namespace jq {
namespace rows {

int launch_q8_0(Args& a, int ctas, bool after, cudaStream_t s) { return launch_format<JQ_TYPE_Q8_0>(a, ctas, after, s); }

}  // namespace rows
}  // namespace jq
