// query_h4.cu -- the query kernels for 4 hash functions (see query.cuh).
#include "query.cuh"

namespace hibf_gb300
{

query_kernels const query_kernels_h4 = make_query_kernels<4>();

} // namespace hibf_gb300
