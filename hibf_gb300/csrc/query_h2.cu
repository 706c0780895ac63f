// query_h2.cu -- the query kernels for 2 hash functions (see query.cuh).
#include "query.cuh"

namespace hibf_gb300
{

query_kernels const query_kernels_h2 = make_query_kernels<2>();

} // namespace hibf_gb300
