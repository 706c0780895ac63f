// query_h5.cu -- the query kernels for 5 hash functions (see query.cuh).
#include "query.cuh"

namespace hibf_gb300
{

query_kernels const query_kernels_h5 = make_query_kernels<5>();

} // namespace hibf_gb300
