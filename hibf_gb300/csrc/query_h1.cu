// query_h1.cu -- the query kernels for 1 hash function (see query.cuh).
#include "query.cuh"

namespace hibf_gb300
{

query_kernels const query_kernels_h1 = make_query_kernels<1>();

} // namespace hibf_gb300
