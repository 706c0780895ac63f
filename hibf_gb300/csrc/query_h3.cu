// query_h3.cu -- the query kernels for 3 hash functions (see query.cuh).
#include "query.cuh"

namespace hibf_gb300
{

query_kernels const query_kernels_h3 = make_query_kernels<3>();

} // namespace hibf_gb300
