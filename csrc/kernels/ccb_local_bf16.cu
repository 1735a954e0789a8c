#include "ccb_local_table.cuh"

template const void* ccb::local_kernel<__nv_bfloat16>(const ccb::LocalKey&);
