#include "ccb_local_table.cuh"

template const void* ccb::local_kernel<__half>(const ccb::LocalKey&);
