#include "ccb_local_table.cuh"

template const void* ccb::local_kernel<float>(const ccb::LocalKey&);
