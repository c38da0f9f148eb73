// Instantiations of the network passes for RowKP (tile configurations of the
// autotuner, and the small tiles of sorts of up to 1024 rows).
#include "net_impl.cuh"

VELO_INSTANTIATE_NET(velo::RowKP, 8, 3)
VELO_INSTANTIATE_NET(velo::RowKP, 9, 2)
VELO_INSTANTIATE_NET(velo::RowKP, 10, 1)
VELO_INSTANTIATE_NET(velo::RowKP, 6, 3)
VELO_INSTANTIATE_NET(velo::RowKP, 7, 3)
