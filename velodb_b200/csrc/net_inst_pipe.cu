// Instantiations of the network passes for the pipeline records: the join
// union records (2 words ordered on the whole of word 0) and the 16-bit key
// pairs of the filter + group-by, sorted (RowU2) and compacted (RowW).
#include "net_impl.cuh"

using JoinRec = velo::RowRec<2, 1, false, velo::KEY_FULL>;
VELO_INSTANTIATE_NET(JoinRec, 8, 4)
VELO_INSTANTIATE_NET(JoinRec, 8, 3)

VELO_INSTANTIATE_NET(velo::RowU2, 8, 3)
VELO_INSTANTIATE_NET(velo::RowU2, 8, 4)
VELO_INSTANTIATE_NET(velo::RowU2, 8, 5)
VELO_INSTANTIATE_NET(velo::RowW, 8, 4)
VELO_INSTANTIATE_NET(velo::RowW, 8, 5)

// generic group-by records (velo_ogroupby): key word plus 0 or 2 sum words
using GbRec1 = velo::RowRec<1, 1, false, velo::KEY_FULL>;
using GbRec3 = velo::RowRec<3, 1, false, velo::KEY_FULL>;
VELO_INSTANTIATE_NET(GbRec1, 8, 4)
VELO_INSTANTIATE_NET(GbRec1, 8, 3)
VELO_INSTANTIATE_NET(GbRec3, 8, 4)
VELO_INSTANTIATE_NET(GbRec3, 8, 3)
VELO_INSTANTIATE_NET(GbRec3, 9, 3)
