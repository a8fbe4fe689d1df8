// k_tree_f64.cu -- the box-tree search (tree_search.cuh) for double data.
#include <algorithm>

#include "tree_search.cuh"

namespace knnsj {

template void launch_tree_search<double>(const TreeLaunch<double>&, int, cudaStream_t);

}  // namespace knnsj
