// k_tree_f32.cu -- the box-tree search (tree_search.cuh) for float data.
#include <algorithm>

#include "tree_search.cuh"

namespace knnsj {

template void launch_tree_search<float>(const TreeLaunch<float>&, int, cudaStream_t);

}  // namespace knnsj
