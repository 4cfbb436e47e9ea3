// tree_f32.cu -- the FP32 kernels of tree.cu.
#define TREE_F32 1
#include "tree.cu"
