// FP64 and mixed paths: whole runs of 1D steps in one persistent launch.
#define JB_NS fast
#define JB_FAST 1
#define JB_NS_NAME "fp64"
#define JB_OPS_NAME fast_ops
#define JB_PART JB_PART_RUN
#include "jb_variant.inc"
