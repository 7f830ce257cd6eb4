// cov_map_high.cu -- the map kernels for six to nine layers.
#define COV_MAP_KERNELS
#include "cov_map.cuh"

void map_kernels_7(int q, MapLow *low, MapHigh *high) { map_kernels_rc<7>(q, low, high); }
void map_kernels_9(int q, MapLow *low, MapHigh *high) { map_kernels_rc<9>(q, low, high); }
