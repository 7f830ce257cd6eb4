// cov_map_low.cu -- the map kernels for up to five layers.
#define COV_MAP_KERNELS
#include "cov_map.cuh"

void map_kernels_3(int q, MapLow *low, MapHigh *high) { map_kernels_rc<3>(q, low, high); }
void map_kernels_5(int q, MapLow *low, MapHigh *high) { map_kernels_rc<5>(q, low, high); }
