// ft_fast_u32.cu -- the fast walk for uint32_t coordinates.
#include "ft_fast_type.cuh"

namespace ft {
FT_FAST_INSTANTIATE(uint32_t)
}
