// ft_fast_u64.cu -- the fast walk for unsigned long long coordinates.
#include "ft_fast_type.cuh"

namespace ft {
FT_FAST_INSTANTIATE(unsigned long long)
}
