// ft_fast_f32.cu -- the fast walk for float coordinates.
#include "ft_fast_type.cuh"

namespace ft {
FT_FAST_INSTANTIATE(float)
}
