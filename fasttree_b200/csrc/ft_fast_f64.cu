// ft_fast_f64.cu -- the fast walk for double coordinates.
#include "ft_fast_type.cuh"

namespace ft {
FT_FAST_INSTANTIATE(double)
}
