// The V-cycle with f32 storage and vectors.
#include "cycle.cuh"

template struct sf::Cycle<float, float>;
