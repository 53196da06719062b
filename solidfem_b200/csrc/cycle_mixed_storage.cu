// The V-cycle with f32 storage, f64 vectors.
#include "cycle.cuh"

template struct sf::Cycle<float, double>;
