// The V-cycle with f64 throughout.
#include "cycle.cuh"

template struct sf::Cycle<double, double>;
