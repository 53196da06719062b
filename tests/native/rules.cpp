// `rules product_lanes <lanes per row> <rows> <longest row>` prints the lanes of the product.
#include "fake_cuda.h"

#include "device.h"

int main(int, char** argv) {
  sf::DevBsr m;
  m.lanes_per_row = std::atoi(argv[2]);
  m.rows = std::atoi(argv[3]);
  m.longest_row = std::atoi(argv[4]);
  std::printf("%d\n", sf::product_lanes(m));
}
