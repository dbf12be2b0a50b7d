// Host tests on a permutation group given by generators (group.cu).
#pragma once
#include <cstdint>

namespace mgbfs2 {

// Whether the group on n points is shown to be A_n or S_n (Jordan's theorem);
// false means "not shown".  Permutations as validated images, gens x n.
bool group_is_giant(const uint32_t* permutations, uint32_t n, uint32_t generators);

}  // namespace mgbfs2
