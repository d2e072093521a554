// Host mesh tables as the engine uses them (hostmesh.cpp).
#pragma once

#include <utility>
#include <vector>

#include "../../include/vmcuda.h"

// Mesh::lookup into a vector the caller keeps; false for a lens whose projection is unknown.
bool vm_hostmesh_ranges_(const vm_hostmesh* mesh, const float Hoc[16], const vm_lens* lens, std::vector<std::pair<int, int>>& ranges);
