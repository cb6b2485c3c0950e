// coordination.h - the coordination-number observable and the VTK writer of the world.
#pragma once

#include <cstdint>
#include <string>

#include "dem_common.cuh"
#include "scene_host.h"

namespace vedo {

struct Box6 { double v[6]; };   // xmin, xmax, ymin, ymax, zmin, zmax

// DOWorld::WriteVTK<ExtFieldWriterT>(filename) (DOWorld_WriteVTK.h:148-243) of the scene's models
// with the given object state (host arrays, [n][3]); with coordination (per object, host), the
// "CoordinateNumber" field of the spheres in object order as outputCoordinateNumVTK adds it.
bool write_world_vtk(const std::string& path, const HScene& s, const double* pos, const double* vel,
                     const double* av, const uint32_t* coordination, std::string& err);

}  // namespace vedo
