// The walk codes of a scene by one sequential enumeration per cone on the
// host (cells x, y, z in order, each heliostat once): what the device's warps
// must find.  Arguments: scene, configuration, sun direction (3), tangent of
// the largest sun-shape angle, largest slope-error angle.  Prints the shadow
// code of every heliostat, then the block code of every sub-heliostat, grid by
// grid.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "device_scene.h"
#include "helio_geom.h"
#include "scene.h"
#include "shadow.h"

static int code(const qm::ShadowGrid& g, int own, int state, const qm::Cone& o) {
  if (state <= 0) return state < 0 ? 0 : 1;
  std::set<int> found;
  for (int x = o.lo[0]; x <= o.hi[0]; ++x)
    for (int y = o.lo[1]; y <= o.hi[1]; ++y)
      for (int z = o.lo[2]; z <= o.hi[2]; ++z) {
        const int2 r = g.ranges[(x * g.cells.y + y) * g.cells.z + z];
        for (int k = r.x; k < r.y; ++k) {
          const int j = g.entries[k].x;
          if (j != own && qm::cone_meets(o, g.bound + 5 * j)) found.insert(j);
        }
      }
  return found.size() <= (size_t)qm::kMaxCandidates ? (int)found.size() + 1 : 0;
}

int main(int argc, char** argv) {
  qm::SceneModel m;
  std::string err;
  qm::SceneConfig cfg;
  if (argc != 8 || qm::read_config_file(argv[2], cfg, err) < 0 || !qm::read_scene_file(argv[1], m, err)) return 1;
  m.config = cfg;
  if (!qm::process_scene(m, err)) return 1;
  const float3 sun = make_float3(atof(argv[3]), atof(argv[4]), atof(argv[5]));
  const float tan_local = atof(argv[6]), slope = atof(argv[7]);
  qm::set_sun(m, sun);
  const float3 axis = qm::neg(sun);
  const float tan_world =
      (float)(tan_local / std::sqrt((double)sun.x * sun.x + (double)sun.y * sun.y + (double)sun.z * sun.z));
  const float theta = std::atan(tan_world) + 2.0f * slope;
  for (int pass = 0; pass < 2; ++pass)
    for (const auto& g : m.grids) {
      std::vector<float4> bound(5 * (size_t)g.num_heliostats);
      std::vector<int2> ranges;
      std::vector<int4> entries;
      for (size_t c = 0; c + 1 < g.cell_hindex.size(); ++c)
        ranges.push_back(make_int2(g.cell_hindex[c], g.cell_hindex[c + 1]));
      for (int h : g.cell_hmatch) entries.push_back(make_int4(h, 0, 0, 0));
      for (int i = 0; i < g.num_heliostats; ++i) {
        const auto& h = m.heliostats[g.start_heliostat + i];
        int2 rc;
        qm::heliostat_record(&g.sub_vertices[3 * (size_t)h.sub_begin], h.num_sub, h.row_col, h.pos, h.normal,
                             &bound[5 * (size_t)i], &rc);
      }
      float top = -3.0e38f;
      for (size_t i = 0; i < bound.size(); i += 5) {
        const float4* c = &bound[i];
        top = std::fmax(top, c[0].y + std::fabs(c[1].y) * c[1].w + std::fabs(c[2].y) * c[2].w + std::fabs(c[3].y) * c[3].w);
      }
      const qm::ShadowGrid view{g.pos, g.interval, g.cells, bound.data(), ranges.data(), entries.data(), top};
      qm::Cone o;
      for (int i = 0; i < g.num_heliostats; ++i) {
        const auto& h = m.heliostats[g.start_heliostat + i];
        if (pass == 0) {
          std::printf("%d\n", code(view, i, qm::shadow_cone(view, i, axis, tan_world, o), o));
          continue;
        }
        const qm::Frame f = qm::make_frame(h.normal, h.type == 1);
        for (int s = 0; s < h.num_sub; ++s) {
          const float3* v = &g.sub_vertices[3 * (size_t)(h.sub_begin + s)];
          const float3 A = v[1], ab = qm::sub(v[0], A), ac = qm::sub(v[2], A);
          const float3 bac[3] = {qm::add(A, ab), A, qm::add(A, ac)};
          const float3 n = h.type == 1 ? qm::to_world(f, h.local_normals[s]) : h.normal;
          std::printf("%d\n", code(view, i, qm::block_cone(view, bac, sun, n, theta, o), o));
        }
      }
    }
  return 0;
}
