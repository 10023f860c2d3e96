// walk_rule.cpp -- the rule that picks a batched launch's walk, on the host:
// configurations that mean the same run the same.  Exit code 0 when they do.
#include <cstdio>
#include <cstring>

#include "scene.h"

int main() {
  kdgr_scene_s scene;
  int bad = 0;
  for (uint32_t leaves : {4u, 30u, 100u})
    for (uint64_t rays : {1000ull, 40000ull, 400000ull, 900000ull, 3000000ull})
      for (int precision : {0, 1})
        for (int hits : {4, 0, 8})
          for (int rpw : {32, 0})
            for (int schedule : {KDGR_SCHED_SM_STRIPS, KDGR_SCHED_WARP_STRIPS}) {
              scene.n_gauss = 1000;
              scene.n_pair_entries = leaves * 1000;
              kdgr_batch_config d, c, want, got;
              kdgr_batch_config_default(&d);
              d.precision = precision;
              c = d;
              c.hit_buffer = hits;
              c.rays_per_warp = rpw;
              c.schedule = schedule;
              want = hits != 8 && schedule == d.schedule ? kdgr::choose_walk(&scene, d, rays) : c;
              got = kdgr::choose_walk(&scene, c, rays);
              if (std::memcmp(&want, &got, sizeof got) != 0) {
                std::printf("%u leaves, %llu rays, precision %d, hit_buffer %d, rays_per_warp %d, schedule %d\n",
                            leaves, (unsigned long long)rays, precision, hits, rpw, schedule);
                bad = 1;
              }
            }
  return bad;
}
