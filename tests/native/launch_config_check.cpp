// Host check of the autotuner's values (launch_config.h): every field's values launch in different shapes
// on top of any other values, the defaults are among them, and a value that stands for a default is known
// as the same launch. Exit status 0 when all hold.
#include <cstdio>

#include "launch_config.h"

using namespace blgpu;

int main() {
  int bad = 0;
  const LaunchConfig defaults;
  for (const LaunchField& f : kLaunchFields) {
    bool has_default = false;
    for (int i = 0; i < f.count; i++) {
      LaunchConfig a = defaults;
      a.*f.field = f.values[i];
      has_default |= same_launches(a, defaults);
      for (int j = i + 1; j < f.count; j++) {
        LaunchConfig b = defaults;
        b.*f.field = f.values[j];
        if (same_launches(a, b)) { printf("values %d and %d are the same launch\n", f.values[i], f.values[j]); bad++; }
      }
    }
    if (!has_default) { printf("a default is not tried\n"); bad++; }
  }
  LaunchConfig named = defaults;
  named.cover_slots = 32;
  named.cover_blocks_per_sm = 64;
  if (!same_launches(named, defaults)) { printf("named defaults differ\n"); bad++; }
  printf("failures %d\n", bad);
  return bad ? 1 : 0;
}
