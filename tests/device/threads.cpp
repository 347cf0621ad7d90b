// Threads that unbind subhaloes of very different sizes at the same time, each with its own
// handle, for tests/test_threads.py: prints the first failed or differing
// calls and, last, their number.
#include "hbtu.h"

#include <atomic>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

static std::atomic<int> failures{0};

static void work(int n, int calls)
{
  hbtu_params p;
  std::memset(&p, 0, sizeof(p));
  p.softening = 0.002;
  p.open_angle = 0.45;
  p.bound_mass_precision = 0.995;
  p.min_num_part = 20;
  p.refine_mostbound = 1;
  p.periodic = 1;
  p.box_size = 100.;
  p.G = 43.0071;
  p.hubble = 100.;
  p.scale_factor = 1.;
  hbtu_handle *h = nullptr;
  if (hbtu_create(&p, &h) != HBTU_OK) {
    failures++;
    return;
  }
  std::vector<float> x(3 * n), v(3 * n), m(n, 0.1f), energy(n), energy0;
  std::vector<int64_t> id(n), order(n), order0;
  unsigned seed = (unsigned)n;
  auto uniform = [&] {
    seed = seed * 1664525u + 1013904223u;
    return (seed >> 8) / 16777216.f - 0.5f;
  };
  for (int i = 0; i < n; i++) {
    id[i] = i;
    for (int j = 0; j < 3; j++) {
      x[3 * i + j] = 50.f + 0.05f * uniform();
      v[3 * i + j] = 5.f * uniform();
    }
  }
  hbtu_particles q;
  std::memset(&q, 0, sizeof(q));
  q.id = id.data();
  q.pos = x.data();
  q.vel = v.data();
  q.mass = m.data();
  q.location = HBTU_HOST;
  hbtu_state st;
  std::memset(&st, 0, sizeof(st));
  for (int j = 0; j < 3; j++) st.ref_pos[j] = st.mostbound_pos[j] = 50.f;
  for (int k = 0; k < calls; k++) {
    hbtu_result r;
    const hbtu_status rc = hbtu_unbind(h, &q, n, &st, order.data(), energy.data(), &r);
    if (k == 0) {
      order0 = order;
      energy0 = energy;
    }
    const bool same = order == order0 && !std::memcmp(energy.data(), energy0.data(), 4 * (size_t)n);
    if (rc != HBTU_OK || !same) {
      if (failures++ < 4) std::printf("n %d call %d: %d %s\n", n, k, (int)rc, hbtu_last_error(h));
      break;
    }
  }
  hbtu_destroy(h);
}

int main()
{
  const int sizes[16] = {2, 2000, 2, 1900, 3, 2000, 2, 1800, 2, 2000, 3, 1900, 2, 2000, 2, 1700};
  std::vector<std::thread> threads;
  for (int n : sizes) threads.emplace_back(work, n, 4000);
  for (auto &t : threads) t.join();
  std::printf("%d\n", failures.load());
  return failures.load() != 0;
}
