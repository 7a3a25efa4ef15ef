// Commits a scene whose tree is validated by all cores while every thread but
// the caller's gets no memory; built and run by test_large_validation.py.
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <thread>
#include <vector>

#include "lrt_b200.h"

static std::atomic<bool> armed{false};
static std::atomic<int> refused{0};
static std::thread::id caller;

void* operator new(std::size_t n)
{
  if (armed && std::this_thread::get_id() != caller) {
    refused++;
    throw std::bad_alloc();
  }
  void* p = std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main()
{
  caller = std::this_thread::get_id();
  std::vector<float> v;
  std::vector<uint32_t> t;
  for (int i = 0; i < 60000; i++) {
    for (int c = 0; c < 3; c++) {
      for (int k = 0; k < 3; k++) v.push_back(std::sin(i * 0.37f + c * 0.01f + k));
      t.push_back(uint32_t(3 * i + c));
    }
  }
  lrt_scene* s = nullptr;
  if (lrt_scene_create("cbvh_embree2", "SuperTreeletAlignedMerged4", &s) != LRT_OK) return 2;
  uint32_t g = 0, inst = 0;
  if (lrt_add_geom_triangles3f(s, v.data(), v.size() / 3, t.data(), t.size(), 4, 12, &g) != LRT_OK) return 3;
  const float m[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1};
  if (lrt_add_instance(s, g, m, &inst) != LRT_OK) return 4;
  armed = true;
  const lrt_status st = lrt_commit_scene(s, 4 | LRT_COMMIT_HOST_ONLY);
  armed = false;
  std::printf("status %d, refused %d\n", int(st), refused.load());
  return st == LRT_OK ? 0 : 5;
}
