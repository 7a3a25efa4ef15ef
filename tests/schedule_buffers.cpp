// Where a scene keeps the tile schedule of an image size on the legacy stream,
// for tests that plant one; built by test_gpu_schedule.py.
#include "device_scene.h"
#include "scene.h"

// out: the buffer that the next launch reads, the one it writes, their words
// and the word offsets of the accumulators and lists.
extern "C" int schedule_buffers(lrt_scene* s, uint32_t width, uint32_t height, uint64_t out[5])
{
  const auto it = s->dev->sched.find(lrt::SchedKey(nullptr, width, height));
  if (it == s->dev->sched.end()) return 1;
  const uint64_t tiles = uint64_t((width + lrt::kImgTileW - 1) / lrt::kImgTileW) * ((height + lrt::kImgTileH - 1) / lrt::kImgTileH);
  out[0] = reinterpret_cast<uint64_t>(it->second.buf[it->second.rd]);
  out[1] = reinterpret_cast<uint64_t>(it->second.buf[1 - it->second.rd]);
  out[2] = lrt::sched_words(tiles);
  out[3] = lrt::sched_acc_offset(tiles);
  out[4] = lrt::sched_lists_offset(tiles);
  return 0;
}
