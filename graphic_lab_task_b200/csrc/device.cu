// device.cu — device half of the scene object: upload of the reference arrays
// plus the derived layouts, and the ray-query entry points of the C-ABI.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <vector>

#include "device_scene.h"
#include "layout.h"
#include "scene.h"
#include "trace_api.h"

namespace lrt {

lrt_status cuda_fail(lrt_scene* s, cudaError_t e, const char* what)
{
  return fail(s, e == cudaErrorMemoryAllocation ? LRT_ERR_OUT_OF_MEMORY : LRT_ERR_CUDA, "%s: %s", what,
              cudaGetErrorString(e));
}

uint32_t preset_flags(const lrt_preset& p)
{
  const uint32_t m = p.render_mode; // need_normal(), BVH2Common.cpp:19-32
  const bool nn = m == 1 || m == 8 || m == 12 || m == 17 || m == 20 || m == 7 || m == 18 || m == 23 || m == 21 ||
                  m == 11 || m == 27;
  uint32_t f = 0;
  if (nn) f |= kFlagNeedNormal;
  if (m == LRT_RENDER_MODE_ST_ITERATIONS) f |= kFlagStIterations;
  if (p.representation_mode == 0) f |= kFlagSurfaceMode;
  if (p.sdf_node_intersect == 3) f |= kFlagBBoxMode;
  f |= (p.sdf_node_intersect & 7u) << kFlagSolverShift;
  return f;
}

uint32_t launch_flags(const lrt_scene* s)
{
  return preset_flags(s->preset) | (s->dev->cleanBoxes ? kFlagCleanBoxes : 0u);
}

namespace {

// True if every box of the nodes has either no NaN coordinate or six.
bool boxes_clean(const lrt_bvh_node* n, size_t count)
{
  for (size_t i = 0; i < count; i++) {
    int nans = 0;
    for (int k = 0; k < 3; k++) nans += std::isnan(n[i].boxMin[k]) + std::isnan(n[i].boxMax[k]);
    if (nans != 0 && nans != 6) return false;
  }
  return true;
}

// Turns `count` uploaded nodes into node records in place (device_layout.h).
// owner: the geometry of each node pair.  *unclean: a box has some but not six
// NaN coordinates.
__global__ void __launch_bounds__(256) k_node_records(float4* __restrict__ nodes, uint64_t count,
                                                      const uint32_t* __restrict__ owner,
                                                      const DevGeom* __restrict__ geoms,
                                                      const uint32_t* __restrict__ leafTable,
                                                      uint32_t* __restrict__ unclean)
{
  const uint64_t i = uint64_t(blockIdx.x) * 256 + threadIdx.x;
  if (i >= count) return;
  const float4 a = nodes[2 * i], b = nodes[2 * i + 1];
  uint32_t word = __float_as_uint(a.w);
  if ((word & kLeafBit) && word != kLeafNormal) {
    const uint32_t g = owner[i >> 1];
    if (g != ~0u) word = kLeafBit | (leafTable[geoms[g].aabbBase + (word & kStartMask)] & ~kLeafBit);
  }
  const int nans = isnan(a.x) + isnan(a.y) + isnan(a.z) + isnan(b.x) + isnan(b.y) + isnan(b.z);
  if (nans != 0 && nans != 6) *unclean = 1u;
  nodes[2 * i] = make_float4(a.x, b.x, a.y, b.y);
  nodes[2 * i + 1] = make_float4(a.z, b.z, __uint_as_float(word), b.w);
}

// {A, B-A, C-A} per reordered triangle slot, from the vertices (float4) and
// indices; IntersectAllTrianglesInLeaf computes exactly these differences
// (BVH2Common.cpp:1585-1589).  One thread per entry of a geometry's leaf table:
// the slots that its leaves cover are the ones whose indices validate has
// checked, and no others are followed (a table may leave gaps, and an entry of
// no triangles may start anywhere).
__global__ void __launch_bounds__(kSoupThreads) k_tri_soup(const float4* __restrict__ verts,
                                                           const uint32_t* __restrict__ indices,
                                                           const uint32_t* __restrict__ leafTable,
                                                           const DevGeom* __restrict__ geoms,
                                                           const uint32_t* __restrict__ startEnd,
                                                           const SoupBlock* __restrict__ blocks,
                                                           float4* __restrict__ soup)
{
  const SoupBlock b = blocks[blockIdx.x];
  const uint64_t a = uint64_t(b.firstLeaf) + threadIdx.x;
  if (a >= startEnd[2 * uint64_t(b.geom) + 1]) return;
  const DevGeom g = geoms[b.geom];
  const uint32_t entry = leafTable[a];
  const uint64_t first = uint64_t(g.triBase) + (entry & kStartMask), end = first + ((entry & kSizeMask) >> 28);
  for (uint64_t t = first; t < end; t++) {
    const uint32_t* idx = indices + 3 * t;
    const float4 A = verts[uint64_t(g.firstVert) + idx[0]], B = verts[uint64_t(g.firstVert) + idx[1]],
                 C = verts[uint64_t(g.firstVert) + idx[2]];
    float4* o = soup + 3 * t;
    o[0] = make_float4(A.x, A.y, A.z, 0.0f);
    o[1] = make_float4(__fsub_rn(B.x, A.x), __fsub_rn(B.y, A.y), __fsub_rn(B.z, A.z), 0.0f);
    o[2] = make_float4(__fsub_rn(C.x, A.x), __fsub_rn(C.y, A.y), __fsub_rn(C.z, A.z), 0.0f);
  }
}

// The records of the few TLAS nodes, made on the host; their leaf words stay.
void tlas_records(const std::vector<lrt_bvh_node>& in, bool sideBySide, std::vector<lrt_bvh_node>& out)
{
  out = in;
  if (!sideBySide) return;
  for (size_t i = 0; i < in.size(); i++) {
    const lrt_bvh_node& n = in[i];
    const float box[6] = {n.boxMin[0], n.boxMax[0], n.boxMin[1], n.boxMax[1], n.boxMin[2], n.boxMax[2]};
    char* o = reinterpret_cast<char*>(&out[i]);
    std::memcpy(o, box, sizeof(box));
    std::memcpy(o + 24, &n.leftOffset, 4);
    std::memcpy(o + 28, &n.escapeIndex, 4);
  }
}

// Below these sizes the triangle soup and the node records are made on the
// host: the buffers, copies, launches and synchronisations of the device's way
// take 60 us.  Measured (us, a commit of one mesh, host / device): 1,000
// triangles 128 / 181, 4,000 168 / 204, 8,000 279 / 274, 24,000 (BUILD_LOW)
// 1,415 / 1,050, 200,000 5,640 / 3,070; 500 meshes of 12 triangles 640 / 1,440.
constexpr uint64_t kHostSoupSlots = 6144;
constexpr size_t kHostRecordPairs = 4096;

template <class T>
lrt_status upload_vec(lrt_scene* s, DeviceScene* d, const T* src, size_t count, const T** out, const char* name)
{
  *out = nullptr;
  if (count == 0) return LRT_OK;
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, count * sizeof(T));
  if (e != cudaSuccess) return cuda_fail(s, e, name);
  d->allocs.push_back(p);
  e = cudaMemcpy(p, src, count * sizeof(T), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return cuda_fail(s, e, name);
  *out = static_cast<const T*>(p);
  return LRT_OK;
}

lrt_status slot_for(lrt_scene* s, cudaStream_t stream, StreamSlot** out)
{
  DeviceScene* d = s->dev;
  auto it = d->slotOf.find(stream);
  int idx;
  if (it == d->slotOf.end()) {
    if (int(d->slotOf.size()) >= kMaxStreams)
      return fail(s, LRT_ERR_INVALID_ARGUMENT, "more than %d streams used with one scene", kMaxStreams);
    idx = int(d->slotOf.size());
    d->slotOf[stream] = idx;
  } else {
    idx = it->second;
  }
  *out = d->slots + idx;
  return LRT_OK;
}

} // namespace

lrt_status sched_prepare(lrt_scene* s, cudaStream_t stream, uint32_t width, uint32_t height, bool natural,
                         const uint32_t** rd, uint32_t** wr)
{
  *rd = nullptr;
  *wr = nullptr;
  if (natural) return LRT_OK;
  DeviceScene* d = s->dev;
  const uint64_t tiles = uint64_t((width + kImgTileW - 1) / kImgTileW) * ((height + kImgTileH - 1) / kImgTileH);
  const size_t clear = sched_lists_offset(tiles) * sizeof(uint32_t); // header, bitmap, cost accumulators
  cudaError_t e = cudaSuccess;
  const SchedKey key(stream, width, height);
  auto it = d->sched.find(key);
  if (it == d->sched.end()) {
    if (d->sched.size() >= kMaxSchedules) { // free the least recently used schedule
      auto old = d->sched.begin();
      for (auto jt = d->sched.begin(); jt != d->sched.end(); ++jt)
        if (jt->second.lastUse < old->second.lastUse) old = jt;
      for (uint32_t* b : old->second.buf) cudaFree(b);
      d->sched.erase(old);
    }
    ImageSchedule fresh;
    for (uint32_t*& b : fresh.buf) {
      if (e == cudaSuccess) e = cudaMalloc(&b, sched_words(tiles) * sizeof(uint32_t));
      if (e == cudaSuccess) e = cudaMemsetAsync(b, 0, clear, stream);
    }
    if (e != cudaSuccess) {
      for (uint32_t* b : fresh.buf) cudaFree(b);
      return cuda_fail(s, e, "tile schedule buffers");
    }
    it = d->sched.emplace(key, fresh).first;
  }
  ImageSchedule& q = it->second;
  q.lastUse = ++d->schedUses;
  e = cudaMemsetAsync(q.buf[1 - q.rd], 0, clear, stream);
  if (e != cudaSuccess) return cuda_fail(s, e, "cudaMemsetAsync");
  *rd = q.buf[q.rd];
  *wr = q.buf[1 - q.rd];
  return LRT_OK;
}

void sched_commit(lrt_scene* s, cudaStream_t stream, uint32_t width, uint32_t height, bool natural)
{
  if (natural) return;
  auto it = s->dev->sched.find(SchedKey(stream, width, height));
  if (it != s->dev->sched.end()) it->second.rd = 1 - it->second.rd;
}

namespace {

// img_w > 0: the n = img_w * img_h rays are an image in row-major order,
// traced in 8x4-pixel tiles, in the stream's tile schedule unless flags has
// LRT_TRACE_NATURAL_ORDER (or LRT_TRACE_COUNT_WORK).
// err: the error word the kernel reports into (default: the slot's).
// staged: the rays and hits are page-locked host memory; a launch whose warps
// all fit one wave then takes its groups by warp index, without a counter.
lrt_status launch(lrt_scene* s, const float4* rays, lrt_hit* hits, uint64_t n, cudaStream_t stream, uint32_t flags,
                  StreamSlot* slot, uint32_t img_w = 0, uint32_t img_h = 0, uint32_t* err = nullptr,
                  bool staged = false)
{
  if (!err) err = &slot->err;
  DeviceScene* d = s->dev;
  DevScene S = d->S;
  S.flags = launch_flags(s);
  S.voxelStepCap = s->voxelStepCap ? s->voxelStepCap : kMaxVoxelSteps;
  if (n < kPrefetchMinRays)
    for (int r = 0; r < kPrefetchRanges; r++) S.pfBytes[r] = 0;
  const bool count = (flags & LRT_TRACE_COUNT_WORK) != 0;
  const uint32_t group = img_w ? 32 : rays_per_warp(n, S.sms);
  const uint64_t warps = img_w ? uint64_t((img_w + kImgTileW - 1) / kImgTileW) * ((img_h + kImgTileH - 1) / kImgTileH)
                               : (n + group - 1) / group;
  const int blocks = blocks_for(warps);
  unsigned long long* work = &slot->work;
  cudaError_t e = cudaSuccess;
  if (staged && !count && blocks <= lrt_exact::row_wave(S, S.flags, d->stackCap))
    work = nullptr;
  else
    e = cudaMemsetAsync(work, 0, count ? offsetof(StreamSlot, err) : sizeof(unsigned long long), stream);
  if (e != cudaSuccess) return cuda_fail(s, e, "cudaMemsetAsync");
  const bool natural = !img_w || count || (flags & LRT_TRACE_NATURAL_ORDER);
  const uint32_t* rd = nullptr;
  uint32_t* wr = nullptr;
  lrt_status st = sched_prepare(s, stream, img_w, img_h, natural, &rd, &wr);
  if (st != LRT_OK) return st;
  if (flags & LRT_TRACE_FAST_MATH)
    e = lrt_fast::launch_trace(S, rays, hits, n, work, slot->counters, err, d->stackCap, blocks, stream, count,
                               img_w, img_h, rd, wr, group);
  else
    e = lrt_exact::launch_trace(S, rays, hits, n, work, slot->counters, err, d->stackCap, blocks, stream,
                                count, img_w, img_h, rd, wr, group);
  if (e != cudaSuccess) return cuda_fail(s, e, "trace launch");
  sched_commit(s, stream, img_w, img_h, natural);
  return LRT_OK;
}

lrt_status limit_fail(lrt_scene* s, uint32_t bits)
{
  return fail(s, LRT_ERR_DEVICE_LIMIT,
              "trace hit a bounded-loop limit (error bits 0x%x: 1 = stack, 2 = voxel march, 4 = transparency layers)",
              bits);
}

// Reads back (and clears) the error word and, if asked, the counters of a slot.
lrt_status finish(lrt_scene* s, cudaStream_t stream, StreamSlot* slot, bool count)
{
  StreamSlot hs;
  cudaError_t e = cudaMemcpyAsync(&hs, slot, sizeof(hs), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(s, e, "trace");
  if (count)
    for (int k = 0; k < LRT_COUNTER_COUNT; k++) s->counters[k] = hs.counters[k];
  if (hs.err) {
    cudaMemsetAsync(&slot->err, 0, sizeof(uint32_t), stream);
    cudaStreamSynchronize(stream);
    return limit_fail(s, hs.err);
  }
  return LRT_OK;
}

// Host-pointer trace of ordinary memory, of at most kStageMaxRays: the rays are
// copied into page-locked memory, from which the kernel reads them and into
// which it writes the hits and its error word, so that the call is one launch
// and one synchronisation.  Device staging took two pageable copies, a memset
// and a read of the slot's state around the same kernel, each with a
// synchronisation of its own.  Measured (us, device staging -> this): one
// ray 55.6 -> 28-35, 4,099 rays 125-164 -> 90-112.  False if the memory cannot be
// had (the caller then stages on the device).
bool host_stage(DeviceScene* d, uint64_t n)
{
  if (n <= d->stageCap) return true;
  uint64_t cap = kStageMinRays;
  while (cap < n) cap *= 2;
  if (d->stage) cudaFreeHost(d->stage);
  d->stage = nullptr;
  d->stageCap = 0;
  void* p = nullptr;
  if (cudaHostAlloc(&p, kStageHeader + cap * (32 + sizeof(lrt_hit)), cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError(); // not sticky: clear it
    return false;
  }
  d->stage = static_cast<unsigned char*>(p);
  d->stageCap = cap;
  return true;
}

// Ordinary memory, which the caller's thread may read and write at once: a
// page-locked, managed or device buffer may have work on the stream still to
// come before it holds the rays, and is copied in stream order.
bool pageable(const void* p)
{
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError(); // not sticky: clear it
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

lrt_status trace_host_staged(lrt_scene* s, const float* rays, lrt_hit* hits, uint64_t n, cudaStream_t stream,
                             uint32_t flags, StreamSlot* slot)
{
  DeviceScene* d = s->dev;
  unsigned char* dev = nullptr;
  cudaError_t e = cudaHostGetDevicePointer(reinterpret_cast<void**>(&dev), d->stage, 0);
  if (e != cudaSuccess) return cuda_fail(s, e, "staging buffer");
  volatile uint32_t* err = reinterpret_cast<uint32_t*>(d->stage);
  unsigned char* hostHits = d->stage + kStageHeader + d->stageCap * 32;
  *err = 0;
  std::memcpy(d->stage + kStageHeader, rays, n * 32);
  lrt_status st = launch(s, reinterpret_cast<const float4*>(dev + kStageHeader),
                         reinterpret_cast<lrt_hit*>(dev + kStageHeader + d->stageCap * 32), n, stream, flags, slot, 0, 0,
                         reinterpret_cast<uint32_t*>(dev), true);
  if (st != LRT_OK) return st;
  e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(s, e, "trace");
  std::memcpy(hits, hostHits, n * sizeof(lrt_hit));
  return *err ? limit_fail(s, *err) : LRT_OK;
}

// Chunk sizes of the pipeline: kPipeChunkMin, doubling up to kPipeChunk,
// chunks of at most kPipeChunk, and the ramp again in reverse, so that the
// first copy in and the last trace and copy out, which nothing overlaps, are
// short.  Inputs too small for the ramps get chunks of kPipeChunkMin.
void pipeline_chunks(uint64_t n, std::vector<uint64_t>& out)
{
  out.clear();
  std::vector<uint64_t> up;
  uint64_t ramp = 0;
  for (uint64_t m = kPipeChunkMin; m < kPipeChunk; m *= 2) {
    up.push_back(m);
    ramp += m;
  }
  if (n <= 2 * ramp) {
    for (uint64_t off = 0; off < n; off += kPipeChunkMin) out.push_back(std::min(kPipeChunkMin, n - off));
    return;
  }
  out = up;
  const uint64_t mid = n - 2 * ramp;
  const uint64_t parts = (mid + kPipeChunk - 1) / kPipeChunk;
  for (uint64_t i = 0; i < parts; i++) out.push_back(mid / parts + (i < mid % parts ? 1 : 0));
  out.insert(out.end(), up.rbegin(), up.rend());
}

// Host-pointer trace in chunks (staging buffers already hold n rays): chunk c
// is copied in on kPipeIn, traced on trace stream c mod kPipeTraceStreams
// once its copy is done, and copied out on kPipeOut once its trace is done.
// The copies of consecutive chunks run back to back in both directions while
// the traces of several chunks run at the same time.  The pipeline starts
// after the work already queued on the caller's stream, and the caller's
// stream waits for it.  Events are re-recorded once per chunk: a wait takes
// the record made before it.  Every trace reports into one error word, which
// the copy-out stream (that has waited for every trace) reads into page-locked
// host memory after the last hits, so one synchronisation ends the call.
lrt_status trace_host_pipelined(lrt_scene* s, const float* rays, lrt_hit* hits, uint64_t n, cudaStream_t stream,
                                uint32_t flags)
{
  DeviceScene* d = s->dev;
  cudaError_t e = cudaSuccess;
  if (!d->pipeStart) {
    for (int p = 0; p < kPipeStreams && e == cudaSuccess; p++) {
      e = cudaStreamCreateWithFlags(&d->pipe[p], cudaStreamNonBlocking);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&d->pipeEv[p], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaHostAlloc(&d->pipeErrHost, sizeof(uint32_t), cudaHostAllocDefault);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&d->pipeStart, cudaEventDisableTiming);
    if (e != cudaSuccess) return cuda_fail(s, e, "pipeline streams");
  }
  cudaStream_t in = d->pipe[kPipeIn], out = d->pipe[kPipeOut];
  StreamSlot* slots[kPipeTraceStreams];
  for (int k = 0; k < kPipeTraceStreams; k++) {
    lrt_status st = slot_for(s, d->pipe[kPipeTrace + k], &slots[k]);
    if (st != LRT_OK) return st;
  }
  uint32_t* err = &slots[0]->err;
  e = cudaEventRecord(d->pipeStart, stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(in, d->pipeStart, 0);
  if (e != cudaSuccess) return cuda_fail(s, e, "pipeline start");
  lrt_status st = LRT_OK;
  std::vector<uint64_t> chunks;
  pipeline_chunks(n, chunks);
  for (uint64_t off = 0, c = 0; c < chunks.size(); off += chunks[c], c++) {
    const uint64_t m = chunks[c];
    const int k = int(c % kPipeTraceStreams);
    cudaStream_t tr = d->pipe[kPipeTrace + k];
    e = cudaMemcpyAsync(d->rays + 2 * off, rays + 8 * off, m * 32, cudaMemcpyHostToDevice, in);
    if (e == cudaSuccess) e = cudaEventRecord(d->pipeEv[kPipeIn], in);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(tr, d->pipeEv[kPipeIn], 0);
    if (e != cudaSuccess) {
      st = cuda_fail(s, e, "rays host->device");
      break;
    }
    st = launch(s, d->rays + 2 * off, d->hits + off, m, tr, flags, slots[k], 0, 0, err);
    if (st != LRT_OK) break;
    e = cudaEventRecord(d->pipeEv[kPipeTrace + k], tr);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(out, d->pipeEv[kPipeTrace + k], 0);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(hits + off, d->hits + off, m * sizeof(lrt_hit), cudaMemcpyDeviceToHost, out);
    if (e != cudaSuccess) {
      st = cuda_fail(s, e, "hits device->host");
      break;
    }
  }
  if (st == LRT_OK) {
    e = cudaMemcpyAsync(d->pipeErrHost, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, out);
    if (e != cudaSuccess) st = cuda_fail(s, e, "error word");
  }
  // the caller's stream waits for the last copy out
  if (cudaEventRecord(d->pipeEv[kPipeOut], out) == cudaSuccess) cudaStreamWaitEvent(stream, d->pipeEv[kPipeOut], 0);
  if (st != LRT_OK) { // drain every stream after a failure
    for (int p = 0; p < kPipeStreams; p++) cudaStreamSynchronize(d->pipe[p]);
    cudaMemsetAsync(err, 0, sizeof(uint32_t), out);
    cudaStreamSynchronize(out);
    return st;
  }
  e = cudaStreamSynchronize(out);
  if (e != cudaSuccess) return cuda_fail(s, e, "hits device->host");
  const uint32_t bits = *d->pipeErrHost;
  if (bits) {
    cudaMemsetAsync(err, 0, sizeof(uint32_t), out);
    cudaStreamSynchronize(out);
    return limit_fail(s, bits);
  }
  return LRT_OK;
}

} // namespace

namespace {

// Makes the triangle soup: 48 bytes a triangle, on the device from its 12 bytes
// of indices and the shared vertices, or, where a few triangles would not pay
// for the buffers, copies and launch that takes, on the host.
lrt_status tri_soup(lrt_scene* s)
{
  DeviceScene* d = s->dev;
  const HostArrays& h = s->h;
  const uint64_t nslots = h.indices.size() / 3;
  d->S.triSoup = nullptr;
  if (nslots == 0) return LRT_OK;
  if (nslots < kHostSoupSlots) {
    std::vector<float> soup;
    build_tri_soup(h, soup);
    return upload_vec(s, d, reinterpret_cast<const float4*>(soup.data()), soup.size() / 4, &d->S.triSoup, "triangles");
  }
  std::vector<SoupBlock> blocks;
  const bool apart = build_soup_blocks(h, blocks);
  // one buffer for what the kernel reads
  const size_t bytes[4] = {h.vertPos.size() * sizeof(float), h.indices.size() * sizeof(uint32_t),
                           h.startEnd.size() * sizeof(uint32_t), blocks.size() * sizeof(SoupBlock)};
  const void* from[4] = {h.vertPos.data(), h.indices.data(), h.startEnd.data(), blocks.data()};
  size_t at[5] = {0};
  for (int k = 0; k < 4; k++) at[k + 1] = at[k] + (bytes[k] + 255) / 256 * 256;
  void *soup = nullptr, *p = nullptr;
  cudaError_t e = cudaMalloc(&soup, nslots * 48);
  if (e != cudaSuccess) return cuda_fail(s, e, "triangles");
  d->allocs.push_back(soup);
  e = cudaMalloc(&p, std::max<size_t>(at[4], 1));
  char* in = static_cast<char*>(p);
  for (int k = 0; k < 4; k++)
    if (e == cudaSuccess) e = cudaMemcpy(in + at[k], from[k], bytes[k], cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemsetAsync(soup, 0, nslots * 48);
  for (size_t first = 0; first < blocks.size() && e == cudaSuccess;) {
    size_t end = blocks.size();
    if (!apart) // geometries that share slots write them in their order
      for (end = first + 1; end < blocks.size() && blocks[end].geom == blocks[first].geom;) end++;
    k_tri_soup<<<unsigned(end - first), kSoupThreads>>>(
        reinterpret_cast<const float4*>(in), reinterpret_cast<const uint32_t*>(in + at[1]), d->S.primIdCount, d->S.geoms,
        reinterpret_cast<const uint32_t*>(in + at[2]), reinterpret_cast<const SoupBlock*>(in + at[3]) + first,
        static_cast<float4*>(soup));
    e = cudaGetLastError();
    first = end;
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
  cudaFree(p);
  if (e != cudaSuccess) return cuda_fail(s, e, "triangles");
  d->S.triSoup = static_cast<const float4*>(soup);
  return LRT_OK;
}

// Makes the node records of a scene without bricks from its uploaded BLAS
// pairs and finds whether their boxes are clean.
lrt_status node_records(lrt_scene* s, uint64_t count)
{
  DeviceScene* d = s->dev;
  uint32_t *owner = nullptr, *flags = nullptr, found = 0;
  const size_t ownerBytes = s->pairGeom.size() * sizeof(uint32_t);
  cudaError_t e = cudaMalloc(&owner, ownerBytes);
  if (e == cudaSuccess) e = cudaMalloc(&flags, sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemcpy(owner, s->pairGeom.data(), ownerBytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(flags, 0, sizeof(uint32_t));
  if (e == cudaSuccess) {
    k_node_records<<<unsigned((count + 255) / 256), 256>>>(reinterpret_cast<float4*>(const_cast<DevPair*>(d->S.pairs)),
                                                           count, owner, d->S.geoms, d->S.primIdCount, flags);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(&found, flags, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  cudaFree(owner);
  cudaFree(flags);
  if (e != cudaSuccess) return cuda_fail(s, e, "node records");
  d->pairsClean = !found;
  return LRT_OK;
}

} // namespace

// Device address of the static scratch array of lrt_trace_nearest_noalloc
// (defined with it at the end of this file), for the current device.
cudaError_t noalloc_scratch_address(void** p);

lrt_status device_upload(lrt_scene* s)
{
  device_release(s);
  cudaError_t e = cudaGetDevice(&s->device);
  if (e != cudaSuccess) return cuda_fail(s, e, "cudaGetDevice (no CUDA device?)");
  DeviceScene* d = new DeviceScene();
  s->dev = d;
  const HostArrays& h = s->h;
  DevScene& S = d->S;
  std::vector<DevGeom> geoms;
  std::vector<float> dense;
  std::vector<DevSbs> sbs;
  std::vector<uint32_t> mask;
  build_geoms(h, geoms);
  build_sbs_dense(h, sbs, dense);
  build_sbs_masks(h, sbs, dense, mask);
  S.kind = kernel_kind(h);
  // Only a brick geometry's pairs are pruned.  (SBS arrays that no geometry
  // names change nothing: the scene's pairs become node records then, of which
  // there is one copy.)
  const bool prune = (S.kind & kKindBricks) != 0;
  HostVec<lrt_bvh_node_pair> pruned;
  if (prune) prune_sbs_pairs(h, geoms, sbs, mask, pruned);
  // (records of few pairs are made on the host, before the upload)
  const bool hostRecords = S.kind == kKindNoBricks && h.allNodePairs.size() < kHostRecordPairs;
  HostVec<lrt_bvh_node_pair> records;
  if (hostRecords) d->pairsClean = build_node_records(h, geoms, s->pairGeom, records);
  const HostVec<lrt_bvh_node_pair>& pairs = prune ? pruned : hostRecords ? records : h.allNodePairs;
  lrt_status st = LRT_OK;
#define UP(dst, vec, T, name)                                                                        \
  if (st == LRT_OK) {                                                                                 \
    const T* p = nullptr;                                                                             \
    st = upload_vec(s, d, reinterpret_cast<const T*>(vec.data()), vec.size() * sizeof(vec[0]) / sizeof(T), &p, name); \
    S.dst = p;                                                                                        \
  }
  std::vector<lrt_bvh_node> tlas;
  tlas_records(h.nodesTLAS, S.kind == kKindNoBricks, tlas);
  UP(tlas, tlas, DevNode, "TLAS nodes")
  UP(pairs, pairs, DevPair, "BLAS node pairs")
  UP(primIdCount, h.primIdCount, uint32_t, "leaf table")
  UP(instances, h.instanceData, DevInstance, "instances")
  UP(geoms, geoms, DevGeom, "geometry table")
  if (st == LRT_OK) st = tri_soup(s);
  UP(primIndices, h.primIndices, uint32_t, "primIndices")
  UP(origNodes, h.origNodes, lrt_bvh_node, "origNodes")
  UP(frameOctreeNodes, h.sdfFrameOctreeNodes, lrt_sdf_frame_octree_node, "frame-octree nodes")
  UP(svsNodes, h.sdfSVSNodes, lrt_sdf_svs_node, "SVS nodes")
  UP(sbsNodes, h.sdfSBSNodes, lrt_sdf_sbs_node, "SBS nodes")
  UP(sbsData, h.sdfSBSData, uint32_t, "SBS data")
  UP(sbsDataF, h.sdfSBSDataF, float, "SBS float data")
  UP(sbsDense, dense, float, "SBS dense bricks")
  UP(sbsMask, mask, uint32_t, "SBS surface-voxel masks")
  UP(sbs, sbs, DevSbs, "SBS table")
  if (st == LRT_OK) {
    if (!prune) {
      d->pairsOrig = S.pairs;
    } else {
      const DevPair* p = nullptr;
      st = upload_vec(s, d, reinterpret_cast<const DevPair*>(h.allNodePairs.data()), h.allNodePairs.size(), &p,
                      "unpruned node pairs");
      d->pairsOrig = p;
    }
  }
  if (S.kind == kKindNoBricks) {
    if (st == LRT_OK && !hostRecords) st = node_records(s, 2 * pairs.size());
  } else { // the uploaded nodes are the records
    d->pairsClean = boxes_clean(reinterpret_cast<const lrt_bvh_node*>(pairs.data()), 2 * pairs.size()) &&
                    boxes_clean(reinterpret_cast<const lrt_bvh_node*>(h.allNodePairs.data()), 2 * h.allNodePairs.size());
  }
  std::vector<PruneLeaf> leaves;
  std::vector<uint32_t> parent;
  build_prune_tree(h, geoms, sbs, leaves, parent);
  if (!leaves.empty()) {
    const PruneLeaf* pl = nullptr;
    const uint32_t *pp = nullptr, *pa = nullptr;
    if (st == LRT_OK) st = upload_vec(s, d, leaves.data(), leaves.size(), &pl, "SBS leaf slots");
    if (st == LRT_OK) st = upload_vec(s, d, parent.data(), parent.size(), &pp, "SBS pair parents");
    if (st == LRT_OK) st = upload_vec(s, d, parent.data(), parent.size(), &pa, "SBS live-child bits");
    d->pruneLeaves = pl;
    d->pruneParent = pp;
    d->pruneAlive = const_cast<uint32_t*>(pa);
    d->pruneLeafCount = uint32_t(leaves.size());
    d->prunePairs = uint32_t(parent.size());
  }
  d->sbsHost = sbs;
  d->pairsOrigBytes = h.allNodePairs.size() * sizeof(lrt_bvh_node_pair);
  // what a traversal reads per node, leaf, brick and voxel, most shared first
  d->pfCand = {{S.tlas, h.nodesTLAS.size() * sizeof(lrt_bvh_node)},
               {S.pairs, pairs.size() * sizeof(lrt_bvh_node_pair)},
               {S.kind == kKindNoBricks ? nullptr : S.primIdCount, h.primIdCount.size() * sizeof(uint32_t)},
               {S.sbsNodes, h.sdfSBSNodes.size() * sizeof(lrt_sdf_sbs_node)},
               {S.sbsMask, mask.size() * sizeof(uint32_t)},
               {S.triSoup, h.indices.size() / 3 * 48},
               {S.origNodes, h.origNodes.size() * sizeof(lrt_bvh_node)},
               {S.frameOctreeNodes, h.sdfFrameOctreeNodes.size() * sizeof(lrt_sdf_frame_octree_node)},
               {S.svsNodes, h.sdfSVSNodes.size() * sizeof(lrt_sdf_svs_node)},
               {S.sbsDense, dense.size() * sizeof(float)}};
  set_prefetch(d);
  d->cleanBoxes = d->pairsClean && boxes_clean(h.nodesTLAS.data(), h.nodesTLAS.size());
  d->tlasCount = h.nodesTLAS.size();
  d->instCount = h.instanceData.size();
#undef UP
  if (st != LRT_OK) {
    device_release(s);
    return st;
  }
  d->stackCap = std::max<uint32_t>(s->info.maxBlasDepth + 1, 8u);
  // The dynamic shared-memory limit is a per-kernel attribute shared by all
  // scenes: raise it once to the largest stack any scene may use.
  e = lrt_exact::set_trace_smem(kMaxStack + 1);
  if (e == cudaSuccess) e = lrt_fast::set_trace_smem(kMaxStack + 1);
  int sms = 0;
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
  if (e == cudaSuccess) e = cudaMalloc(&d->slots, sizeof(StreamSlot) * kMaxStreams);
  if (e == cudaSuccess) {
    d->allocs.push_back(d->slots);
    e = cudaMemset(d->slots, 0, sizeof(StreamSlot) * kMaxStreams);
  }
  if (e != cudaSuccess) {
    st = cuda_fail(s, e, "trace setup");
    device_release(s);
    return st;
  }
  S.sms = uint32_t(sms);
  S.instCount = uint32_t(d->instCount);
  // The allocation-free trace's static array is looked up here, with the
  // scene's device current, not in the trace call: under lazy module loading
  // the first lookup loads this file's module and places the array in device
  // memory, which an upload may do and lrt_trace_nearest_noalloc must not.
  // A failed lookup fails only that entry point.
  void* base = nullptr;
  d->noallocErr = noalloc_scratch_address(&base);
  if (d->noallocErr != cudaSuccess) cudaGetLastError(); // not sticky: clear it
  d->noallocBase = static_cast<unsigned char*>(base);
  return LRT_OK;
}

// After a commit that changed only instances (UpdateInstance, or ClearScene
// and AddInstance over the same geometry): write the new TLAS and instances
// into their buffers (new buffers where the counts changed) and leave every
// BLAS, brick and mask array on the device as it is.
lrt_status device_update_instances(lrt_scene* s)
{
  DeviceScene* d = s->dev;
  const HostArrays& h = s->h;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev != s->device)
    return fail(s, LRT_ERR_INVALID_ARGUMENT, "commit on device %d of a scene uploaded to device %d", dev, s->device);
  lrt_status st = LRT_OK;
  auto put = [&](const void* src, size_t count, size_t elem, size_t& have, const void** ptr, const char* name) {
    if (st != LRT_OK) return;
    if (count != have) {
      void* p = nullptr;
      e = cudaMalloc(&p, count * elem);
      if (e != cudaSuccess) {
        st = cuda_fail(s, e, name);
        return;
      }
      d->allocs.push_back(p);
      *ptr = p; // the old buffer stays listed in allocs and is freed with the scene
      have = count;
    }
    e = cudaMemcpy(const_cast<void*>(*ptr), src, count * elem, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) st = cuda_fail(s, e, name);
  };
  std::vector<lrt_bvh_node> tlas;
  tlas_records(h.nodesTLAS, d->S.kind == kKindNoBricks, tlas);
  put(tlas.data(), tlas.size(), sizeof(DevNode), d->tlasCount,
      reinterpret_cast<const void**>(&d->S.tlas), "TLAS nodes");
  put(h.instanceData.data(), h.instanceData.size(), sizeof(lrt_instance_data), d->instCount,
      reinterpret_cast<const void**>(&d->S.instances), "instances");
  if (st != LRT_OK) return st;
  d->S.instCount = uint32_t(d->instCount);
  d->cleanBoxes = d->pairsClean && boxes_clean(h.nodesTLAS.data(), h.nodesTLAS.size());
  return LRT_OK;
}

void set_prefetch(DeviceScene* d)
{
  DevScene& S = d->S;
  uint64_t total = 0;
  int k = 0;
  for (int r = 0; r < kPrefetchRanges; r++) {
    S.pfPtr[r] = nullptr;
    S.pfBytes[r] = 0;
  }
  for (const auto& c : d->pfCand) {
    const uint64_t bytes = c.second & ~uint64_t(15); // whole 16-byte granules (cudaMalloc bases are aligned)
    if (!c.first || bytes == 0 || k == kPrefetchRanges || total + bytes > kPrefetchMaxBytes) continue;
    S.pfPtr[k] = static_cast<const char*>(c.first);
    S.pfBytes[k] = bytes;
    total += bytes;
    k++;
  }
}

void device_release(lrt_scene* s)
{
  if (s->dev) {
    delete s->dev;
    s->dev = nullptr;
  }
}

} // namespace lrt

using namespace lrt;

extern "C" {

lrt_status lrt_trace_nearest(lrt_scene* s, const float* rays, lrt_hit* hits, uint64_t n, void* stream_p,
                             uint32_t flags)
{
  if (!s) return LRT_ERR_INVALID_ARGUMENT;
  if (!s->committed || !s->dev) return fail(s, LRT_ERR_NOT_COMMITTED, "trace before CommitScene/upload");
  if (n == 0) return LRT_OK;
  if (!rays || !hits) return fail(s, LRT_ERR_INVALID_ARGUMENT, "lrt_trace_nearest: NULL rays or hits");
  lrt_status st = check_preset(s);
  if (st != LRT_OK) return st;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_p);
  StreamSlot* slot = nullptr;
  st = slot_for(s, stream, &slot);
  if (st != LRT_OK) return st;
  DeviceScene* d = s->dev;
  if (flags & LRT_TRACE_DEVICE_POINTERS) {
    if ((reinterpret_cast<uintptr_t>(rays) | reinterpret_cast<uintptr_t>(hits)) & 15)
      return fail(s, LRT_ERR_INVALID_ARGUMENT, "device rays/hits must be 16-byte aligned");
    // A trace whose warps take 32 rays each (rays_per_warp) and that repeats
    // the previous trace's ray count on this stream (a renderer's frames) goes
    // through the image-order kernel as an image 8 rays wide, whose 8x4 tiles are the same
    // 32 consecutive rays: the groups are then handed out in the stream's
    // schedule for this ray count (slowest groups first, the slowest split
    // over 2 to 8 warps when the previous launch was tail-bound).  Traces of
    // changing counts keep plain row order and allocate no schedule.
    uint64_t& last = d->lastRays[stream];
    const bool repeat = last == n;
    last = n;
    if (repeat && !(flags & (LRT_TRACE_COUNT_WORK | LRT_TRACE_NATURAL_ORDER)) && rays_per_warp(n, d->S.sms) == 32 &&
        (n + 7) / 8 <= 0xFFFFFFFFull)
      return launch(s, reinterpret_cast<const float4*>(rays), hits, n, stream, flags, slot, 8, uint32_t((n + 7) / 8));
    return launch(s, reinterpret_cast<const float4*>(rays), hits, n, stream, flags, slot);
  }
  if (n <= kStageMaxRays && !(flags & LRT_TRACE_COUNT_WORK) && pageable(rays) && pageable(hits) && host_stage(d, n))
    return trace_host_staged(s, rays, hits, n, stream, flags, slot);
  if (n > d->cap) {
    if (d->rays) cudaFree(d->rays);
    if (d->hits) cudaFree(d->hits);
    d->rays = nullptr;
    d->hits = nullptr;
    d->cap = 0;
    cudaError_t e = cudaMalloc(&d->rays, n * 32);
    if (e == cudaSuccess) e = cudaMalloc(&d->hits, n * sizeof(lrt_hit));
    if (e != cudaSuccess) return cuda_fail(s, e, "staging buffers");
    d->cap = n;
  }
  if (n >= kPipeMinRays && !(flags & LRT_TRACE_COUNT_WORK)) return trace_host_pipelined(s, rays, hits, n, stream, flags);
  cudaError_t e = cudaMemcpyAsync(d->rays, rays, n * 32, cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return cuda_fail(s, e, "rays host->device");
  st = launch(s, d->rays, d->hits, n, stream, flags, slot);
  if (st != LRT_OK) return st;
  e = cudaMemcpyAsync(hits, d->hits, n * sizeof(lrt_hit), cudaMemcpyDeviceToHost, stream);
  if (e != cudaSuccess) return cuda_fail(s, e, "hits device->host");
  return finish(s, stream, slot, (flags & LRT_TRACE_COUNT_WORK) != 0);
}

lrt_status lrt_trace_nearest_image(lrt_scene* s, const float* rays_dev, lrt_hit* hits_dev, uint32_t width,
                                   uint32_t height, void* stream_p, uint32_t flags)
{
  if (!s) return LRT_ERR_INVALID_ARGUMENT;
  if (!s->committed || !s->dev) return fail(s, LRT_ERR_NOT_COMMITTED, "trace before CommitScene/upload");
  if (width == 0 || height == 0) return LRT_OK;
  if (!rays_dev || !hits_dev || ((reinterpret_cast<uintptr_t>(rays_dev) | reinterpret_cast<uintptr_t>(hits_dev)) & 15))
    return fail(s, LRT_ERR_INVALID_ARGUMENT, "lrt_trace_nearest_image: rays/hits must be 16-byte aligned device memory");
  lrt_status st = check_preset(s);
  if (st != LRT_OK) return st;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_p);
  StreamSlot* slot = nullptr;
  st = slot_for(s, stream, &slot);
  if (st != LRT_OK) return st;
  return launch(s, reinterpret_cast<const float4*>(rays_dev), hits_dev, uint64_t(width) * height, stream, flags, slot,
                width, height);
}

// Waits for the stream's traces and reports a bounded-loop limit hit by any of
// them (device-pointer traces are asynchronous).
lrt_status lrt_trace_sync(lrt_scene* s, void* stream_p, int32_t read_counters)
{
  if (!s) return LRT_ERR_INVALID_ARGUMENT;
  if (!s->dev) return fail(s, LRT_ERR_NOT_COMMITTED, "no device scene");
  StreamSlot* slot = nullptr;
  lrt_status st = slot_for(s, static_cast<cudaStream_t>(stream_p), &slot);
  if (st != LRT_OK) return st;
  return finish(s, static_cast<cudaStream_t>(stream_p), slot, read_counters != 0);
}

lrt_status lrt_ray_query_nearest_hit(lrt_scene* s, const float pn[4], const float df[4], lrt_hit* out)
{
  if (!s || !pn || !df || !out) return fail(s, LRT_ERR_INVALID_ARGUMENT, "RayQuery_NearestHit: NULL argument");
  float ray[8];
  std::memcpy(ray, pn, 16);
  std::memcpy(ray + 4, df, 16);
  return lrt_trace_nearest(s, ray, out, 1, nullptr, 0);
}

lrt_status lrt_ray_query_any_hit(lrt_scene* s, const float pn[4], const float df[4], int32_t* out)
{
  if (!s || !pn || !df || !out) return fail(s, LRT_ERR_INVALID_ARGUMENT, "RayQuery_AnyHit: NULL argument");
  // BVH2Common.cpp:3394-3399: negate tfar to request stop-on-first-hit
  float d2[4] = {df[0], df[1], df[2], -df[3]};
  lrt_hit h;
  lrt_status st = lrt_ray_query_nearest_hit(s, pn, d2, &h);
  if (st != LRT_OK) return st;
  *out = h.geomId != 0xFFFFFFFFu;
  return LRT_OK;
}

lrt_status lrt_set_voxel_step_limit(lrt_scene* s, uint32_t steps)
{
  if (!s) return LRT_ERR_INVALID_ARGUMENT;
  s->voxelStepCap = steps;
  return LRT_OK;
}

lrt_status lrt_get_work_counters(lrt_scene* s, uint64_t counters[LRT_COUNTER_COUNT])
{
  if (!s || !counters) return LRT_ERR_INVALID_ARGUMENT;
  std::memcpy(counters, s->counters, sizeof(s->counters));
  return LRT_OK;
}

lrt_status lrt_generate_eye_rays(lrt_scene* s, const lrt_camera* cam, float* rays_dev, void* stream)
{
  if (!cam || !rays_dev) return fail(s, LRT_ERR_INVALID_ARGUMENT, "lrt_generate_eye_rays: NULL argument");
  if (reinterpret_cast<uintptr_t>(rays_dev) & 15)
    return fail(s, LRT_ERR_INVALID_ARGUMENT, "rays must be 16-byte aligned");
  DevCamera c;
  std::memcpy(c.proj_inv, cam->proj_inv, sizeof(c.proj_inv));
  std::memcpy(c.world_view_inv, cam->world_view_inv, sizeof(c.world_view_inv));
  c.width = cam->width;
  c.height = cam->height;
  c.tnear = cam->tnear;
  c.tfar = cam->tfar;
  cudaError_t e = lrt_exact::launch_eye_rays(c, reinterpret_cast<float4*>(rays_dev), static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return s ? cuda_fail(s, e, "eye rays") : LRT_ERR_CUDA;
  return LRT_OK;
}

} // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free trace (lrt_trace_nearest_noalloc)
//
// For callers that cannot call cudaMalloc once their scene is uploaded: a host
// application that hands the whole GPU memory budget to its own pool, or that
// forbids device allocation inside its frame loop.  The trace kernel's
// scratch — the persistent grid's ray counter, the work counters and the
// bounded-loop error word — and, for host buffers, the staging copies of the
// rays and hits live in one file-scope __device__ array instead of memory
// from cudaMalloc.  Its size is fixed: 256 bytes of launch state plus room for
// kNoAllocMaxRays rays and hits (1 MiB + 256 B in all).  A device holds it
// from the first scene upload on that device (which looks its address up)
// until the process exits.
// ---------------------------------------------------------------------------
namespace {

constexpr uint64_t kNoAllocMaxRays = 16384; // host-buffer calls: rays per call
constexpr size_t kNoAllocStateBytes = 256;  // one StreamSlot, padded
constexpr size_t kNoAllocBytes = kNoAllocStateBytes + kNoAllocMaxRays * (32 + sizeof(lrt_hit));
static_assert(sizeof(lrt::StreamSlot) <= kNoAllocStateBytes, "launch state fits its 256 bytes");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

} // namespace

// The array's device address for the current device.  The symbol's name is
// only a host-side stand-in for the array and must never reach a kernel.
cudaError_t lrt::noalloc_scratch_address(void** p) { return cudaGetSymbolAddress(p, g_noalloc_scratch); }

extern "C" lrt_status lrt_trace_nearest_noalloc(lrt_scene* s, const float* rays, lrt_hit* hits, uint64_t n,
                                                void* stream_p, uint32_t flags)
{
  using namespace lrt;
  if (!s) return LRT_ERR_INVALID_ARGUMENT;
  if (!s->committed || !s->dev) return fail(s, LRT_ERR_NOT_COMMITTED, "trace before CommitScene/upload");
  if (n == 0) return LRT_OK;
  if (!rays || !hits) return fail(s, LRT_ERR_INVALID_ARGUMENT, "lrt_trace_nearest_noalloc: NULL rays or hits");
  if (flags & LRT_TRACE_COUNT_WORK)
    return fail(s, LRT_ERR_INVALID_ARGUMENT, "lrt_trace_nearest_noalloc: LRT_TRACE_COUNT_WORK is not supported");
  const bool onDevice = (flags & LRT_TRACE_DEVICE_POINTERS) != 0;
  if (!onDevice && n > kNoAllocMaxRays)
    return fail(s, LRT_ERR_INVALID_ARGUMENT,
                "lrt_trace_nearest_noalloc: %llu rays exceed the static scratch capacity of %llu rays per call",
                (unsigned long long)n, (unsigned long long)kNoAllocMaxRays);
  if (onDevice && ((reinterpret_cast<uintptr_t>(rays) | reinterpret_cast<uintptr_t>(hits)) & 15))
    return fail(s, LRT_ERR_INVALID_ARGUMENT, "device rays/hits must be 16-byte aligned");
  lrt_status st = check_preset(s);
  if (st != LRT_OK) return st;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(s, e, "cudaGetDevice");
  if (dev != s->device)
    return fail(s, LRT_ERR_INVALID_ARGUMENT,
                "lrt_trace_nearest_noalloc: make the scene's device (%d) current, not %d", s->device, dev);
  if (!s->dev->noallocBase)
    return fail(s, LRT_ERR_CUDA, "lrt_trace_nearest_noalloc: the static scratch array was not found at upload: %s",
                cudaGetErrorString(s->dev->noallocErr));
  unsigned char* base = s->dev->noallocBase;
  StreamSlot* slot = reinterpret_cast<StreamSlot*>(base);
  float4* srays = reinterpret_cast<float4*>(base + kNoAllocStateBytes);
  lrt_hit* shits = reinterpret_cast<lrt_hit*>(base + kNoAllocStateBytes + kNoAllocMaxRays * 32);
  cudaStream_t stream = static_cast<cudaStream_t>(stream_p);
  DeviceScene* d = s->dev;
  DevScene S = d->S;
  S.flags = launch_flags(s);
  S.voxelStepCap = s->voxelStepCap ? s->voxelStepCap : kMaxVoxelSteps;
  // the array keeps the previous call's contents: the ray counter and the
  // error word must start at zero
  e = cudaMemsetAsync(slot, 0, sizeof(StreamSlot), stream);
  if (e != cudaSuccess) return cuda_fail(s, e, "cudaMemsetAsync(static scratch)");
  const float4* krays = onDevice ? reinterpret_cast<const float4*>(rays) : srays;
  lrt_hit* khits = onDevice ? hits : shits;
  if (!onDevice) {
    e = cudaMemcpyAsync(srays, rays, n * 32, cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return cuda_fail(s, e, "rays host->static scratch");
  }
  const uint64_t warps = (n + 31) / 32;
  const int blocks = blocks_for(warps);
  if (flags & LRT_TRACE_FAST_MATH)
    e = lrt_fast::launch_trace(S, krays, khits, n, &slot->work, slot->counters, &slot->err, d->stackCap, blocks,
                               stream, false);
  else
    e = lrt_exact::launch_trace(S, krays, khits, n, &slot->work, slot->counters, &slot->err, d->stackCap, blocks,
                                stream, false);
  if (e != cudaSuccess) return cuda_fail(s, e, "trace launch");
  if (!onDevice) {
    e = cudaMemcpyAsync(hits, shits, n * sizeof(lrt_hit), cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return cuda_fail(s, e, "hits static scratch->host");
  }
  uint32_t err = 0;
  e = cudaMemcpyAsync(&err, &slot->err, sizeof(err), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(s, e, "trace");
  if (err)
    return fail(s, LRT_ERR_DEVICE_LIMIT,
                "trace hit a bounded-loop limit (error bits 0x%x: 1 = stack, 2 = voxel march, 4 = transparency layers)", err);
  return LRT_OK;
}
