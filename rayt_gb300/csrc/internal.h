// Internal declarations shared by the host C++ and the CUDA translation units.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>
#include "../../include/rayt_gb300.h"

namespace rayt {

// ---- errors -----------------------------------------------------------------
void set_error(const std::string& msg);
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);
#define RAYT_CUDA_TRY(expr)                                   \
  do {                                                        \
    cudaError_t e_ = (expr);                                  \
    if (e_ != cudaSuccess) return ::rayt::cuda_fail(e_, #expr); \
  } while (0)

constexpr int32_t kNoHit = 0x7fffffff;
constexpr uint32_t kRootParent = (1u << 24) - 1;

// Waits until a kernel of stream s has set the host-mapped *word to `value`,
// which is the last thing it does; everything queued on s before that kernel is
// done then.  Or, given `early`, until early(arg).
int wait_word(const unsigned int* word, unsigned int value, cudaStream_t s, bool (*early)(const int*) = nullptr,
              const int* arg = nullptr);

// ---- traversal ----------------------------------------------------------------
// Views' images (and recorded feedback words) share one buffer; view v starts
// at pixel pix_base (a multiple of 64).  A ray is identified by its pixel's
// index in that buffer, below 2^30.
constexpr int kMaxViews = 512;
constexpr int kViewsPerLaunch = 64;   // view descriptors travel in the launch parameters
constexpr int kMaxClients = 64;       // served mode: client framebuffers per server

// One view of a tracing launch.
struct ViewDesc {
  float m[16];             // view_proj_inv, row-major
  int width, height;
  int tiles_x;             // columns of 32-pixel tiles
  uint32_t tiles_x_inv;    // reciprocal(tiles_x)
  int tile_base;           // first tile of this view in the launch's tile space
  float lod;               // lod_voxel_size
  int pix_base;            // first pixel of the view in the shared image buffer
  float origin[4];         // InitTracingFrame's ray origin (m[2], m[6], m[10], 0) / m[14], per view
  const float* coords;     // PixelCoords(width, height) in device memory
};

// InitTracingFrame's normalised pixel coordinates, which depend only on the
// view's size: centres (x + 0.5) / W * 2 - 1 for x in [0, W), corners
// x / W * 2 - 1 for x in [0, W], then the same for y.  Computed once on the
// host with IEEE float arithmetic (the same operations and rounding as the
// kernel would do per ray), so looking them up changes no bit.
size_t pixel_coords_count(int w, int h);
void pixel_coords(int w, int h, float* out);
// The per-view origin the same way: (m[2], m[6], m[10], 0) / m[14].
void view_origin(const float* m, float* origin);

// Words of a pass: its counters, then the flags for rays without a feedback
// word, one per 128-byte line (a warp sets the flag of its CTA's number: one
// flag for all took a launch's warps, ending together, 5 ns each).  A tracing
// state is two of these and the feedback bitmaps: a pass counts into one of
// the two and reads the rays of the pass before from the other, and its unique
// kernel leaves the other and the bitmaps zero for the pass after it.
constexpr int kNoWordFlags = 32, kNoWordStride = 32;
struct PassState {
  int rays;                // rays appended to the output list
  int pad;
  unsigned long long start_ns;  // when the pass's traversal began
  int work[12];            // persistent kernel: work counter per launch
  int no_word[kNoWordFlags * kNoWordStride];
};
constexpr int kPassInts = sizeof(PassState) / 4;

// Parameters of a traversal launch but for its views.
struct TraceCore {
  // cache (the reference's cache format)
  const uint32_t* links;
  const uint32_t* far_ptrs;
  const char4* normals;    // may be null
  const uchar4* colors;    // may be null
  uint32_t root;           // node index of the root (cache node indices are unsigned 32-bit)
  int nodes_in_block;
  int block_shift;         // log2(nodes_in_block), -1 when it is no power of two
  uint32_t node_limit;     // nodes in the cache (max_blocks * nodes_in_block)
  uint32_t far_limit;      // far pointers in the cache (max_blocks * 8)
  uchar4 empty_pixel;      // a pixel that shows the background
  // outputs of every view
  uchar4* image;           // RGBA8, row 0 of each view at the bottom
  uchar4* host_image;      // optional: the same pixels also written here (page-locked host memory)
  int32_t* words_dense;    // optional per-pixel feedback words (recording)
  // first pass: the views of this launch and their tiles (32 rays each)
  int n_views;
  int total_tiles;
  int tile_w_log2;         // a warp's 32 first-pass rays cover (1 << tile_w_log2) x (32 >> tile_w_log2) pixels
  // faulted rays carried between passes: record i of the input list, and the
  // output list the rays that fault in this pass are appended to
  const float4* in_origin;
  const float4* in_dir;
  const int* in_parent;
  const uint32_t* in_ray;
  const int* n_in;
  float4* out_origin;      // xyz origin, w LOD bias
  float4* out_dir;         // xyz direction, w LOD coefficient
  int* out_parent;
  uint32_t* out_ray;
  // optional depth output (all four set, or all null): per pixel the distance
  // along the ray to what it shows and the cache node that shaded it; records
  // carry the distance a faulted ray advanced so far
  float* depth;
  int32_t* hit_node;
  const float* in_adv;
  float* out_adv;
  // feedback
  uint32_t* fault_bits;    // one bit per tree block
  int fault_bit_limit;     // number of tree blocks (bits in fault_bits)
  uint32_t* hit_bits;      // bit 2*cache_block + dup
  PassState* words;        // of this pass
  bool stamp;              // the launch notes when the pass began
  unsigned long long* counters;  // optional: rays, link fetches, far fetches, iterations, hits, faults
  // served mode (zero in the per-frame path).  Client slot i owns the pixels
  // [client_base[i], client_base[i + 1]) of the image buffer.
  int restart;             // faulted rays are recorded with their camera origin and traced afresh
  int n_clients;
  int client_base[kMaxClients + 1];
  unsigned long long finish_mask;  // continuation rays of these slots are finished, not traced
  int* client_faults;      // per slot: rays that faulted in this pass
  // persistent kernels
  int* work;               // persistent kernel: work counter, zero before the launch
  int refill;              // idle lanes that let a warp take new rays (< 32)
  int step_budget;         // iterations a warp runs between refill checks
  int lanes;               // rays per warp (a power of two; see trace_lanes)
};
struct TraceParams : TraceCore {
  ViewDesc views[kViewsPerLaunch];
};
// What a launch of one view (or of no views: later passes) carries: parameters
// of 9 KB cost the host 3 us more per graph launch than these.
struct TraceParams1 : TraceCore {
  ViewDesc views[1];
};

// ceil(2^32 / d), or the largest word for d = 1 (see first_pass_pixel).
inline uint32_t reciprocal(int d) { return d > 1 ? (uint32_t)(((1ull << 32) + (uint32_t)d - 1) / (uint32_t)d) : ~0u; }
inline int log2_or_minus_one(int v) { return v > 0 && (v & (v - 1)) == 0 ? __builtin_ctz((unsigned)v) : -1; }
// FinishTracingFrame's pixel where nothing was hit, over background bg.
uchar4 finish_empty(const float* bg);
// The reference's background (gpu-ray-tracer.cpp:190).
constexpr float kBackground[4] = {0.0f, (float)(216 / 255.), 1.0f, 1.0f};

// Frames on their way to host memory: image k goes to `host` when no ray of its
// client faulted (faults[slot] == 0), else nothing happens.
struct DeliverParams {
  int images;
  const int* faults;
  struct {
    const uchar4* image;
    uchar4* host;  // device address of page-locked memory
    int64_t pixels;
    int slot;
  } at[kMaxClients];
};
cudaError_t launch_deliver(const DeliverParams& p, cudaStream_t s);

// Faulted-ray records carried from one pass to the next (device arrays).
struct RayList {
  float4* origin = nullptr;  // xyz advanced to the fault, w LOD bias
  float4* dir = nullptr;     // xyz direction, w LOD coefficient
  int* parent = nullptr;     // node the ray faulted under
  uint32_t* ray = nullptr;   // pixel index in the image buffer
  float* adv = nullptr;      // distance advanced over earlier passes (depth output only)
};

// first: rays come from the views' cameras (refill = 32: one lane per ray of
// the `rays` = total_tiles * 32; refill < 32: the persistent work-stealing
// kernel over `grid` CTAs, 0 = as many as are resident).  Otherwise the `rays`
// faulted rays of the input list, one lane each.
// Rays per warp (TraceParams::lanes) for a launch over `rays` rays.
int trace_lanes(bool first, int rays);
cudaError_t launch_trace(const TraceParams& p, bool first, bool count, int rays, int grid, cudaStream_t s);
// The same launch as a kernel node of a CUDA graph; l must stay valid until the
// node is added or updated.
struct TraceLaunch {
  TraceParams1 one;       // p, when it has at most one view
  void* args[1];
  cudaKernelNodeParams kp;
};
void trace_node_params(const TraceParams* p, bool first, bool count, int rays, int grid, TraceLaunch* l);
// Resident CTAs of the persistent traversal kernel on the current device.
int trace_persistent_grid(bool count);
cudaError_t launch_finish(const TraceCore& p, int max_rays, cudaStream_t s);
cudaError_t launch_fill_i32(int* p, int32_t v, size_t n, cudaStream_t s);
// The reference's debug depth view (raytracer.cl) of views[0] into image.
cudaError_t launch_depth_view(const TraceParams1& p, cudaStream_t s);

// Feedback bitmaps -> the reference's sorted unique array, in host-mapped
// memory; clears the tracing state for the next pass (see PassState) and ends
// by publishing the pass's number, so that the host need not wait for the
// stream.
struct UniqueResult {     // host-mapped
  int unique, faults;     // unique count (incl. NO_HIT), fault count
  int rays;               // rays the pass appended to its output list
  float trace_ms, unique_ms;
  int client_faults[kMaxClients];
  unsigned int pass;      // passes done; written last
};
struct UniqueFromBitsParams {
  uint32_t* fault_bits;
  int fault_words;
  uint32_t* hit_bits;
  int hit_words;
  PassState* words;      // of this pass
  PassState* previous;   // of the pass before
  bool later;            // the pass traced the rays of the pass before (pixels without one have no word)
  int total_pixels;
  const int* client_faults;  // served mode: per client, copied; may be null
  int* next_client_faults;   // and the next tick's, cleared
  unsigned int* passes;  // passes done, on the device
  int32_t* unique_out;   // room for fault bits + hit bits + 1
  UniqueResult* result;
};
cudaError_t launch_unique_from_bits(const UniqueFromBitsParams& p, cudaStream_t s);
cudaError_t unique_node_params(const UniqueFromBitsParams* q, void** args, cudaKernelNodeParams* kp);


// ---- radix sort / scan / unique -------------------------------------------------
// Memory of a call: `scratch` (any contents), `status` (look-back words, zero or
// left by earlier calls), `result` and `err` (device or mapped host memory the
// host reads once the stream has finished).  `epoch` (27 bits, from
// lookback_epoch_step) tags the call's look-back words.  err becomes 1 when a
// bounded wait gave up.
// `done`: the call's last kernel sets *flag (host-mapped) to `number` when all its
// CTAs have ended; what the call wrote is visible then.  *ctas is zero before
// and after.  flag null: nothing is published.
struct DoneFlag {
  int* ctas = nullptr;
  unsigned int* flag = nullptr;
  unsigned int number = 0;
};
size_t feedback_scratch_bytes(int n);
size_t feedback_status_bytes(int n);
// Compaction (drop NO_HIT, NodeToBlock) and sorted unique.  result[0] receives
// the unique count (incl. NO_HIT), unless the keys span too wide a range for a
// bitmap: feedback_unique_needs_radix(result) says so, and
// feedback_unique_radix_device, on the same memory, then sorts them.  In mapped
// host memory, where the caller has cleared it, result says so as soon as that
// is known, and the second may be launched behind the rest of the first.
cudaError_t feedback_unique_device(const int32_t* words, int n, int nib, int32_t* unique_out, void* scratch,
                                   unsigned long long* status, uint32_t epoch, int* result, int* err,
                                   const DoneFlag& done, cudaStream_t s);
bool feedback_unique_needs_radix(const int* result);
cudaError_t feedback_unique_radix_device(int n, int32_t* unique_out, void* scratch, unsigned long long* status,
                                         uint32_t epoch, int* result, int* err, const DoneFlag& done,
                                         cudaStream_t s);
size_t sort_scratch_bytes(int n);
size_t sort_status_bytes(int n);
// Sorts in place; or, where *again (mapped host memory, cleared by the caller) is
// set, sort_needs_passes(again), leaves some order of the same keys, which
// sort_passes_device, on the same memory, then sorts.
cudaError_t sort_i32_device(int32_t* data, int n, void* scratch, unsigned long long* status, uint32_t epoch,
                            int* again, int* err, const DoneFlag& done, cudaStream_t s);
bool sort_needs_passes(const int* again);
cudaError_t sort_passes_device(int32_t* data, int n, void* scratch, unsigned long long* status, uint32_t epoch,
                               int* err, const DoneFlag& done, cudaStream_t s);
size_t scan_status_bytes(int n);
cudaError_t scan_i32_device(int32_t* data, int n, unsigned long long* status, uint32_t epoch, int* err,
                            const DoneFlag& done, cudaStream_t s);

// ---- stand-alone primitives (prims.cpp) -------------------------------------------
// Serialises every sort/scan/unique entry point on all devices: they share
// scratch memory and the look-back epoch, and each one holds the lock until
// its stream has finished its work.
std::mutex& prims_mutex();
// Called (with prims_mutex held) before each call on the current device: its
// epoch.  Before the epoch would repeat a tag still present in a look-back
// table (after 2^27 - 1 calls), clears every look-back table of the device on
// s and restarts at 1.
int lookback_epoch_step(cudaStream_t s, uint32_t* epoch);
// Registers a look-back table on the current device besides the library's own
// (the allocation-free entry point's static array), so lookback_epoch_step
// clears it too.
void register_lookback_area(void* p, size_t bytes);
// Runs one wait on a word nothing publishes, with a limit of limit_s seconds
// (restored to 1 s after); the wait must give up and set *err.
cudaError_t bounded_wait_probe(double limit_s, int* err, cudaStream_t s);

// ---- block upload --------------------------------------------------------------
constexpr int kMaxChannels = 8;
// A batch of up to this many blocks, and of patches, carries its slots, block
// numbers and patch records in the launch parameters.
constexpr int kInlineBlocks = 128, kInlinePatches = 256;
// Device time of the batches, in device memory: a batch's last kernel adds the
// batch's.
struct UploadClock {
  unsigned long long start_ns;  // of the batch under way
  unsigned long long total_ns;  // of the batches done
  unsigned long long* host;     // total_ns in host-mapped memory
};
struct UploadParams {
  const uint8_t* stage;        // block contents, `stride` bytes apart
  size_t stride;               // content bytes rounded up to 16 (keeps every block aligned)
  const int* slots;            // destination cache slot per staged block
  int blocks;
  int nodes_in_block;
  int channels;
  int chan_bytes[kMaxChannels];
  uint8_t* chan[kMaxChannels]; // channel 0 = node links
  // With `file` set, the contents are read where they lie in the mapped block
  // file instead of from `stage`: block b's content starts at
  // file + file_first + file_stride * block_ids[b], at any alignment.
  const uint8_t* file;
  uint64_t file_first;         // header bytes + the 76-byte block header
  uint64_t file_stride;
  const int* block_ids;
  UploadClock* clock;          // mapped reads: the batch's beginning is noted here
  int parts;                   // CTAs per block (mapped reads; set by launch_upload)
  // mapped reads of blocks whose channel sections are whole words: the word at
  // which each section begins, and the content's words (0: other blocks)
  uint32_t section[kMaxChannels + 1];
};
struct Patch {
  uint32_t index;  // node-link index (below 2^32) or far-pointer index
  uint32_t value;
  uint32_t far;    // 1: far-pointer buffer, 0: node-link buffer
};
// `host_slots` and `host_blocks`: the batch's slots and block numbers in host
// memory (mapped reads).
cudaError_t launch_upload(const UploadParams& p, const int* host_slots, const int* host_blocks, cudaStream_t s);
// n patches, in host memory when there are at most kInlinePatches, else at the
// device address `patches`.  `clock`: this ends the batch.
cudaError_t launch_patches(const Patch* patches, int n, uint32_t* links, uint32_t* far_ptrs, UploadClock* clock,
                           cudaStream_t s);

// ---- glibc-compatible rand() stream -------------------------------------------
// The additive feedback generator behind glibc's rand()/srand() (TYPE_3:
// r[i] = r[i-3] + r[i-31], 16807 LCG seeding, 310 discarded outputs), as
// published in descriptions of the glibc random() algorithm.
class LibcRand {
 public:
  explicit LibcRand(uint32_t seed = 1) { Seed(seed); }
  void Seed(uint32_t seed);
  int Next();
 private:
  int32_t r_[34];
  int i_ = 0;
};

}  // namespace rayt
