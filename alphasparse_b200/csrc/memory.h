// Device memory of plans and copies from and to host memory.
#ifndef ASP_MEMORY_H
#define ASP_MEMORY_H

#include <cuda_runtime.h>
#include <stddef.h>

#include <mutex>
#include <vector>

namespace asp
{
// Device memory for plans. cudaMalloc and cudaFree of a plan's arena take one to three milliseconds each on this part, more than
// everything else that makes a small plan; freed arenas are therefore kept for the next plan: blocks of at most 256 MB, 1 GB in
// all per device (the longest idle ones go first), given back when the last context of the device is destroyed, by device_trim(), or when
// an allocation of this library fails. Safe from several threads.
// device_free() waits for the device first, as cudaFree does: kernels in flight may still read the block.
// `spare`: fails where an allocation would leave less than that (0: does not look).
cudaError_t device_alloc(int device, size_t bytes, void **out, size_t *got, size_t spare = 0);
void device_free(int device, void *p, size_t got) noexcept;
// cudaMalloc, a second time without idle blocks if the first fails: for whatever does not come from the pool
cudaError_t device_malloc(int device, size_t bytes, void **out);
bool device_has_room(int device, size_t bytes); // free or kept idle by the pool
void device_trim(int device);
void device_pool_retain(int device);  // a context was created ...
void device_pool_release(int device); // ... or destroyed

// What the device calls [p, p + bytes) of host memory, where all of it lies in one page-locked range that the device may write, else NULL. (The
// ends alone do not say it: a buffer may begin in one registered range and end in another.)
void *device_view(const void *p, size_t bytes);

// Copies between pageable host memory and the device. The runtime moves such a copy through its own pinned buffer with one
// thread (8 to 12 GB/s measured, page faults of a fresh destination included); here all cores fill or empty a ring of pinned
// pieces while the copy engine works on the others. Pinned memory is copied directly. 16 MB per context, allocated with the
// first copy that is worth it, freed with the context.
class Stager
{
    static const size_t kPiece = 1u << 20;
    static const int kPieces = 16;
    std::mutex one; // copies of several threads take turns: they share the ring
    unsigned char *ring = nullptr;
    cudaEvent_t done[kPieces] = {};
    int owner[kPieces] = {}; // event that a slot is free after
    bool off = false; // no pinned memory to be had: plain copies
    int next = 0;

    bool ready();
    // the adjacent slots that the next piece goes through, free to be written, and the event to record after its copy
    cudaError_t take(int slots, unsigned char **p, int *event);
    bool free_now(int slots) const;

  public:
    static bool pinned(const void *host);
    struct Segment
    {
        size_t off;
        const void *host;
        size_t bytes;
    };
    void release();
    // host buffers may be reused as soon as these return, as after a pageable cudaMemcpyAsync
    cudaError_t to_device(void *dev, const void *host, size_t bytes, cudaStream_t st);
    // the same in pieces of about `piece` bytes; sent.f(sent.with, n) is called when the copies of the first n bytes are on the stream. An
    // error of it ends the copy.
    struct Sent
    {
        cudaError_t (*f)(void *, size_t);
        void *with;
    };
    cudaError_t to_device(void *dev, const void *host, size_t bytes, cudaStream_t st, size_t piece, const Sent &sent);
    // many arrays of one device block (ascending offsets): as few copies as the pieces make
    cudaError_t to_device(void *dev, const std::vector<Segment> &segments, cudaStream_t st);
    cudaError_t to_device(void *dev, const Segment *segments, size_t count, cudaStream_t st, size_t piece = 0, const Sent *sent = nullptr);
    // complete on return
    cudaError_t to_host(void *host, const void *dev, size_t bytes, cudaStream_t st);
};
} // namespace asp
#endif
