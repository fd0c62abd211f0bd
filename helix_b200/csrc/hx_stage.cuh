// hx_stage.cuh -- moving large pageable host buffers to and from the device (hx_stage.cu).
#pragma once
#include "hx_common.cuh"

// One copy of a batch: pageable host memory on one side.
struct HxCopy { void* dev; void* host; size_t bytes; };

// Exclusive use of the current device's staging area (page-locked slots, copy streams, device workspace) for the duration of
// one call.  A second caller waits.
class HxStage {
public:
    HxStage();
    ~HxStage();                                  // gives the area back to the next caller
    int status() const { return rc_; }           // HX_OK or the error of the set-up
    cudaStream_t stream() const;                 // work between an upload and a download goes here
    int workspace(void** dptr, size_t bytes);    // device memory, valid until the object ends
    int upload(const HxCopy* c, int n);          // later work on stream() sees the data; the host buffers have been read
    int download(const HxCopy* c, int n);        // what stream() has produced so far; the host buffers have been written
private:
    struct HxStageArea* a_;
    int rc_;
    bool big_ = false, open_ = false;            // open_: copies may be in flight
    int run(const HxCopy* c, int n, bool up);
};

// cudaMalloc on the current device; where memory is short the idle staging area gives its workspace back first.  Leaves no error
// behind for the next launch check.
cudaError_t hx_dev_malloc(void** p, size_t bytes);
