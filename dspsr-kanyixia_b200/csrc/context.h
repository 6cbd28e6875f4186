// context.h -- the library context (one device, one stream, the last error
// message), shared by the translation units that implement the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <memory>
#include <mutex>
#include <string>
#include <vector>

// Status words of the convolutions made on a context (WaitFlag in capi.cu):
// host memory that the device can write, a page at a time (an allocation per
// engine took 1.3 ms of its creation).  Shared with the engines, which may
// outlive their context; the pages go with the last of them.
struct dspsr_b200_wait_words
{
  static constexpr int PER_PAGE = 1024;
  std::mutex lock;
  std::vector<int*> pages, spare, used;
  // a word that reads 0, or null when no page can be had
  int* take ();
  void give (int* word);
  // whether any word in use is set
  bool any_set ();
  ~dspsr_b200_wait_words ();
};

struct dspsr_b200_context
{
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string error;
  float* d_lut = nullptr;     // scratch LUT for the standalone unpacker
  float2* d_fb_tab = nullptr; // pass tables of the standalone filterbank's FFT
  unsigned fb_tab_n = 0;      // ... for this transform length
  std::shared_ptr<dspsr_b200_wait_words> waits;
};

struct dspsr_b200_rfi_proposer;

namespace b200 {
// the context, channels per block and block length a proposer was made for
void rfi_proposer_shape (const dspsr_b200_rfi_proposer* proposer, dspsr_b200_context** ctx,
                         unsigned* nchan, unsigned* M);
} // namespace b200
