// Layouts shared by the kernels and the host code that fills them (int64 words).
#pragma once

namespace pe {

// Per-image descriptors of the batched segmentation / instance kernels, kDescFields words each
// (panoptic_evaluator_gb300/_batch.py builds the same table).
enum DescField : int {
  kTarget = 0,    // segmentation: int32 target slot map; instance: gt masks (uint8)
  kPred,          // int32 prediction slot map (segmentation)
  kMasks,         // detection masks, uint8 0/1, rows `kMaskStride` bytes apart (unsorted order)
  kPixels,
  kMaskStride,
  kChunkBegin,    // first work chunk of this image
  kDetBegin,      // offset into flat per-detection arrays
  kSlotBegin,     // offset into flat per-target-slot arrays
  kPSlotBegin,    // offset into flat per-prediction-slot arrays
  kPairBegin,     // offset of this image's G x P pair histogram
  kDPairBegin,    // offset of this image's D x G detection histogram
  kD,
  kG,
  kP,
  kFlags,         // bit 0: slot maps 16-byte vectorisable; bit 1: masks 16-byte vectorisable
  kReserved,
  kDescFields
};

// Per-image descriptors of pe_prefix (panoptic_evaluator_gb300/prefix.py builds the same table).
enum PrefixField : int {
  kPrefixTarget = 0,   // int32 target slot map
  kPrefixMasks,        // uint8 0/1 masks in generation order, rows kPrefixStride bytes apart
  kPrefixPixels,
  kPrefixStride,
  kPrefixChunkBegin,   // first 4096-pixel chunk of this image
  kPrefixN,            // masks
  kPrefixG,            // target slots
  kPrefixDetBegin,     // offset into flat per-mask arrays (classes) and raw rows / N
  kPrefixSlotBegin,   // offset into flat per-slot arrays (gc, crowd, ga)
  kPrefixQBegin,       // first output row (checkpoint) of this image
  kPrefixQ,            // checkpoints of this image
  kPrefixPairBegin,    // offset of this image's [Q][G][N+1] histograms
  kPrefixRawBegin,     // offset of this image's [N][G] raw intersections
  kPrefixFlags,        // bit 0: target map 16-byte vectorisable, bit 1: mask rows 16-byte vectorisable
  kPrefixStepBegin,    // offset of this image's step table (N+1 entries: checkpoint index or -1)
  kPrefixCountBegin,   // reserved: offset of this image's [T][C][2] counters
  kPrefixFields
};

}  // namespace pe
