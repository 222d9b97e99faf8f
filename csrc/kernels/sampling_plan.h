// Which sampler takes rows of bf16 logits (sampling.cu): one CTA per row, or a cluster of eight.
#pragma once

namespace ogb {

// A cluster finishes a row sooner (one row of 32000, top-p: 63 -> 19 us; of 1024 26 -> 18), but eight CTAs are a fifth of what the chip holds of them: 37 rows
// at a time take 17 us a round whatever their length, where one-CTA rows run 148 or 296 at a time.  us, one CTA -> cluster, flat and sure rows with
// top-p 0.9: 1024 logits 27 -> 37 and 25 -> 35 at 64 rows; 32000 72 -> 41 and 39 -> 37 at 64, 74 -> 84 and 41 -> 78 at 148; 65536 at 148 rows 0.7 and
// 1.2 of the one-CTA time; from 128256 on the cluster is faster at any number of rows (256: 426 -> 203, 199 -> 143).
inline bool sample_cluster_pays(int rows, int vocab) { return rows <= 32 || rows <= vocab / 512 || vocab >= 112 * 1024; }

}  // namespace ogb
