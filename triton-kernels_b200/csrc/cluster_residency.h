// How many thread-block clusters the GPU holds at once.
#pragma once

namespace b200attn {

// Clusters of `c` CTAs (1, 2, 4 or 8), `per_sm` of them to an SM (1 to 3), that the GPU holds at once.  Those of four and eight leave SMs
// over in each of its processing clusters: a decode call of 16 clusters of eight at one CTA per SM went in two waves and took 20.4 us
// instead of 15.4 planned (two sequences of 4 096 keys, 32/8 heads, D 128).  The driver is asked once (`ask`; the answer depends on the
// device model only); without a GPU the figures are those it gave for a B200.
int clusters_held(int c, int per_sm, int sm_count, bool ask);

}  // namespace b200attn
