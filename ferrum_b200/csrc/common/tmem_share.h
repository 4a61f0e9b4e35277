// Which CTAs with tensor memory may share an SM.  tcgen05.alloc waits, without a limit, until the columns are there, and the
// CTAs of a cluster keep theirs until all of them have met.  Two clusters that shared two SMs, each with one CTA holding the
// columns the other's partner waits for, would wait for ever (kernels of two streams run side by side).  So whatever holds
// tensor memory over a cluster barrier takes at least kClusterLeastSmem of shared memory, and a kernel whose clusters take so
// many columns that another such CTA could not allocate beside it takes the rest: the two do not fit one SM.
#pragma once

namespace fb {

constexpr int kSmSmem = 228 * 1024, kCtaSmem = 1024;  // shared memory of an SM, and what every CTA takes besides its own
constexpr int kClusterLeastSmem = 64 * 1024;
constexpr int kClusterAloneSmem = kSmSmem - kClusterLeastSmem - 2 * kCtaSmem + 1024;

}  // namespace fb
