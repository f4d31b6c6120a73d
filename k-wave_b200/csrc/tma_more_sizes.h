// More transform lengths of the TMA-fed column passes, beside tma_sizes.h: the
// lengths above 256, whose line a tensor copy covers as a box of several
// segments (make_spec_map), and the lengths of ct_more_sizes.h.
#pragma once
#include "ct_more_sizes.h"

#define KWB_TMA_LONG_SIZES(X) \
  X(270) X(288) X(300) X(320) X(324) X(360) X(375) X(384) X(400) X(405) X(432) X(450) X(480) X(486) X(500) \
  X(512) X(540) X(576) X(600) X(625) X(640) X(648) X(675) X(720) X(729) X(750) X(768) X(800) X(810) X(864) \
  X(900) X(960) X(972) X(1000) X(1024)
#define KWB_TMA_MORE_SIZES(X) KWB_TMA_LONG_SIZES(X) KWB_CT_MORE_SIZES(X)
