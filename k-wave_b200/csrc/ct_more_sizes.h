// More transform lengths with compile-time FFT kernels, beside ct_sizes.h: the
// lengths from 64 to 1024 with a factor 7 and the 2^a 3^b 5^c 7^d lengths from
// 40 to 63.  On the runtime-plan engine, whose stages ping-pong between two
// shared-memory buffers with run-time index arithmetic, a 112 x 98 x 126
// absorbing step took 493 us.
#pragma once

#define KWB_CT_MORE_SIZES(X) \
  X(40) X(42) X(45) X(48) X(49) X(50) X(54) X(56) X(60) X(63) X(70) X(84) X(98) X(105) X(112) X(126) X(140) \
  X(147) X(168) X(175) X(189) X(196) X(210) X(224) X(245) X(252) X(280) X(294) X(315) X(336) X(343) X(350) \
  X(378) X(392) X(420) X(441) X(448) X(490) X(504) X(525) X(560) X(567) X(588) X(630) X(672) X(686) X(700) \
  X(735) X(756) X(784) X(840) X(875) X(882) X(896) X(945) X(980) X(1008)
