// fft_lengths.cuh -- the line lengths of the built-in passes: all 2, 3, 5,
// 7-smooth ones 24 .. 512 (build.py compiles fft_len.cu for each of them).
#pragma once

#define CRAVA_LINE_LENGTHS(X) \
  X(24) X(25) X(27) X(28) X(30) X(32) X(35) X(36) X(40) X(42) X(45) X(48) \
  X(49) X(50) X(54) X(56) X(60) X(63) X(64) X(70) X(72) X(75) X(80) X(81) \
  X(84) X(90) X(96) X(98) X(100) X(105) X(108) X(112) X(120) X(125) X(126) X(128) \
  X(135) X(140) X(144) X(147) X(150) X(160) X(162) X(168) X(175) X(180) X(189) X(192) \
  X(196) X(200) X(210) X(216) X(224) X(225) X(240) X(243) X(245) X(250) X(252) X(256) \
  X(270) X(280) X(288) X(294) X(300) X(315) X(320) X(324) X(336) X(343) X(350) X(360) \
  X(375) X(378) X(384) X(392) X(400) X(405) X(420) X(432) X(441) X(448) X(450) X(480) \
  X(486) X(490) X(500) X(504) X(512)
