// The packed 16-bit SSW kernel (ssw16.cuh).
#pragma once
#include "extend.h"

namespace sa {

constexpr uint32_t SSW16_MAX_QLEN = 511;
// Below this many tasks a block's two warps share a task's byte and word passes.  Both passes
// then always run, so it pays while a launch lasts as long as one task: 2000 pairs to SAM
// (waves of 30 to 500 tasks) 3.46 ms, 4.01 never shared; a session of 24 requests 11.0 and
// 12.0 ms.  Alignment calls, whose tasks have no diagonal, gain up to about 10,000 tasks (4,000
// of 100-300 nt 2.0 and 2.2 ms, 8,000 2.4 and 2.9) and lose beyond (16,000 of 250 nt 2.6 and
// 2.4 ms; 60,000 of 100-300 nt 6.8 and 6.1 ms).  Mapping's larger waves, whose tasks mostly
// have a diagonal that spares them the byte pass, take the same either way (100k pairs to SAM
// within 1 %).  4096 is on the safe side: below it both kinds gain.
constexpr uint32_t SSW16_PAIR_TASKS = 4096;

struct Ssw16Args {
    SswTask* tasks;
    const uint32_t* order;
    uint32_t n_tasks;
    const PrepRec* prep;
    const uint8_t* arena;
    AlignScores sc;
    int bias;
    uint32_t* counters;
    uint32_t qmax;     // tasks of longer reads are left to another kernel
    uint32_t* redo;    // tasks to run again on the warp-per-task kernel, and their count
    uint32_t* n_redo;
    int32_t* hscratch;  // per-job scratch (PrepRec::h_off), for ungapped tasks' CIGARs
    cudaStream_t st;
};

// The longest read whose scores fit (0: these scores do not).  Scores are scaled by 32 in
// 16 bits: match * L <= 1022 keeps every H with its row key below 2^15, and
// gap_extend * ceil(L / 8) <= 1024 the raise above -2^15, which a word pass takes through a
// lane's two pieces from 0 on (match 3, extension 24: reads up to 336 of the 340 nt that the
// scores allow).  The other limits keep the raise's row offsets (gap_extend <= 31, and no
// more than a lane's rows add to the score) and a word pass's first lane of two rows or more
// (a byte pass overflows at 255 - mismatch, which takes 12 rows or more) within what the
// kernel assumes; the lazy-F raise is exact for gap_open > gap_extend.
uint32_t ssw16_max_qlen(const AlignScores& sc);

// The end searches of every task of a read up to a.qmax nt; longest: the longest such read.
void launch_ssw16(const Ssw16Args& a, uint32_t longest);
void launch_ssw16_pair(const Ssw16Args& a, uint32_t longest);

}  // namespace sa
