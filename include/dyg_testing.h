/*
 * dyg_testing.h -- failures that the library's own tests arrange on the host.
 * Nothing here makes a device fail: a wait is given something that never
 * comes and ends at its limit.  No program needs these calls.
 */
#ifndef DYG_TESTING_H
#define DYG_TESTING_H
#include "dyg.h"
#ifdef __cplusplus
extern "C" {
#endif

/* The next grid barrier of a launch on g (more than 16 blocks, or the weighted
 * row index) finds arrivals on its counter that never came, so that its blocks
 * give up after spin_limit reads (> 4096; the default is about a minute's). */
dyg_status dyg_testing_stall_barrier(dyg_graph *g, uint32_t spin_limit);

/* The next prefix scan on g (an export, a compaction) misses its first tile:
 * the others wait for it until their limit. */
dyg_status dyg_testing_stall_scan(dyg_graph *g);

/* Device memory runs short on this host thread: its next `pass` allocations
 * succeed, the `fail` after them do not (an allocation that must not fail is
 * tried twice).  (0, 0) ends it. */
void dyg_testing_fail_allocations(uint32_t pass, uint32_t fail);

#ifdef __cplusplus
}
#endif
#endif /* DYG_TESTING_H */
