/* ff_copy.h -- copies of caller memory into page-locked buffers by several threads. */
#ifndef FF_COPY_H
#define FF_COPY_H

#include <stddef.h>

#ifdef __cplusplus
extern "C" {
#endif

typedef struct ff_copy_pool ff_copy_pool;

/* Helper threads for ff_copy: as many as asked for, but never more than a third of the CPUs the process may run on and
 * at most 3.  The threads start with the first copy that is worth sharing.  NULL when out of memory.  In a process forked
 * from the one that made the pool, ff_copy copies without helpers and ff_copy_pool_destroy does nothing. */
ff_copy_pool* ff_copy_pool_create(int helpers);
void ff_copy_pool_destroy(ff_copy_pool* p);

/* memcpy(dst, src, bytes), shared with the pool's threads from 512 KB up; returns when every byte is in place.  One
 * caller at a time per pool.  p may be NULL (the caller alone).  streaming: the destination is not read by a CPU next
 * (stores that bypass the caches). */
void ff_copy(ff_copy_pool* p, void* dst, const void* src, size_t bytes, int streaming);

#ifdef __cplusplus
}
#endif
#endif
