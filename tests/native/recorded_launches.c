/* The CUDA layer as seen by csrc/host/fg_cuda_api.c, without a GPU: launches are written down instead of made,
 * memory is host memory.  What only computes sizes (fgk_team_fits and the like) is the real library's. */
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "fg_kernels.h"

static char record[1 << 16];
static size_t used;

const char *recorded_launches(void) { return record; }
void recorded_clear(void) { record[used = 0] = 0; }

static int note(const char *format, ...) {
    va_list list;
    va_start(list, format);
    const int n = vsnprintf(record + used, sizeof(record) - used, format, list);
    va_end(list);
    if (n > 0 && (size_t)n < sizeof(record) - used) used += (size_t)n;
    return 0;
}

int fgk_device_count(int *count) { *count = 1; return 0; }
int fgk_set_device(int device) { (void)device; return 0; }
int fgk_device_sm_count(int device, int *sm_count) { (void)device; *sm_count = 148; return 0; }
int fgk_stream_create(void **stream) { *stream = NULL; return 0; }
int fgk_stream_destroy(void *stream) { (void)stream; return 0; }
int fgk_stream_synchronize(void *stream) { (void)stream; return 0; }
int fgk_stream_capturing(void *stream, int *capturing) { (void)stream; *capturing = 0; return 0; }
int fgk_malloc(void **pointer, size_t bytes) { *pointer = malloc(bytes); return *pointer ? 0 : 2; }
int fgk_free(void *pointer) { free(pointer); return 0; }
int fgk_host_alloc(void **pointer, size_t bytes) { return fgk_malloc(pointer, bytes); }
int fgk_host_free(void *pointer) { free(pointer); return 0; }
int fgk_memset_async(void *pointer, int value, size_t bytes, void *stream) { (void)stream; memset(pointer, value, bytes); return 0; }
int fgk_copy_to_device_async(void *to, const void *from, size_t bytes, void *stream) { (void)stream; memcpy(to, from, bytes); return 0; }
int fgk_copy_to_host_async(void *to, const void *from, size_t bytes, void *stream) { (void)stream; memcpy(to, from, bytes); return 0; }
const char *fgk_error_string(int e) { (void)e; return "none"; }
int fgk_stream_prepare(void) { return 0; }
int fgk_persistent_prepare(void) { return 0; }
int fgk_team_prepare(void) { return 0; }
int fgk_nucleus_prepare(uint32_t most_teams[FGK_NUCLEUS_TEAM_SIZES]) {
    for (uint32_t i = 0; i < FGK_NUCLEUS_TEAM_SIZES; i++) most_teams[i] = 296u >> i;
    return 0;
}
int fgk_static_scratch_address(int device, void **address) { (void)device; *address = NULL; return 1; }

int fgk_launch_stream_select(const fgk_stream_launch *l, void *stream) {
    (void)stream;
    return note("stream only_raising=%u uniforms=%d\n", l->only_raising, l->uniforms != NULL);
}
int fgk_launch_persistent_select(const fgk_stream_launch *l, uint32_t ctas, void *stream) {
    (void)stream;
    return note("ring skip_raising=%u general=%u ctas=%u uniforms=%d\n", l->skip_raising, l->general, ctas, l->uniforms != NULL);
}
int fgk_launch_team_select(const fgk_stream_launch *l, uint32_t team, uint32_t chunk, uint32_t form, uint32_t which, void *stream) {
    (void)stream;
    (void)form;
    return note("team which=%u team=%u covers=%d uniforms=%d\n", which, team, (uint64_t)team * chunk >= l->vocab, l->uniforms != NULL);
}
int fgk_launch_nucleus_select(const fgk_nucleus_launch *l, void *stream) { (void)l; (void)stream; return note("nucleus\n"); }
int fgk_launch_history_build(const fgk_stream_launch *l, void *stream) { (void)l; (void)stream; return note("history\n"); }
int fgk_launch_merge_select(const fgk_merge_launch *l, void *stream) { (void)l; (void)stream; return note("merge\n"); }
