/* The C host layer over a backend whose every call fails, to see what it makes of that.  Test code only. */
#include <string.h>

#include "../../openfish_b200/csrc/backend.h"
#include "openfish_b200.h"

#define FAILS { return OPENFISH_B200_ERR_CUDA; }
int ofb_gpubuf_create(int T, int N, int state_len, openfish_gpubuf_t **out) FAILS
int ofb_gpubuf_destroy(openfish_gpubuf_t *gpubuf) FAILS
int ofb_gpubuf_check_owner(const openfish_gpubuf_t *gpubuf) { return OPENFISH_B200_OK; }
int ofb_gpubuf_check(const openfish_gpubuf_t *gpubuf, int T, int N, int state_len) { return OPENFISH_B200_OK; }
int ofb_decode_submit(int T, int N, int C, const void *scores, int state_len, const ofb_decode_params_t *params,
                      const openfish_gpubuf_t *gpubuf, uint8_t *moves, char *sequence, char *qstring) FAILS
int ofb_decode_submit_5wide(int T, int N, const void *scores5, int state_len, float clamp, const ofb_decode_params_t *params,
                            const openfish_gpubuf_t *gpubuf, uint8_t *moves, char *sequence, char *qstring) FAILS
int ofb_decode_wait(const openfish_gpubuf_t *gpubuf) FAILS
int ofb_last_decode_ms(const openfish_gpubuf_t *gpubuf, float ms[8]) {
    for (int i = 0; i < 8; ++i) ms[i] = 3.0f; /* (what had been read before the call that failed) */
    return OPENFISH_B200_ERR_CUDA;
}
int ofb_stream_wait_decode(void *stream, const openfish_gpubuf_t *gpubuf) FAILS
int ofb_selfcheck_wait(const openfish_gpubuf_t *gpubuf, unsigned limit_us) FAILS
int ofb_rotary(void *x, const void *sin_t, const void *cos_t, int batch, int seqlen, int nheads, int rotary_half,
               long long stride_batch, long long stride_seq, long long stride_head) FAILS
int ofb_selfcheck_arith(double err[2]) FAILS
float ofb_last_rotary_ms(void) { return 0.f; }
int ofb_set_device(int device) FAILS
int ofb_device_upload(const void *host, size_t bytes, void **out) FAILS
int ofb_device_free(void *device) FAILS
int ofb_device_download(void *host, const void *device, size_t bytes) FAILS
const char *ofb_error_text(void) { return "the backend says no"; }
