/* Entry points between the library's own files (not part of the C ABI). */
#ifndef PHP_INTERNAL_H
#define PHP_INTERNAL_H

#include "php_fdtd.h"

extern "C" {
/* php_create with or without the second E and H buffers that a large
 * domain's interior launch uses (interior_sweep_tma); the results are the
 * same, bit for bit. */
__attribute__((visibility("hidden"))) int php_create_buffers(const php_desc* desc, bool split, php_ctx** out);
/* Device bytes without those buffers, and what they may add. */
__attribute__((visibility("hidden"))) int php_estimate_buffers(const php_desc* desc, uint64_t* bytes, uint64_t* more);
/* Whether the context holds them. */
__attribute__((visibility("hidden"))) bool php_holds_second_level(const php_ctx* ctx);
}

#endif
