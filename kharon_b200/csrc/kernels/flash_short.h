// Attention of short sequences (flash_short.cu): up to KH_FLASH_SHORT_T positions, called by the entry points of flash_tcgen05.cu where it is faster.
#pragma once
#define KH_FLASH_SHORT_T 64
int kh_flash_short_fwd(const void* qkv, void* out, void* lse, int B, int T, int H, int hd, int ld, float scale, void* stream);
int kh_flash_short_bwd(const void* qkv, const void* out, const void* dout, const void* lse, void* dqkv, void* delta, int B, int T,
                       int H, int hd, int ld, float scale, void* stream);
