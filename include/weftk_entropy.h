/*
 * weftk_entropy.h — chunked order-0 rANS decode of PRIM payloads on the GPU (C ABI of libweftk.so).
 *
 * Replaces the reference decoder's entropy stage for the primitive payload:
 * `decode_prim_payload` (src/weft/prim_chunks.py:80-125) over `decode_bytes` / the rANS
 * decoder (src/weft/entropy.py:121-189, mode byte and header layout :192-217), and its GPU
 * twin (src/weft/gpu_entropy.py:90-211, one thread per chunk).  Each chunk is either raw
 * (mode 0: <u8 0, u32 n, n bytes>) or rANS (mode 1: <u8 1, u32 n, u16 n_sym, n_sym x <u8 sym,
 * u16 freq>, u32 state, u32 emitted, emitted bytes>, 12-bit probabilities, state lower bound
 * 2^23, bytes consumed from the end of the emitted run).  One warp decodes one chunk: the lanes
 * build the 4096-slot symbol table together, then one lane runs the (sequential) state chain.
 * Every read stays inside its chunk's coded bytes and every write inside its raw range; a chunk
 * that does not parse is reported through weftk_device_status (WEFTK_E_ARG) and left unwritten.
 */
#ifndef WEFTK_ENTROPY_H
#define WEFTK_ENTROPY_H

#include "weftk.h"

#ifdef __cplusplus
extern "C" {
#endif

/* One coded chunk: bytes [coded_offset, coded_offset + coded_length) of the payload decode
 * to bytes [raw_offset, raw_offset + raw_length) of the output (a CIDX entry,
 * src/weft/prim_chunks.py:23-77). */
typedef struct WeftRansChunk {
    int64_t coded_offset;
    int64_t coded_length;
    int64_t raw_offset;
    int64_t raw_length;
} WeftRansChunk;

/* Decode n_chunks chunks of d_payload (payload_len bytes) into d_out (out_len bytes). */
int weftk_rans_decode_chunks(const uint8_t* d_payload, int64_t payload_len, const WeftRansChunk* d_chunks,
                             int n_chunks, uint8_t* d_out, int64_t out_len, void* stream);

/* A primitive-stack file in host memory: its bytes and where its parts stand in them (byte offsets of
 * what follows each block's own header).  Geometry, colours and residuals are dequantized as
 * src/weft/primitives.py:102-177 and src/weft/render.py:231-232 do, target rects as :321-334. */
typedef struct WeftSceneFile {
    const uint8_t* blob;
    int64_t blob_len;
    int64_t prim, prim_len; /* the PRIM payload */
    int64_t cidx;           /* n_chunks entries of 24 bytes */
    int64_t toc;            /* n_tiles + 1 u32 offsets */
    int64_t qtree;          /* n_tiles entries of 5 bytes: x u16, y u16, side u8 */
    int64_t res0;           /* n_tiles x 3 int8, or -1 */
    int64_t res1;           /* n_res1 x 48 int8 */
    int32_t n_chunks, n_tiles, n_res1;
    int32_t enc_w, enc_h;   /* the size the tiles cover */
    int32_t out_w, out_h;   /* the size to render */
    int32_t _pad;
} WeftSceneFile;

/*
 * The whole decoder walk of a file: chunks entropy-decoded, tiles parsed and rendered on the device, one
 * upload of the file.  out: out_h x out_w x 3 float32, host memory (on_device 0) or the current device's
 * (on_device 1, ordered on `stream`); the call returns with it written.  Pixels no tile covers are 0.
 * *irregular != 0: the file is not of the ordinary form (chunks that do not cover the tiles' bytes in
 * order, a payload, primitive or tile that does not parse exactly, a rect beyond the walk's limits);
 * the output is then undefined and a general decoder has to judge the file.
 */
int weftk_decode_scene(const WeftSceneFile* file, float* out, int on_device, int* irregular, void* stream);

#ifdef __cplusplus
}
#endif

#endif /* WEFTK_ENTROPY_H */
