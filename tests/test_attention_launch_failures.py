"""What the host side of the attention forward leaves behind when one of its steps fails (no GPU: the compiled launcher is linked with stand-ins for the
CUDA runtime and for the table of operand parts).  The launcher hands the kernel the parts of O to write and says so in the table; when a tensor map,
the item counter or the launch fails, the caller forms O by other kernels, which write only the FP32 array, so the table must not say so then."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "sb_internal.h"
static int encodes, fail_encode, fail_counter, fail_launch, launches, parts_valid, hint_valid, find_ok;
static char room[4096];
static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                       CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return ++encodes == fail_encode ? CUDA_ERROR_INVALID_VALUE : CUDA_SUCCESS;
}
extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { memset(a, 0, sizeof *a); a->numRegs = 128; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) { *fn = (void*)encode; if (q) *q = cudaDriverEntryPointSuccess; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { launches++; return fail_launch ? cudaErrorInvalidValue : cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { abort(); }
cudaError_t cudaGetLastError(void) { return fail_launch && launches ? cudaErrorInvalidValue : cudaSuccess; }
unsigned* sb_amax_take(sb_ctx_t*, const float*, size_t) { hint_valid = 1; return (unsigned*)room; }
void sb_amax_forget(sb_ctx_t*, const float*) { hint_valid = 0; }
int sb_parts_find(sb_ctx_t*, const float*, size_t, void** h, float** w, int* fresh) { if (!find_ok) return 0; *h = room; *w = (float*)room; *fresh = SB_PARTS_MAKE; parts_valid = 1; return 1; }
void sb_parts_set_amax(sb_ctx_t*, const float*, float*) {}
void sb_parts_invalidate(sb_ctx_t*, const float*) { parts_valid = 0; }
void sb_resolve_host_seq(sb_ctx_t*) {}
}
unsigned* sb_item_counter(sb_ctx_t*) { return fail_counter ? NULL : (unsigned*)room; }
static int run(int hd) {
    static int starts[2] = {0, 200};
    sb_ctx_t* c = (sb_ctx_t*)calloc(1, sizeof *c);
    c->pub.gpu_sm_count = 148; c->h_seq = starts; c->h_seq_n = 1; c->attn_seq_starts = (const uint32_t*)room;
    encodes = launches = parts_valid = hint_valid = 0;
    float* p = (float*)(((uintptr_t)room + 15) & ~(uintptr_t)15);
    const int rc = sb_attention_fused_forward(c, p, p + 4, p + 8, p + 12, p + 16, p + 20, p, p, p, p + 24, p, 200, 2, 1, hd);
    free(c->map_cache); free(c);
    return rc;
}
int main(void) {
    int bad = 0, failed = 0;
    for (int hd = 64; hd <= 128; hd += 64)
        for (find_ok = 0; find_ok < 2; find_ok++) {
            fail_encode = fail_counter = fail_launch = 0;
            int rc = run(hd);
            if (rc != 0 || launches != 1 || !hint_valid || parts_valid != find_ok) { printf("hd %d: plain call: rc %d launches %d hint %d parts %d\n", hd, rc, launches, hint_valid, parts_valid); bad++; }
            const int maps = encodes;
            for (int what = 1; what <= maps + 2; what++) {
                fail_encode = what <= maps ? what : 0; fail_counter = what == maps + 1; fail_launch = what == maps + 2;
                rc = run(hd);
                failed += rc != 0;
                if (rc == 0 || hint_valid || parts_valid || (launches && !fail_launch)) {
                    printf("hd %d, parts %d, failing step %d of %d: rc %d, O's maximum %s, its parts %s, launches %d\n", hd, find_ok, what, maps + 2, rc, hint_valid ? "announced" : "not announced",
                           parts_valid ? "marked as made" : "not marked", launches);
                    bad++;
                }
            }
        }
    printf("%d failures injected, %d left something behind\n", failed, bad);
    return bad != 0;
}
"""


def test_a_failed_forward_marks_nothing_as_made(tmp_path):
    from seraph_b200 import build
    build.build()
    obj = os.path.join(ROOT, "seraph_b200", "build", "attention_fused.cu.o")
    if not os.path.exists(obj):
        obj = str(tmp_path / "attention_fused.o")
        subprocess.run([build.NVCC, "-O1", "-std=c++17", *build.ARCH, "-c", os.path.join(build.CSRC, "attention_fused.cu"), "-o", obj], check=True)
    src, exe = str(tmp_path / "driver.cpp"), str(tmp_path / "driver")
    with open(src, "w") as f:
        f.write(DRIVER)
    subprocess.run(["g++", "-O1", "-w", "-I" + build.CUDA_INC, "-I" + build.CSRC, src, obj, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    assert " failures injected" in r.stdout and not r.stdout.startswith("0 failures")
