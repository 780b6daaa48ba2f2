"""Host side of the kernel launches on a fake CUDA runtime of two devices (no GPU): the permission for more than 48 KB of dynamic
shared memory belongs to one device, so every device that a process launches from has to be given it."""
import ctypes as c
import glob
import os
import re
import shutil
import subprocess

import pytest

from neuronx_distributed_llama3_2_b200.ops import _lib

FAKE = r"""
#include <stddef.h>
#include <string.h>
typedef struct { unsigned x, y, z; } dim3_t;
typedef struct { dim3_t grid, block; size_t smem; void* stream; void* attrs; unsigned n; } config_t;
static int device, last, refused, launches;
static struct { const void* f; int bytes[2]; } allowed[512];
static int n_allowed;
static int* slot(const void* f) {
    for (int i = 0; i < n_allowed; ++i) if (allowed[i].f == f) return allowed[i].bytes;
    allowed[n_allowed].f = f;
    return allowed[n_allowed++].bytes;
}
static int launch(const void* f, size_t smem) {
    ++launches;
    if (smem > 48 * 1024 && smem > (size_t)slot(f)[device]) { ++refused; return last = 1; }
    return 0;
}
int fake_use(int d) { device = d; refused = launches = last = 0; return 0; }
int fake_refused(void) { return refused; }
int fake_launches(void) { return launches; }
int cudaGetDevice(int* d) { *d = device; return 0; }
int cudaFuncSetAttribute(const void* f, int attr, int v) { if (attr == 8) slot(f)[device] = v; return 0; }
int cudaDeviceGetAttribute(int* v, int attr, int d) { *v = attr == 16 ? 148 : 1; return 0; }
int cudaGetLastError(void) { int e = last; last = 0; return e; }
int cudaPeekAtLastError(void) { return last; }
const char* cudaGetErrorString(int e) { return "refused by the fake runtime"; }
int cudaLaunchKernel(const void* f, dim3_t g, dim3_t b, void** a, size_t smem, void* s) { return launch(f, smem); }
int cudaLaunchKernelExC(const config_t* cfg, const void* f, void** a) { return launch(f, cfg->smem); }
int cudaMemsetAsync(void* p, int v, size_t n, void* s) { return 0; }
int cudaFree(void* p) { return 0; }
int cudaGetSymbolAddress(void** p, const void* s) { *p = (void*)0x7000000; return 0; }
static int encode(void* map) { memset(map, 0, 128); return 0; }
int cudaGetDriverEntryPoint(const char* name, void** fn, unsigned long long flags, int* q) { *fn = (void*)encode; *q = 0; return 0; }
static struct { dim3_t g, b; size_t smem; void* s; } pushed;
unsigned __cudaPushCallConfiguration(dim3_t g, dim3_t b, size_t smem, void* s) {
    pushed.g = g; pushed.b = b; pushed.smem = smem; pushed.s = s;
    return 0;
}
int __cudaPopCallConfiguration(dim3_t* g, dim3_t* b, size_t* smem, void** s) {
    *g = pushed.g; *b = pushed.b; *smem = pushed.smem; *s = pushed.s;
    return 0;
}
static void* handle;
void** __cudaRegisterFatBinary(void* p) { return &handle; }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterFunction(void** h, const char* f, char* d, const char* n, int t, void* a, void* b, void* e, void* g, int* w) {}
void __cudaRegisterVar(void** h, char* v, char* d, const char* n, int e, size_t s, int k, int g) {}
"""
OBJECTS = ("rmsnorm", "gemm_tcgen05", "gemm_smallm", "flash_attn_tc", "flash_attn_bwd_tc", "decode_attention", "moe_forward",
           "moe_sparse", "attn_tc_host", "tma_host", "runtime")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    if shutil.which("g++") is None or not (shutil.which(_lib._nvcc()) or glob.glob(_lib._nvcc())):
        pytest.skip("needs nvcc and g++")
    objects = [os.path.join(_lib.BUILD_DIR, o + ".o") for o in OBJECTS]
    _lib.build(force=not all(map(os.path.exists, objects)))
    out = tmp_path_factory.mktemp("fake")
    (out / "fake.c").write_text(FAKE)
    subprocess.run(["gcc", "-w", "-O1", "-fPIC", "-c", str(out / "fake.c"), "-o", str(out / "fake.o")], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", str(out / "fake.so"), *objects, str(out / "fake.o")], check=True)
    return c.CDLL(str(out / "fake.so"))


P, L, F = (lambda n=1: c.c_void_p(n << 20)), c.c_longlong, c.c_float           # pointers are passed on, never followed


def _strides(n):
    return (L * (3 * n))(*([1 << 20, 128, 4096] * n))


CALLS = {
    "rmsnorm_bwd": lambda lib: lib.nxd_rmsnorm_bwd(P(1), P(2), P(3), P(4), None, P(5), P(6), None, 0, P(7), 64, 8192, None),
    "rmsnorm_bwd_static": lambda lib: lib.nxd_rmsnorm_bwd_static(P(1), P(2), P(3), P(4), None, P(5), P(6), None, 0, 64, 4096, None),
    "gemm": lambda lib: lib.nxd_gemm_bf16(0, P(1), P(2), P(3), 256, 256, 256, L(256), L(256), L(256), 0, 0, None),
    "gemm_swiglu": lambda lib: lib.nxd_gemm_swiglu_bf16(P(1), P(2), P(3), 256, 256, 256, L(256), L(256), L(256), None),
    "experts": lambda lib: lib.nxd_moe_sorted_forward(P(1), P(2), P(3), None, P(4), P(5), None, None, None, P(6), P(7), L(64), 2, 256,
                                                      256, 4, 0, 1, F(1), F(1), F(1), F(0), None),
    "smallm": lambda lib: lib.nxd_gemm_smallm_bf16(P(1), P(2), None, P(3), 4, 2048, 2048, L(2048), L(2048), L(2048), L(0), 0, None),
    "portion": lambda lib: lib.nxd_attn_prefill_cache_tc(P(1), P(2), P(3), L(1 << 20), L(1 << 17), L(128), L(1 << 20), L(1 << 17), L(128),
                                                         L(2), 1024, None, 0, 0, P(4), P(5), None, None, None, None, 2, 256, 4, 2, 128,
                                                         F(0.1), 0, 0, F(0), None, None, None, None, L(0), 0, F(1), L(0), None),
    "attention": lambda lib: lib.nxd_flash_attn_fwd_tc(P(1), P(2), P(3), P(4), None, _strides(4), 1, 4, 2, 256, 256, 128, F(0.1), 1, None),
    "attention_bwd": lambda lib: lib.nxd_flash_attn_bwd_tc(*(P(i) for i in range(1, 10)), None, P(10), P(11), P(12), _strides(8), 1, 4, 4,
                                                           256, 256, 128, F(0.1), 1, None),
    "token": lambda lib: lib.nxd_decode_attn(P(1), P(2), P(3), P(4), None, L(1 << 20), L(1 << 17), 0, 0, P(5), P(6), 2, 8, 2, 128, 4,
                                             F(0.1), None),
}


@pytest.mark.parametrize("name", CALLS)
def test_every_device_is_given_its_shared_memory(library, name):
    library.nxd_last_error.restype = c.c_char_p
    for device in (0, 1, 0):
        library.fake_use(device)
        rc = CALLS[name](library)
        assert rc == 0 and library.fake_refused() == 0, (device, rc, library.nxd_last_error())
        assert library.fake_launches() > 0


# one wave of two CTAs per SM for groups of query heads, more where the FMA kernel serves (148 SMs)
@pytest.mark.parametrize("B,n_q,n_kv,max_len,splits", [(12, 64, 16, 4000, 1), (12, 16, 16, 4000, 2), (5, 32, 32, 4000, 2), (1, 32, 8, 4000, 32),
                                                       (1, 8, 8, 100000, 37), (64, 8, 1, 200, 2), (1, 32, 1, 100000, 64)])
def test_splits_of_a_token_step(library, B, n_q, n_kv, max_len, splits):
    assert library.nxd_decode_attn_splits(B, n_q, n_kv, max_len) == splits


def test_kernels_trigger_behind_their_tensor_memory():
    """A programmatic dependent that allocates tensor memory and then waits for the grid before it must not find CTAs of that grid
    that have none yet: in the source of every kernel that allocates, the allocation comes before the trigger."""
    root = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
    seen = set()
    for path in glob.glob(os.path.join(root, "*.cu")):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for start in re.finditer(r"__global__", text):
            first = text.index("{", start.end())
            depth, end = 1, first + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            body = text[first:end]
            trigger, alloc = body.find("pdl_trigger()"), body.find("tmem_alloc")
            if trigger >= 0 and alloc >= 0:
                seen.add(os.path.basename(path))
                assert alloc < trigger, f"{os.path.basename(path)}: {text[start.start():first][:120]}"
    assert {"gemm_smallm.cu", "gemm_tcgen05.cu", "flash_attn_tc.cu"} <= seen
