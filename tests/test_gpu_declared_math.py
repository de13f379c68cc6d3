"""The device forms of the declared scalar functions (csrc/declared_math.cuh, csrc/common.cuh) on their own, compiled into a small
test library with the product's flags: against the CPU oracle over every float whose result is not a constant, and a sample of the rest."""
import concurrent.futures as cf
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "strix-halo-engine-lab_b200")

SOURCE = """
#include "declared_math.cuh"
using namespace b200moe;
__global__ void exp_kernel(const u32* x, u32 n, int gfx1151, float* out) {
    const u32 i = blockIdx.x * 256u + threadIdx.x;
    if (i < n) out[i] = gfx1151 ? gfx1151_expf(__uint_as_float(x[i])) : declared_exp(__uint_as_float(x[i]));
}
extern "C" int exp_bits(const u32* x, u32 n, int gfx1151, float* out) {
    exp_kernel<<<(n + 255) / 256, 256>>>(x, n, gfx1151, out);
    return cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import importlib.util
    spec = importlib.util.spec_from_file_location("b200moe_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    d = tmp_path_factory.mktemp("declared")
    (d / "math.cu").write_text(SOURCE)
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-I", os.path.join(PKG, "csrc"), "-shared", "-o", str(d / "math.so"), str(d / "math.cu")], check=True)
    torch.zeros(1, device="cuda")
    return C.CDLL(str(d / "math.so"))


def bits_of(x):
    return int(np.array([x], np.float32).view(np.uint32)[0])


@pytest.mark.parametrize("gfx1151", [1, 0])
def test_exp_for_every_float(device, oracle, gfx1151):
    """Both exponentials: every float of magnitude 2^-26 (below, 1 is the result) to 104.5 (above, 0 or infinity), of either sign, and the first
    patterns of every 2^12 of all others, infinities and NaNs included."""
    lo, hi, step = bits_of(2.0 ** -26), bits_of(104.5), 1 << 22
    chunks = [np.arange(a + sign, min(a + step, hi) + sign, dtype=np.uint32) for sign in (0, 1 << 31) for a in range(lo, hi, step)]
    rest = (np.arange(1 << 20, dtype=np.uint64) << np.uint64(12)).astype(np.uint32)
    chunks += [rest, rest + np.uint32(1)]

    def host(c):
        out = np.empty(c.size, np.float32)
        oracle.lib.orc_exp_bits(C.c_void_p(c.ctypes.data), C.c_uint32(c.size), gfx1151, C.c_void_p(out.ctypes.data))
        return out

    with cf.ThreadPoolExecutor(8) as pool:
        for c, want in zip(chunks, pool.map(host, chunks)):
            x = torch.from_numpy(c.view(np.int32)).cuda()
            got = torch.empty(c.size, dtype=torch.float32, device="cuda")
            assert device.exp_bits(C.c_void_p(x.data_ptr()), C.c_uint32(c.size), gfx1151, C.c_void_p(got.data_ptr())) == 0
            got = got.cpu().numpy()
            wrong = (got.view(np.uint32) != want.view(np.uint32)) & ~(np.isnan(got) & np.isnan(want))
            assert not wrong.any(), (hex(int(c[wrong][0])), float(got[wrong][0]), float(want[wrong][0]), int(wrong.sum()))
