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
// over_127 against the division for every float from 2^-119 on
__global__ void over_127_kernel(u32* wrong) {
    for (u32 i = 0x04000000u + blockIdx.x * 256u + threadIdx.x; i < 0x7f800000u; i += gridDim.x * 256u)
        if (__float_as_uint(over_127(__uint_as_float(i))) != __float_as_uint(__fdiv_rn(__uint_as_float(i), 127.0f))) atomicAdd(wrong, 1u);
}
extern "C" int over_127_wrong(u32* wrong) {
    over_127_kernel<<<1480, 256>>>(wrong);
    return cudaGetLastError();
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


def test_over_127_is_the_quotient(device):
    assert bits_of(2.0 ** -119) == 0x04000000
    wrong = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert device.over_127_wrong(C.c_void_p(wrong.data_ptr())) == 0
    assert wrong.item() == 0


@pytest.mark.parametrize("rows", [1, 300])
def test_a8_groups_with_nan(oracle, rows):
    """Both forms of the quantiser on groups with 0, 1, 31 and 32 NaNs of either sign: a NaN does not count for the maximum and its code is -127;
    a group of NaNs alone keeps a NaN as its delta."""
    from b200moe import ops
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, 32 * 32), dtype=np.float32)
    groups = x.reshape(-1, 32)
    for i, g in enumerate(groups):
        n = (0, 1, 31, 32)[i % 4]
        g[rng.permutation(32)[:n]] = np.array([0x7fc00000, 0xffc00001], np.uint32).view(np.float32)[i // 4 % 2]
    codes, deltas, sums = oracle.quantize_a8(x)
    got = [t.cpu().numpy() for t in ops.enqueue_quantize_a8(torch.from_numpy(x).cuda())]
    alone = np.isnan(groups).all(axis=1).reshape(rows, -1)
    assert np.array_equal(got[0], codes) and np.array_equal(got[2], sums)
    assert np.isnan(got[1][alone]).all() and np.array_equal(got[1][~alone].view(np.uint32), deltas[~alone].view(np.uint32))
