"""Which kernel a call launches, and with how many CTAs: the library's objects linked against a runtime that records
launches instead of running them (fake_cuda_runtime.cpp).  Needs nvcc, no GPU."""
import ctypes as C
import glob
import os
import re
import shutil
import subprocess

import pytest

from speedoza_b200 import abi
from speedoza_b200.build import OBJDIR, build_library

HERE = os.path.dirname(os.path.abspath(__file__))
BASE = 1 << 32                     # operand addresses that nothing reads


class Launch(C.Structure):
    _fields_ = [("kernel", C.c_void_p), ("grid", C.c_uint), ("block", C.c_uint), ("cluster", C.c_uint), ("smem", C.c_uint)]


class Device:
    """The library over a fresh fake runtime: nothing that an earlier test made it remember."""

    def __init__(self, path):
        self.lib = C.CDLL(path)
        self.lib.fake_launch.restype = C.POINTER(Launch)
        symbols = subprocess.run(["nm", "-C", path], capture_output=True, text=True, check=True).stdout
        self.names = {int(a, 16): n for a, n in re.findall(r"^([0-9a-f]+) [tT] (.*)$", symbols, flags=re.M)}
        at = next(a for a, n in self.names.items() if n == "fake_launch_count")
        self.base = C.cast(self.lib.fake_launch_count, C.c_void_p).value - at

    def launches(self, call):
        """(kernel, grid, cluster) of every launch that call() makes, and its status."""
        self.lib.fake_reset()
        code = call()
        found = []
        for i in range(self.lib.fake_launch_count()):
            l = self.lib.fake_launch(i).contents
            name = re.search(r"(\w+_kernel(?:<[^>]*>)?)", self.names[l.kernel - self.base]).group(1)
            found.append((re.sub(r"\b(\d+)u\b", r"\1", name), l.grid, l.cluster))
        return found, code

    def product(self, m, n, k, entry="qwen36_nvfp4_gemm"):
        p = [abi.DevicePtr(BASE + (i << 34)) for i in range(5)]
        spec = abi.Nvfp4GemmSpec(m, n, k, p[0], p[1], abi.DevicePtr(0), p[2], p[3], abi.DevicePtr(0), p[4], abi.DevicePtr(0), 0, 1.0)
        return self.launches(lambda: getattr(self.lib, entry)(C.byref(spec)))


@pytest.fixture(scope="module")
def linked(tmp_path_factory):
    build_library()
    source = os.path.join(HERE, "fake_cuda_runtime.cpp")
    folder = str(tmp_path_factory.mktemp("fake_cuda"))
    wrapped = re.findall(r"__wrap_(\w+)\(", open(source).read())
    subprocess.run(["nvcc", "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-c", source, "-o", folder + "/fake.o"], check=True)
    subprocess.run(["nvcc", "-shared", "-o", folder + "/fake.so", folder + "/fake.o", *sorted(glob.glob(OBJDIR + "/*.cu.o")), "-ldl",
                    *[f for w in wrapped for f in ("-Xlinker", "--wrap=" + w)]], check=True)
    return folder + "/fake.so"


@pytest.fixture
def device(linked, tmp_path):
    return Device(shutil.copy(linked, tmp_path))  # a copy is a library of its own to the loader


GEMV, TILES, CLUSTERS = "nvfp4_gemv_mma_kernel<1, false>", "nvfp4_gemm_tc_kernel<8, true>", "nvfp4_gemm_splitk_kernel<8, true>"


@pytest.mark.parametrize("entry", ["qwen36_nvfp4_gemm", "qwen36_decode_nvfp4_gemv"])
@pytest.mark.parametrize("m,k,kernel", [
    # the last round of tiles too empty, or K too short, for the block-scaled tiles to win
    (24576, 4096, GEMV), (24576, 5120, GEMV), (40960, 4096, GEMV), (57344, 4096, GEMV), (58880, 5120, GEMV), (22016, 3072, GEMV),
    (22016, 5120, GEMV), (11008, 5120, GEMV), (12288, 2048, GEMV),
    # clusters cost more than they give
    (3072, 2048, GEMV), (9216, 2048, GEMV), (4608, 4096, GEMV), (3072, 5120, GEMV), (1536, 8192, GEMV), (1024, 5120, GEMV),
    (34816, 5120, TILES), (28672, 4096, TILES), (12288, 5120, TILES), (14336, 2048, TILES), (18944, 4096, TILES), (44800, 5120, TILES),
    (248320, 5120, TILES), (11904, 3072, TILES), (12288, 2304, TILES), (24576, 2304, TILES), (24576, 4352, TILES), (24576, 4608, TILES),
    (5120, 17408, CLUSTERS), (2048, 6144, CLUSTERS), (2048, 12288, CLUSTERS), (4608, 6144, CLUSTERS), (4608, 17408, CLUSTERS),
    (5120, 6144, CLUSTERS), (4864, 3584, CLUSTERS), (3072, 6656, CLUSTERS), (1536, 12288, CLUSTERS)])
def test_one_token_runs_on_the_kernel_that_measured_faster(device, m, k, kernel, entry):
    launches, code = device.product(m, 1, k, entry)
    assert code == abi.SUCCESS and [name for name, _, _ in launches] == [kernel]


def test_one_token_operands_off_sixteen_bytes_run_on_the_gemv(device):
    """Eight-byte aligned activation codes: what the GEMV takes and the tiles do not."""
    p = [abi.DevicePtr(BASE + (i << 34)) for i in range(5)]
    spec = abi.Nvfp4GemmSpec(34816, 1, 5120, p[0], p[1], abi.DevicePtr(0), abi.DevicePtr(p[2].ptr + 8), p[3], abi.DevicePtr(0), p[4],
                             abi.DevicePtr(0), 0, 1.0)
    launches, code = device.launches(lambda: device.lib.qwen36_nvfp4_gemm(C.byref(spec)))
    assert code == abi.SUCCESS and [name for name, _, _ in launches] == [GEMV]


@pytest.mark.parametrize("entry", ["qwen36_nvfp4_gemm", "qwen36_decode_nvfp4_gemv"])
@pytest.mark.parametrize("m,k", [(34816, 5120), (5120, 17408)])
def test_one_token_runs_on_the_gemv_where_the_tiles_decline(device, m, k, entry):
    """The two-dimensional tensor maps of the tiles are refused; those of the GEMV have five and three dimensions."""
    device.lib.fake_refuse_2d_maps(1)
    launches, code = device.product(m, 1, k, entry)
    assert code == abi.SUCCESS and [name for name, _, _ in launches] == [GEMV]


def split_choice(device, m_blocks, k_blocks, at_most):
    """CTAs per row block: the longest CTA's K-blocks over all rounds are fewest, the smaller of equals; 1 = no clusters."""
    best, least = 1, k_blocks * -(-m_blocks // 148)
    for split in range(2, min(148 // m_blocks, at_most, k_blocks // 2) + 1):
        longest = -(-m_blocks // device.lib.fake_clusters(split)) * -(-k_blocks // split)
        if longest < least:
            best, least = split, longest
    return best


def test_split_k_clusters_are_as_large_as_fit_one_per_row_block(device):
    """Every row-block count that can be split, over K-block counts that meet in the same slots of the table of known choices
    ((31 row blocks + 7 K-blocks) mod 64); asked twice, the second time in another order."""
    shapes = [(mb, kb) for mb in range(1, 76) for kb in (4, 16, 24, 68, 80, 88)]
    tables = (2, "nvfp4_gemm_{}_kernel<8, false>", 8), (9, "nvfp4_gemm_{}_kernel<16, false>", 8), (17, "nvfp4_gemm_{}_kernel<32, false>", 5)
    for tokens, kernel, at_most in tables:
        for mb, kb in shapes + shapes[::-7] + shapes[::-3]:
            split = split_choice(device, mb, kb, at_most)
            want = (kernel.format("splitk"), mb * split, split) if split > 1 else (kernel.format("tc"), mb, 1)
            assert device.product(128 * mb, tokens, 256 * kb) == ([want], abi.SUCCESS), (mb, kb)
    # 16 row blocks, where clusters of eight have room for 15 only, and 36, where those of four have room for 34
    assert [split_choice(device, mb, 24, 8) for mb in (15, 16, 28, 36)] == [8, 6, 4, 3]


def test_a_failed_occupancy_query_is_asked_again(device):
    """No answer from the device costs the call its clusters, not the process."""
    want = Device(shutil.copy(device.lib._name, device.lib._name + ".fresh")).product(2048, 5, 6144)
    assert want[0][0][0] == "nvfp4_gemm_splitk_kernel<8, false>"
    device.lib.fake_fail_occupancy(7)                                   # two to eight CTAs a cluster
    assert device.product(2048, 5, 6144) == ([("nvfp4_gemm_tc_kernel<8, false>", 16, 1)], abi.SUCCESS)
    assert device.product(2048, 5, 6144) == want
    device.lib.fake_fail_occupancy(1)
    assert device.product(8192, 600, 5120)[0][0][0] != "nvfp4_gemm_pair6_kernel<false>"
    assert device.product(8192, 600, 5120)[0][0][0] == "nvfp4_gemm_pair6_kernel<false>"


def test_a_failed_occupancy_query_of_decode_attention_is_asked_again(device):
    p = [abi.DevicePtr(BASE + (i << 34)) for i in range(9)]
    spec = abi.AttentionDecodeSpec(0, 599, *p[:5], abi.DevicePtr(0), p[5], abi.AttentionShape(24, 4, 256, 0), 1, abi.DevicePtr(0), *p[6:], 256, 0)

    def kernels():
        launches, code = device.launches(lambda: device.lib.qwen36_attention_decode(C.byref(spec)))
        assert code == abi.SUCCESS
        return [re.sub("<.*", "", name) for name, _, _ in launches]

    device.lib.fake_fail_occupancy(2)                                   # sixteen CTAs, eight
    assert "decode_one_launch_kernel" not in kernels()
    assert kernels() == ["decode_one_launch_kernel"]


@pytest.mark.parametrize("offset", [0, 4])
def test_argmax_keys_off_their_alignment_are_cleared_as_bytes(device, offset):
    p = [abi.DevicePtr(BASE + (i << 34)) for i in range(6)]
    spec = abi.Bf16MatvecArgmaxRowsSpec(3, 4096, 1024, p[0], p[1], p[2], abi.DevicePtr(0), abi.DevicePtr(p[3].ptr + offset), 64, p[4])
    launches, code = device.launches(lambda: device.lib.qwen36_bf16_matvec_argmax_rows(C.byref(spec)))
    assert code == abi.SUCCESS
    assert ("bf16_argmax_clear_kernel" in [name for name, _, _ in launches], device.lib.fake_memsets()) == ((True, 0) if offset == 0 else (False, 1))
