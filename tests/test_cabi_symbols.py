"""The C-ABI library loads without a GPU and exports every symbol include/crownest_ops.h declares."""
import ctypes
import os
import re

from conftest import ROOT
from crownest_b200 import _lib


def header_symbols():
    text = open(os.path.join(ROOT, "include", "crownest_ops.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(cn_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    L = ctypes.CDLL(_lib.SO_PATH)
    names = header_symbols()
    assert len(names) >= 7
    for n in names:
        assert hasattr(L, n), f"{n} is declared in the header but not exported"
    # and the Python binding knows each of them
    assert set(names) <= set(_lib.exported_symbols()), set(names) - set(_lib.exported_symbols())


def test_error_string_and_version_need_no_gpu():
    L = _lib.lib()
    assert b"sm_100a" in L.cn_version()
    # a refused shape is reported before any CUDA call
    assert L.cn_nvfp4_gemv(None, None, None, None, 4, 100, 1, 4, 1, None) == 1
    assert b"multiple of 256" in L.cn_last_error_string()


def test_shared_memory_attribute_is_booked_per_kernel_and_device():
    """The large dynamic shared-memory attribute belongs to a (kernel, device) pair: a process that launches on a second
    GPU must set it there again, and a larger request on the same GPU too. cn_smem_book is the book every launch consults."""
    L = _lib.lib()
    k1, k2 = ctypes.c_void_p(0x1000), ctypes.c_void_p(0x2000)
    assert L.cn_smem_book(k1, 0, 100 * 1024, 0) == 1  # asked without committing: still to do
    assert L.cn_smem_book(k1, 0, 100 * 1024, 1) == 1
    assert L.cn_smem_book(k1, 0, 100 * 1024, 1) == 0  # covered now
    assert L.cn_smem_book(k1, 0, 64 * 1024, 1) == 0   # a smaller size is covered by the larger
    assert L.cn_smem_book(k1, 0, 200 * 1024, 1) == 1  # a larger one is not
    assert L.cn_smem_book(k1, 1, 100 * 1024, 1) == 1  # another device: its own call
    assert L.cn_smem_book(k2, 0, 100 * 1024, 1) == 1  # another kernel: its own call
    assert L.cn_smem_book(k1, 1, 100 * 1024, 1) == 0


def test_where_activations_are_held_in_fixed_point():
    """A rule of the matrix and the type alone: both sides of each of its lines (rows, k, gate / up)."""
    from crownest_b200 import CN_BF16, CN_F32
    bits = _lib.lib().cn_nvfp4_gemv_fixed_bits
    # bf16: 40 tiles of 128 rows up to three chunks of 256 values (74 with gate / up), 64 up to six, 74 beyond; long rows from a size on; few long rows never
    for yes, no in [((4993, 256, 0), (4992, 256, 0)), ((4993, 512, 0), (4992, 512, 0)), ((4993, 768, 0), (4992, 768, 0)), ((4673, 256, 1), (4672, 256, 1)), ((4673, 768, 1), (4672, 768, 1)),
                    ((8065, 1024, 0), (8064, 1024, 0)), ((8065, 1536, 0), (8064, 1536, 0)), ((9345, 1792, 0), (9344, 1792, 0)), ((4033, 1024, 1), (4032, 1024, 1)), ((1954, 4096, 0), (1953, 4096, 0)),
                    ((1368, 5120, 0), (1367, 5120, 0)), ((501, 8192, 0), (500, 8192, 0)), ((1281, 17408, 0), (1280, 17408, 0))]:
        assert bits(*yes, CN_BF16) == 22 and bits(*no, CN_BF16) == 0, (yes, no)
    for yes, no in [((1, 2048, 0), (1, 1024, 0)), ((1, 1280, 1), (1, 1024, 1)), ((64, 768, 0), (63, 768, 0)), ((64, 1792, 0), (64, 768, 1)), ((8192, 512, 0), (8191, 512, 0)), ((5860, 512, 1), (5859, 512, 1))]:
        assert bits(*yes, CN_F32) == 31 and bits(*no, CN_F32) == 0, (yes, no)
    assert bits(0, 4096, 0, CN_F32) == bits(4096, 100, 0, CN_F32) == bits(4096, 4096, 0, 2) == 0


def test_the_cut_of_a_row_needs_no_device():
    """Into how many parts a row is cut fixes the order of its sum: a rule of the matrix alone, the same on every GPU and on none."""
    cut = _lib.lib().cn_nvfp4_gemv_cut
    for rows in (1, 128, 2048, 4096, 5120, 9728, 17408, 40960, 248320):
        for k in (256, 512, 1024, 4096, 5376, 17408):
            for gu in (0, 1):
                c = cut(rows, k, gu)
                assert c in (1, 2, 4, 6, 8) and c <= k // 256, (rows, k, gu, c)
    # a few that were timed
    assert [cut(*m) for m in ((4096, 4096, 0), (5120, 5120, 0), (7168, 5120, 0), (5120, 17408, 0), (17408, 5120, 1), (16384, 2048, 0))] == [4, 4, 4, 6, 1, 1]
    # 152 to 192 and 313 tiles, which leave most SMs one CTA or a short second round without a cluster
    assert [cut(*m) for m in ((9728, 5120, 1), (12288, 4096, 1), (20000, 2048, 1), (20224, 4096, 0))] == [4, 4, 2, 4]
    assert cut(0, 4096, 0) == 0 and cut(4096, 128, 0) == 0
