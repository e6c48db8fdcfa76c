"""What the C entry points decide on the host, in front of any launch.  No GPU is needed."""

import ctypes
import subprocess
import sys

import pytest

from cornstarch_b200.csrc.build import LIB_PATH


@pytest.mark.parametrize("call,code", [
    ("csb_glu_fwd(None, None, C.c_long(5), 0, 0, None)", 0),
    ("csb_glu_bwd(None, None, None, C.c_long(5), 0, 0, None)", 0),
    ("csb_glu_fwd(None, None, C.c_long(0), 8, 0, None)", 0),
    ("csb_colsum(None, None, None, 0, 0, 5, 0, None)", -1),
])
def test_no_columns(call, code):
    """Sizes with nothing to launch, in a process of their own: an error code or success, no division by an extent of zero."""
    if not LIB_PATH.exists():
        pytest.skip("the native library is not built")
    src = f"import ctypes as C; print(C.CDLL({str(LIB_PATH)!r}).{call})"
    res = subprocess.run([sys.executable, "-c", src], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0 and int(res.stdout) == code, (res.returncode, res.stdout, res.stderr)


FULL, CAUSAL, BITFIELD = 0, 1, 2


def _splits():
    if not LIB_PATH.exists():
        pytest.skip("the native library is not built")
    return ctypes.CDLL(str(LIB_PATH)).csb_attn_bwd_splits


@pytest.mark.parametrize("mode", [FULL, CAUSAL, BITFIELD])
@pytest.mark.parametrize("Hq,Hk", [(32, 8), (32, 32), (16, 4), (8, 1), (64, 1), (20, 20)])
def test_scratch_of_the_split_attention_backward_is_bounded(mode, Hq, Hk):
    """fp32 parts of dK and dV: 2 * n * B * Sk * Hk * 128 floats, 128 MiB at most, and none for sequences that fill the GPU
    many times over anyway."""
    splits = _splits()
    for B in (1, 2, 3, 4, 16):
        for S in (1, 64, 77, 128, 333, 729, 1024, 2048, 3571, 4096, 8192, 12288, 16384, 32768, 65536):
            n = splits(mode, B, S, S, Hq, Hk)
            assert 1 <= n <= 16
            assert n == 1 or 2 * n * B * S * Hk * 128 * 4 <= 128 << 20, (B, S, n)
            if B * Hk * S >= 65536 * 8:
                assert n == 1, (B, S, n)


def test_split_counts():
    splits = _splits()
    # small grids are split, and one block per key block is kept where the predicted gain is within the prediction's error
    assert all(splits(CAUSAL, 1, S, S, 32, 8) > 1 for S in (128, 333, 1024, 2048, 3072))
    assert splits(CAUSAL, 1, 1500, 1500, 8, 1) > 8 and splits(FULL, 1, 8192, 8192, 32, 8) == 2
    assert splits(CAUSAL, 1, 4096, 4096, 32, 8) == splits(FULL, 1, 4096, 4096, 32, 8) == 1
    assert splits(FULL, 1, 65536, 65536, 32, 8) == splits(FULL, 4, 729, 729, 16, 16) == 1


# weights that are not adjacent: one launch where a tile suits them all, separate calls where the widths leave only a narrow one
@pytest.mark.parametrize("T,K,widths,one", [
    (1531, 4096, (4096, 1024, 1024), True), (729, 1152, (1152, 1152, 1152), True), (77, 1152, (1152, 1152, 1152), True),
    (4575, 5120, (5120, 640, 640), False), (7300, 5120, (5120, 640, 640), False), (8192, 4096, (4096, 128, 128), False),
    (251, 4096, (11008, 11008), False), (8192, 1024, (4096, 128), False), (64, 264, (136, 256), False), (64, 264, (128,) * 5, False),
])
def test_separate_weights_are_joined_where_that_is_faster(T, K, widths, one):
    if not LIB_PATH.exists():
        pytest.skip("the native library is not built")
    bn, cg = ctypes.c_int(-1), ctypes.c_int(-1)
    rc = ctypes.CDLL(str(LIB_PATH)).csb_gemm_cols_choice((ctypes.c_int * len(widths))(*widths), len(widths), T, K, ctypes.byref(bn), ctypes.byref(cg))
    assert rc == 0 and (bn.value > 0) == one
    assert not one or all(w % bn.value == 0 for w in widths)
