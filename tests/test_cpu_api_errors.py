"""Error behaviour of the drop-in surface on a host without a GPU.

The reference raises ValueError for a bad image count
(pysift/core.py:3998-4004) and a bad DSP scale count
(pysift/core.py:1203-1204); this package also raises NotImplementedError for
the learned orientation / descriptor / matcher options it does not carry,
ValueError for unknown blend and RANSAC options, and, with no CUDA device,
RuntimeError instead of falling back to a CPU path.
"""
import numpy as np
import pytest
import torch


def test_pysift_argument_errors():
    from pysift_b200 import PySIFT
    with pytest.raises(ValueError, match="dsp_n_scales"):
        PySIFT(dsp_n_scales=2)
    with pytest.raises(NotImplementedError, match="orientation"):
        PySIFT(orientation='orinet')
    with pytest.raises(NotImplementedError, match="descriptor"):
        PySIFT(descriptor='hardnet')


@pytest.mark.skipif(torch.cuda.is_available(), reason="checks the behaviour without a CUDA device")
def test_pysift_without_a_device_fails_loudly():
    from pysift_b200 import PySIFT
    with pytest.raises(RuntimeError, match="CUDA"):
        PySIFT()


@pytest.mark.parametrize("kw,exc", [
    (dict(matcher='lightglue'), NotImplementedError),
    (dict(orientation='orinet'), NotImplementedError),
    (dict(descriptor='hardnet'), NotImplementedError),
    (dict(pca_dims=32), NotImplementedError),
    (dict(blend='average'), ValueError),
    (dict(n_blend_levels=9), ValueError),
    (dict(n_blend_levels=0), ValueError),
    (dict(ransac_method='lmeds'), ValueError),
])
def test_stitcher_argument_errors(kw, exc):
    from pysift_b200 import GPUPyStitch
    with pytest.raises(exc):
        GPUPyStitch(**kw)


@pytest.mark.parametrize("n", [0, 1, 4])
def test_stitch_image_count(n):
    from pysift_b200 import GPUPyStitch
    st = GPUPyStitch.__new__(GPUPyStitch)  # the count is checked before any device state is used
    imgs = [np.zeros((8, 8, 3), np.uint8)] * n
    with pytest.raises(ValueError, match="2 or 3 images"):
        st.stitch(*imgs)
    with pytest.raises(ValueError, match="2 or 3 images"):
        st.stitch(imgs)


def test_detect_config_ranges():
    from pysift_b200 import _lib
    from pysift_b200.core import build_detect_config
    with pytest.raises(ValueError, match="n_scales"):
        build_detect_config(5, _lib.MAX_LEVELS, 1.6, 0.04, 10.0, False, 3, False, True, True, True)
    with pytest.raises(ValueError, match="n_octaves"):
        build_detect_config(_lib.MAX_OCTAVES + 1, 3, 1.6, 0.04, 10.0, False, 3, False, True, True, True)


def test_c_abi_argument_checks_without_a_device():
    """The new C entry points reject bad sizes and misaligned rows before any
    CUDA call (so these run on a host without a GPU)."""
    import ctypes
    from pysift_b200 import _lib
    lib = _lib.load()
    sz = ctypes.c_size_t()
    assert lib.pysift_pca_basis_workspace_size(128, ctypes.byref(sz)) == 0 and sz.value >= 128 * 128 * 8
    assert lib.pysift_pca_basis_workspace_size(65, ctypes.byref(sz)) == -1       # odd D
    assert lib.pysift_pca_basis_workspace_size(130, ctypes.byref(sz)) == -1      # D > 128
    fake = ctypes.c_void_p(256)  # never dereferenced: the checks fail first
    assert lib.pysift_pca_basis(fake, 64, 65, fake, 1 << 20, fake, None, None) == -1   # P > D
    assert lib.pysift_pca_basis(fake, 64, 0, fake, 1 << 20, fake, None, None) == -1    # P < 1
    assert lib.pysift_pca_basis(fake, 64, 32, fake, 16, fake, None, None) == -2        # workspace too small
    # exact uint8 matching wants 16-byte aligned rows
    odd = ctypes.c_void_p(256 + 8)
    args = (0.75, fake, 1 << 30, fake, fake, fake, fake, fake, fake, fake, None)
    assert lib.pysift_match_u8_exact(odd, 10, fake, 10, 128, *args) == -1
    assert lib.pysift_match_u8_split_fp8(fake, 10, odd, 10, 128, *args) == -1
    assert "aligned" in lib.pysift_last_error().decode()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32, torch.float16, torch.bfloat16, torch.int64])
def test_differentiable_keypoint_tables_of_any_type(dtype):
    """Rows [octave, scale index, row, column, angle] of a table as torch holds
    them, in the library's layout; types numpy lacks too."""
    from types import SimpleNamespace
    from pysift_b200 import _lib, grad
    from pysift_b200.core import build_detect_config
    sift = SimpleNamespace(_cfg=build_detect_config(5, 3, 1.6, 0.04, 10.0, False, 3, False, False, True, True))
    table = torch.tensor([[0, 1, 30, 40, 90], [2, 3, 5, 9, 12], [1, 2, 17, 128, 250]], dtype=torch.float64).to(dtype)
    rows, n_oct, top, sizes, used = grad._levels_plan(table, sift, (96, 130))
    assert rows.dtype == torch.float32
    assert (rows[:, 0] == torch.tensor([1, 2 * _lib.MAX_LEVELS + 3, _lib.MAX_LEVELS + 2])).all()
    assert torch.equal(rows[:, 1:], table[:, 2:].float())
    assert (n_oct, top) == (3, 3) and sizes[:3] == [(96, 130), (48, 65), (24, 33)]
    assert [i for i, b in enumerate(used) if b] == [1, _lib.MAX_LEVELS + 2, 2 * _lib.MAX_LEVELS + 3]


def test_differentiable_descriptors_keep_maps_of_named_levels_only():
    """The backward workspace: the levels, and two floats a pixel for each level
    the table names (the adjoint chain needs nothing beside them)."""
    import ctypes
    from pysift_b200 import _lib
    from pysift_b200.core import build_detect_config
    cfg = build_detect_config(4, 3, 1.6, 0.04, 10.0, False, 3, False, False, True, True)
    H, W, n_oct, top = 300, 416, 3, 3

    def size(used, backward):
        n = ctypes.c_size_t()
        assert _lib.load().pysift_desc_levels_workspace_size(ctypes.byref(cfg), H, W, n_oct, top, used, backward,
                                                             ctypes.byref(n)) == _lib.OK
        return n.value

    planes = [-(-H >> o) * -(-(-(-W >> o)) // 32) * 32 * 4 for o in range(n_oct)]  # 256-byte multiples
    used = (ctypes.c_uint8 * (n_oct * _lib.MAX_LEVELS))()
    assert size(used, 0) == size(None, 0) == sum((top + 1) * p for p in planes)
    assert size(used, 1) == size(used, 0)
    used[1] = used[2] = used[_lib.MAX_LEVELS + 3] = 1
    assert size(used, 1) == size(used, 0) + 2 * (2 * planes[0] + planes[1])
    assert size(None, 1) == size(None, 0) + 2 * sum((top + 1) * p for p in planes)
