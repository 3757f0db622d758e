"""The per-16 block-scaled product with its scales in the reference's layout (one launch, up to one tile per SM) against the route
that turns them into atoms first: equal bytes at the edges of tiles, of K stages and of the sizes that take either route."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, offset, seed=0):
    """Random codes and UE8M0 bytes 2^-27 .. 2^13, with rows of zero codes; the scales `offset` bytes into a buffer."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    byte = lambda lo, hi, *s: torch.randint(lo, hi, s, generator=g, device="cuda", dtype=torch.int32).to(torch.uint8)
    a, b = byte(0, 256, M, K // 2), byte(0, 256, N, K // 2)
    a[M // 2] = 0

    def scales(n):
        buf = byte(100, 141, offset + K // 16 * n)
        return buf[offset:].view(K // 16, n)

    return a, b, scales(M // 2), scales(N)


@pytest.mark.parametrize("K", [32, 256, 288, 1024, 1056, 2048])
@pytest.mark.parametrize("M,N", [(2, 1), (2, 7), (64, 128), (126, 129), (128, 200), (130, 255), (254, 257), (1022, 512), (1150, 2048), (1154, 2048), (4734, 512), (4738, 512)])
def test_natural_scales_equal_the_atoms_route(monkeypatch, M, N, K):
    from velox_voice_b200 import _lib, ops
    from test_host_path_gpu import _NoHost

    ops._host()
    one = -(-M // 128) * -(-N // 128) <= torch.cuda.get_device_properties(0).multi_processor_count and K <= 1024
    assert bool(_lib.load().vx_bsgemm_natural_sf_supported(M, N, K)) == one
    for offset in (0, 1, 2):
        a, b, sa, sb = _operands(M, N, K, offset, seed=offset)
        sb[0, 0] = 255  # UE8M0 NaN: its row of B poisons its column and nothing else
        got = ops.dgx_mxfp4_blkscale_gemm(a, b, sa, sb)
        with monkeypatch.context() as m:
            m.setattr(ops, "_native", _NoHost())
            want = ops.dgx_mxfp4_blkscale_gemm(a, b, sa, sb)
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(), want.nan_to_num()), (M, N, K, offset)
    assert _lib.device_status() == 0


def test_natural_scales_refusals():
    """What the flag does not take is an argument error before any launch."""
    import ctypes as C

    from velox_voice_b200 import _lib

    lib = _lib.load()
    assert [lib.vx_bsgemm_natural_sf_supported(*s) for s in ((0, 8, 64), (3, 8, 64), (2, 8, 48), (2, 0, 64), (2, 8, 64))] == [0, 0, 0, 0, 1]
    a, b, sa, sb = _operands(64, 64, 64, 0)
    out = torch.empty(64, 64, device="cuda")

    def call(**kw):
        f = dict(fmt=_lib.FMT_BLK16_A, M=64, N=64, K=64, a_codes=a.data_ptr(), lda=32, b_codes=b.data_ptr(), ldb=32, a_scales=sa.data_ptr(),
                 b_scales=sb.data_ptr(), epilogue=_lib.EPI_NONE, out_dtype=_lib.DT_F32, out=out.data_ptr(), ldo=64, flags=2048)
        f.update(kw)
        d = _lib.GemmDesc()
        d.struct_size = C.sizeof(d)
        for k, v in f.items():
            setattr(d, k, v)
        return lib.vx_bsgemm(C.byref(d), torch.cuda.current_stream().cuda_stream)

    assert call() == 0
    torch.cuda.synchronize()
    for kw in (dict(fmt=_lib.FMT_MX32), dict(epilogue=_lib.EPI_BIAS), dict(out_dtype=_lib.DT_BF16), dict(M=63), dict(flags=2048 + 4), dict(M=128 * 200)):
        assert call(**kw) == -1, kw
