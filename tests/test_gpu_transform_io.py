"""Upload, load_forward and download of the Transform trait on the B200: field values of uploaded
coefficients, and load_forward's padding, at the lengths and row sizes where the device staging and
the element order change (shared-memory lengths keep natural order, longer ones the kernels')."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P1 = (1 << 31) - 1


@pytest.fixture(scope="module")
def gpu():
    from montmul_b200 import B200
    return B200()


def _coeffs(seed, size):
    c = np.random.default_rng(seed).integers(0, 1 << 32, size=size, dtype=np.uint64).astype(np.uint32)
    c[: min(8, size)] = [0, 1, P1 - 1, P1, P1 + 1, 2 * P1, 0xFFFFFFFE, 0xFFFFFFFF][: min(8, size)]
    return c


# The last two pass the staging bounds (2^24 words per upload copy, 2^20 elements per download copy).
@pytest.mark.parametrize("length,count", [(8, 1), (16, 3), (1 << 14, 2), (1 << 15, 3), (1 << 18, 1), (64, 270_000), (1 << 15, 520)])
def test_upload_then_download_is_the_coefficients(gpu, length, count):
    c = _coeffs(length + count, length * count)
    f1, f2 = gpu.download_raw(gpu.upload(c, length, count))
    want = c.reshape(count, 2, length // 2).transpose(0, 2, 1).reshape(-1, 2)
    assert np.array_equal(f2, want.astype(np.uint64)) and np.array_equal(f1, want % P1)


@pytest.mark.parametrize("length,k", [(8, 1), (64, 31), (64, 33), (64, 64), (1 << 14, 8191), (1 << 15, 1), (1 << 15, 16_385)])
def test_load_forward_pads_with_zeros(gpu, length, k):
    count = 3
    c = _coeffs(k, k * count)
    padded = np.zeros((count, length), np.uint32)
    padded[:, :k] = c.reshape(count, k)
    a = gpu.load_forward(c, k, length, count)
    b = gpu.upload(padded, length, count)
    gpu.forward(b, length, count)
    for x, y in zip(gpu.download_raw(a), gpu.download_raw(b)):
        assert np.array_equal(x, y)


def test_upload_and_download_at_the_memory_limit(gpu):
    """With room for the buffer and little else: the upload has no staging of its own, and a download whose staging
    does not fit puts the elements in order on the host."""
    import torch
    length, count = 1 << 15, 512   # 192 MiB of elements from 64 MiB of coefficients
    c = _coeffs(7, length * count)
    small = gpu.upload(c[:length], length, 1)   # the kernels are loaded
    gpu.download_raw(small)
    torch.zeros(1, device="cuda")
    torch.cuda.empty_cache()
    fill = []
    try:
        fill.append(torch.empty(gpu.free_memory() - (226 << 20), dtype=torch.uint8, device="cuda"))
        buf = gpu.upload(c, length, count)
        room = gpu.free_memory() - (8 << 20)
        if room > 0:
            fill.append(torch.empty(room, dtype=torch.uint8, device="cuda"))
        f1, f2 = gpu.download_raw(buf)
    finally:
        del fill
        torch.cuda.empty_cache()
    want = c.reshape(count, 2, length // 2).transpose(0, 2, 1).reshape(-1, 2)
    assert np.array_equal(f2, want.astype(np.uint64)) and np.array_equal(f1, want % P1)
