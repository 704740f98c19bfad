"""Reading binary records on both sides of the size (1 MiB) from which the flag pass runs on its own thread: all
records of full length (no offsets uploaded) or zeros among them, at an offset into a longer buffer, truncated
and corrupt ones; against the encoder's input."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5000, 9000])
@pytest.mark.parametrize("zeros", [False, True])
def test_round_trip(n, zeros):
    from sdpvibe_b200 import mpf
    from sdpvibe_b200.sdp_io import decode_bigfloats, encode_bigfloats
    L, nl = 26, 18
    g = torch.Generator(device="cuda").manual_seed(n)
    w = torch.randint(-(1 << 31), (1 << 31) - 1, (L, n), dtype=torch.int32, device="cuda", generator=g)
    A = mpf.normalize(w, torch.randint(-900, 900, (n,), device="cuda", generator=g), L)
    if zeros:
        A.m[:, ::3] = 0
        A.e[::3] = mpf.EZ
    rec = encode_bigfloats(A, nl)
    buf = b"\x07" * 11 + rec + b"tail"
    B, end = decode_bigfloats(buf, 11, n, nl, L)
    assert end == 11 + len(rec)
    C = mpf.normalize(B.m, B.e, L)                                   # decoded mantissas are not renormalised
    assert torch.equal(C.m, A.m) and torch.equal(C.e, A.e)
    with pytest.raises(ValueError):                                  # one record short
        decode_bigfloats(buf[:11 + len(rec) - 1], 11, n, nl, L)
    with pytest.raises(ValueError):
        decode_bigfloats(buf, len(buf) + 3, n, nl, L)
    bad = bytearray(buf)
    last = len(bad) - 4 - (1 if zeros and (n - 1) % 3 == 0 else 13 + 8 * nl)
    if bad[last] == 0:
        bad[last + 1:last + 5] = (nl + 1).to_bytes(4, "little")      # |size| > nl in the last record
        with pytest.raises(ValueError):
            decode_bigfloats(bytes(bad), 11, n, nl, L)


def test_pinned_buffer_is_free_on_return():
    """A pinned buffer overwritten right after the call: the records read are those of the call."""
    from sdpvibe_b200 import mpf
    from sdpvibe_b200.sdp_io import decode_bigfloats, encode_bigfloats
    L, nl, n = 26, 18, 400000
    rec = encode_bigfloats(mpf.from_float(torch.arange(1.0, n + 1.0, dtype=torch.float64, device="cuda"), L), nl)
    buf = torch.empty((len(rec),), dtype=torch.uint8, pin_memory=True)
    arr = buf.numpy()
    arr[:] = np.frombuffer(rec, dtype=np.uint8)
    A, _ = decode_bigfloats(rec, 0, n, nl, L)
    for _ in range(3):
        B, _ = decode_bigfloats(arr, 0, n, nl, L)
        arr[-(1 << 20):] = 0
        assert torch.equal(A.m, B.m) and torch.equal(A.e, B.e)
        arr[:] = np.frombuffer(rec, dtype=np.uint8)


def test_count_beyond_the_buffer():
    from sdpvibe_b200.sdp_io import decode_bigfloats
    with pytest.raises(ValueError):
        decode_bigfloats(b"\x01" * 64, 0, 1 << 36, 18, 26)


def test_round_trip_zeros_above_the_limit():
    """zeros among records of over 1 MiB (9000 records with a third of them zero stay below it)"""
    test_round_trip(15000, True)
