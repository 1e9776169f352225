"""The sort of up to 32,768 pairs, which runs all its passes in one launch of
one CTA or of a cluster of 8 or 16, against numpy's stable argsort: both sides
of every size where the form changes, an odd number of passes, the largest key
(the value that pads the last tile), and all keys equal. Bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 1024, 1025, 2048, 2049, 5000, 8192, 8193, 16384, 16385, 32767, 32768, 32769])
@pytest.mark.parametrize("bits", [8, 24, 30, 32])
def test_one_launch_sort(upf_lib, n, bits):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + bits)
    for kind in ("random", "largest", "equal", "nearly sorted"):
        keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
        if kind == "largest":
            keys[rng.random(n) < 0.3] = (1 << bits) - 1
        elif kind == "equal":
            keys[:] = keys[0]
        elif kind == "nearly sorted":
            keys = np.sort(keys)
            keys[:-1:7], keys[1::7] = keys[1::7].copy(), keys[:-1:7].copy()
        vals = rng.permutation(n).astype(np.uint32)
        k = torch.from_numpy(keys.view(np.int32)).cuda()
        v = torch.from_numpy(vals.view(np.int32)).cuda()
        nbytes = upf_lib.lib().upf_radix_sort_temp_bytes(n)
        tmp = torch.empty(max(nbytes, 1), dtype=torch.uint8, device="cuda")
        upf_lib.check(upf_lib.lib().upf_radix_sort_pairs(C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), n,
                                                         bits, C.c_void_p(tmp.data_ptr()), nbytes, None),
                      "upf_radix_sort_pairs")
        torch.cuda.synchronize()
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[order]), kind
        assert np.array_equal(v.cpu().numpy().view(np.uint32), vals[order]), kind
