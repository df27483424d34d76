"""Any sized iterable of integers serves as the primes of a call."""
import pytest

from rabung_atlas32_b200 import _lib, codec
from rabung_atlas32_b200.census import _as_u32_array, to_records


@pytest.mark.parametrize("primes", [[3, 5, 7], (3, 5, 7), b"\x03\x05\x07", bytearray(b"\x03\x05\x07\x0b"),
                                    memoryview(b"\x03\x05"), range(3, 9, 2), {3: "a", 5: "b"}, {3, 5}, [], b""])
def test_sized_iterables_of_integers(primes):
    want = [int(p) for p in primes]
    assert list(_as_u32_array(primes)) == want
    n = sum(bin(codec.expected_mask(p)).count("1") for p in want)
    out = (_lib.cz_profile * max(1, n))()
    for i in range(n):
        out[i].r, out[i].M, out[i].L, out[i].witness, out[i].K = 2, i + 1, 3, 4, 5
    recs = to_records(primes, out, list(range(len(want))))
    assert [(r.p, r.a4, len(r.profiles)) for r in recs] == \
           [(p, i, bin(codec.expected_mask(p)).count("1")) for i, p in enumerate(want)]
    assert [v.M for r in recs for v in r.profiles] == list(range(1, n + 1))


@pytest.mark.parametrize("primes", [[-1], [1 << 32], [3, 1 << 40]])
def test_out_of_the_domain(primes):
    with pytest.raises(ValueError, match="32-bit domain"):
        _as_u32_array(primes)
