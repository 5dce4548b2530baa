"""n whose first candidate q is a Mersenne number with a prime exponent: it passes
the strong test to base 2 and has no factor below 4096, so only the other bases
reject it.  Beyond 1024 bits their kernel alone runs them (up to 1024 bits the first
survivors' bases run beside base 2); 2, 3 and 4 limbs a lane."""
import importlib.util
import os

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


@pytest.fixture(scope="module")
def B():
    spec = importlib.util.spec_from_file_location("big_oracle", os.path.join(ROOT, "oracle", "big_oracle.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("exponent", [1277, 2029, 2207, 3067, 3079, 4091])
def test_other_bases_reject_a_base2_pseudoprime(ctx, B, exponent):
    m = 2**exponent - 1
    assert B.sprp(m, 2) and not B.sprp(m, 3)
    assert all(m % r for r in B.small_primes(4096))
    assert ctx.check_big(m + 3, p_limit=3)[:2] == (0, 0)
    # the passers behind it are still tried, in order
    want = B.minimal_p(m + 5, p_limit=100, primes=B.small_primes(100))
    assert want != 5 and ctx.check_big(m + 5, p_limit=100)[0] == want
