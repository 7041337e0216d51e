"""Size limit of the set-up kernel from its source (CPU only): the shared memory of a CTA (227 KB) holds
at least every molecule that 140 bytes an atom and 8 a shell did, for one to three shells an atom, and
the carve-up of the kernel stays inside what the host asks for."""
import os
import re

SETUP = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gfn1-rs_b200", "csrc", "setup.cu")
MAX_REF = 5
SMEM = 227 * 1024


def _bytes(nat):
    with open(SETUP) as fh:
        text = fh.read()
    expr = re.search(r"size_t setup_smem_bytes\(int max_nat\) \{\s*return ([^;]*);", text).group(1)
    expr = expr.replace("sizeof(double)", "8").replace("sizeof(int)", "4").replace("(size_t)max_nat", str(nat))
    return eval(expr.replace("kMaxRef", str(MAX_REF)))  # noqa: S307 - the formula above


def test_limit_is_at_least_what_it_was():
    limit = max(n for n in range(1, 3000) if _bytes(n) <= SMEM)
    for shells in (1, 2, 3):
        before = max(n for n in range(1, 3000) if 128 * n + 256 + 4 * (3 * n + 2 + 2 * shells * n) <= SMEM)
        assert limit >= before
    assert limit == 1660


def test_carve_up():
    """Doubles: xyz 3, cn, cnd, edis, two times kMaxRef weights; ints: zs, two offset tables, three counts.
    The pair tables (8 + 16 bytes a shell, three shells an atom) lie in the weights' 80 bytes an atom."""
    for nat in (1, 3, 1660):
        at = 8 * (3 + 1 + 1 + 1 + 2 * MAX_REF) * nat + 4 * (nat + 2 * (nat + 1) + 3)
        assert at <= _bytes(nat)
        assert 3 * nat * 24 <= 8 * 2 * MAX_REF * nat
