"""Dictionary files of many terms in any order: every term comes back at its
id, with spaces, without text, from a file that does not end its last line."""
import random

import pytest


@pytest.mark.parametrize("sizes", [(0, 0, 0), (1, 0, 0), (3, 1, 2), (20_000, 40, 5000)])
@pytest.mark.parametrize("shuffle", [False, True])
def test_terms_at_their_ids(built, tmp_path, sizes, shuffle):
    import vedas_gb300 as vg

    rng = random.Random(sum(sizes))
    want, lines = [], []
    for base, n in zip((1, 1, 50_000_000), sizes):
        terms = ["x" * rng.randrange(0, 40) + (" y %d" % i if i % 3 else "") for i in range(n)]
        entries = [f"{base + i} {t}" for i, t in enumerate(terms)]
        if shuffle:
            rng.shuffle(entries)
        lines += [str(n)] + entries
        want.append(terms)
    path = tmp_path / "a.vdd"
    path.write_text("\n".join(lines))
    d = vg.Dict.open(str(path))
    kinds = ("so", "p", "l")
    assert [d.size(k) for k in kinds] == list(sizes)
    for k, terms in zip(kinds, want):
        assert list(d.terms(k)) == terms
    again = tmp_path / "b.vdd"
    d.write(str(again))
    d.close()
    d = vg.Dict.open(str(again))
    for k, terms in zip(kinds, want):
        assert list(d.terms(k)) == terms
    d.close()


@pytest.mark.parametrize("text", ["", "1\n", "1\nx y\n", "1\n1x\n", "2\n1 a\n3 b\n0\n0\n", "1\n1 a\n0\n"])
def test_broken_files_are_refused(built, tmp_path, text):
    import vedas_gb300 as vg

    path = tmp_path / "a.vdd"
    path.write_text(text)
    with pytest.raises(Exception):
        vg.Dict.open(str(path))
