"""N-Triples ingest where its kernel's parts meet: pieces of 16384 bytes of
text (plus 1024 of the next), 2048 listed lines per piece, terms of any length
and alignment, and the term table's searches (few hash bits: long searches;
one bit: searches that give up, resolved on the host)."""
import numpy as np
import pytest

from oracle import oracle_py

pytestmark = pytest.mark.gpu
PIECE = 16384


def statements(rng, n, terms=400, longest=60):
    """Statements over a pool of terms of mixed lengths, some of them prefixes
    of each other or equal up to the dictionary they belong to."""
    def word():
        return "".join(rng.choice(list("abcdefg0123456789/#%.:"), size=rng.integers(1, longest)))

    iris = [f"<{word()}>" for _ in range(terms)] + ["<a>", "<ab>", "<abc>", "<abcdefgh>", "<abcdefghi>"]
    blanks = [f"_:b{i}" for i in range(terms // 10 + 1)] + ["_:b1x", "_:b.x"]
    lits = [f'"{word()}"' for _ in range(terms // 2)] + ['"a"', '"a"@en', '"a"@en-GB', '"a"^^<abc>', '"q\\"uote"', '""']
    preds = iris[:7] + ["<abc>"]
    out = []
    for _ in range(n):
        s = rng.choice(iris + blanks)
        o = rng.choice(iris + blanks + lits)
        ws = rng.choice([" ", "\t", "  "])
        out.append(f"{s}{ws}{rng.choice(preds)}{ws}{o}{rng.choice([' .', '.', ' . # note', ' .\r'])}"
                   if not (o.startswith("_:")) else f"{s} {rng.choice(preds)} {o} .")
    return out


def check(ctx, text, bits=63):
    import vedas_gb300 as vg

    if isinstance(text, str):
        text = text.encode()
    for literal_dict in (False, True):
        s, p, o, d = oracle_py.ingest_ntriples(text, literal_dict)
        vg.set_ingest_hash_bits(bits)
        try:
            ing = vg.ingest_ntriples(ctx, text, literal_dict=literal_dict)
        finally:
            vg.set_ingest_hash_bits(63)
        assert ing.n == len(s)
        for got, want in zip(ing.columns(), (s, p, o)):
            assert np.array_equal(got, want)
        for k in ("so", "p", "l"):
            assert ing.dict.terms(k) == d[k]
        ing.free()


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("bits", [63, 3, 1])
def test_mixed_terms(ctx, seed, bits):
    rng = np.random.default_rng(seed)
    lines = statements(rng, 3000)
    for _ in range(200):
        lines.insert(int(rng.integers(0, len(lines))), str(rng.choice(["", "# comment", "   ", "\t# x", "\r"])))
    check(ctx, "\n".join(lines) + ("\n" if seed % 2 else ""), bits)


def test_a_search_gives_up(ctx):
    """Far more terms than a search visits, all from two places of the table."""
    lines = [f"<s{i}> <p> <o{i * 7919 % 60000}> ." for i in range(20000)]
    check(ctx, "\n".join(lines), 1)


@pytest.mark.parametrize("shift", [-2, -1, 0, 1, 2, 1023, 1024, 1025])
def test_lines_at_piece_ends(ctx, shift):
    """A newline lands `shift` bytes from the end of the first piece."""
    head = "<x> <y> <z> .\n" * 900
    pad = PIECE + shift - len(head) - len('<pad> <y> "" .')
    text = head + '<pad> <y> "' + "v" * pad + '" .\n' + "<last> <y> <z> .\n" * 300
    check(ctx, text)
    check(ctx, text[:-1])
    check(ctx, head + '<pad> <y> "' + "v" * pad + '" .')


@pytest.mark.parametrize("length", [1000, 1024, 5000, PIECE, 3 * PIECE + 17, 200_001])
def test_long_terms(ctx, length):
    lines = ["<a> <b> <c> ."] * 40
    for i, tail in enumerate(["x", "y", "x"]):
        lines += [f"<{'k' * length}{tail}> <b> \"{'m' * (length + i)}\" .", "<a> <b> <d> ."]
    check(ctx, "\n".join(lines) + "\n")


@pytest.mark.parametrize("blank", [2047, 2048, 2049, 16383, 16384, 40_000])
def test_many_short_lines(ctx, blank):
    check(ctx, "\n" * blank + "<a> <b> <c> .\n" + "\n" * blank + "<d> <b> <a> .\n" + "#\n" * blank)


@pytest.mark.parametrize("text", ["", "\n", "#", "<a> <b> <c>.", " \t<a>\t<b> _:x . \n"])
def test_tiny_texts(ctx, text):
    check(ctx, text)


@pytest.mark.parametrize("bad", ["<a> <b> .", "<a> <b> <c>", "<a><b> <c> .", "\"l\" <b> <c> .", "<a> _:b <c> .",
                                 "<a> <b> \"open .", "<a> <b> <c> . x", "<a b> <c> <d> .", "<a> <b> \"x\"^^y ."])
def test_malformed_lines_are_numbered(ctx, bad):
    import vedas_gb300 as vg

    lines = ["<a> <b> <c> ."] * 3000
    lines[2500] = lines[2900] = bad
    with pytest.raises(vg.VgError, match="line 2501") as e:
        vg.ingest_ntriples(ctx, "\n".join(lines).encode())
    assert e.value.status == 6


def test_dictionary_texts_in_chunks(ctx):
    """Dictionary texts of more than 64 MiB come to the host in several copies
    (a term longer than that in one of its own)."""
    import vedas_gb300 as vg

    long = "k" * (70 << 20)
    lines = [f"<s{i}> <p> <{'v' * 900}{i}> ." for i in range(40_000)] + [f"<{long}> <p> \"{long}\" .", "<z> <p> <s1> ."]
    text = "\n".join(lines).encode()
    ing = vg.ingest_ntriples(ctx, text, literal_dict=True)
    n = 40_000
    assert ing.dict.size("so") == 2 * n + 2 and ing.dict.size("l") == 1
    for i in (0, 1, n // 2, n - 1):
        assert ing.dict.term("so", 2 * i + 1) == f"<s{i}>"
        assert ing.dict.term("so", 2 * i + 2) == f"<{'v' * 900}{i}>"
    assert ing.dict.term("so", 2 * n + 1) == f"<{long}>" and ing.dict.term("so", 2 * n + 2) == "<z>"
    assert ing.dict.term("l", 50_000_000) == f'"{long}"' and ing.dict.term("p", 1) == "<p>"
    s, p, o = ing.columns()
    assert np.array_equal(s, np.append(np.arange(n) * 2 + 1, [2 * n + 1, 2 * n + 2]))
    assert np.array_equal(o, np.append(np.arange(n) * 2 + 2, [50_000_000, 3])) and (p == 1).all()
    ing.free()


PART = 16 << 20   # longer texts than two such parts are parsed as they arrive


def fill(rng, size):
    block = "\n".join(statements(rng, 2000)) + "\n"
    return block * (size // len(block) + 1)


@pytest.mark.parametrize("edge", [-1500, -1, 0, 700])
def test_text_in_parts(ctx, edge):
    """Lines of 3,000 bytes around the end of a part, one longer than a part,
    blank lines, and no newline at the end."""
    rng = np.random.default_rng(edge + 2000)
    text = fill(rng, 2 * PART + PART // 2)
    at = text.rindex("\n", 0, PART + edge - 1400) + 1
    text = text[:at] + f'<q> <r> "{"w" * 3000}" .\n\n<q2> <r> "{"w" * 3000}" .\n' + text[at:2 * PART] + \
        f'\n<far> <r> "{"z" * (PART + 100)}" .\n' + text[:100_000].rsplit("\n", 1)[0]
    check(ctx, mend(text))


def mend(text):
    """The line that the cut at 2 * PART broke becomes a comment."""
    cut = text.index("\n<far>")
    b = text.rindex("\n", 0, cut) + 1
    return text[:b] + "#" + text[b:]


def test_more_lines_than_samples_promise(ctx):
    """Long comments, where the samples fall, between runs of short lines."""
    rng = np.random.default_rng(8)
    short = "\n".join(statements(rng, 300)) + "\n" * 2000
    check(ctx, ("#" + "x" * (1 << 20) + "\n" + short) * 34)


def test_malformed_line_in_a_later_part(ctx):
    import vedas_gb300 as vg

    lines = ["<a> <b> <c> ."] * (3 * PART // 14)
    lines[-7] = "<a> <b>"
    with pytest.raises(vg.VgError, match=f"line {len(lines) - 6}"):
        vg.ingest_ntriples(ctx, "\n".join(lines).encode())
