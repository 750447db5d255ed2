"""Programs and listings are cut into runs that several host threads lower and print: the cuts must not show."""
import numpy as np
import pytest

import cubit_b200


@pytest.fixture(scope="module")
def codec():
    c = cubit_b200.Codec(devices=())
    yield c
    c.close()


# (in front, statement, behind); {label} is the address of a label of the program.
LINES = [("", "IADD3 R5, PT, PT, R9, R4, R5", ""), ("[B------:R-:W-:-:S01] ", "FADD R1, R2, R3", ""), ("", "@P0 BRA {label}", ""),
         ("/*0010*/ ", "NOP", " // comment ; NOP"), ("{here}: ", "EXIT", ""), ("", "__raw__0x1234", " # comment"),
         ("", "BSSY B0, {label}", "")]


@pytest.mark.parametrize("lines", [1, 7, 8, 600, 4001])
@pytest.mark.parametrize("ending", ["\n", " ;\n", " ;\r\n"])
def test_program_equals_its_statements(codec, lines, ending):
    """Every statement of a program lowers to what it lowers to alone at its address, with its label (also of a run behind
    it) spelled as an address: 4,001 lines of about 30 bytes are several runs of 16 KiB."""
    base, period = 0x40, len(LINES)
    text = ["%%% skipped: not an instruction"]
    alone = []
    for i in range(lines):
        front, statement, behind = LINES[i % period]
        target = (i * 7919) % lines // period * period + 4     # the line of a label, or beyond the program
        name = f"L_{target}" if target < lines else "0x10"
        addr = "0x%x" % (base + 16 * target) if target < lines else "0x10"
        text.append((front + statement + ("" if ";" in ending and behind else behind)).format(here=f"L_{i}", label=name))
        alone.append(codec.lower_text(statement.format(label=addr), base + 16 * i, program=False))
    got = codec.lower_text(ending.join(text) + ending, base)
    assert len(got[0]) == lines
    for k, plane in enumerate(got):
        want = np.concatenate([a[k] for a in alone], axis=1 if k == 1 else 0)
        assert (plane == want).all(), ("form", "slots", "ctrl", "clear", "set")[k]


@pytest.mark.parametrize("at", [0, 700, 2999])
def test_first_failing_statement_is_reported(codec, at):
    """The message names the earliest statement without a table entry, whichever run it is in."""
    lines = ["NOP"] * 3000
    lines[at] = "FADD P0, P1"
    lines[2999] = "IADD3 SR_TID.X" if at != 2999 else lines[2999]
    with pytest.raises(ValueError, match=f"^encode error at addr 0x{16 * at:x}: no operand-compatible table entry; attempted keys: "
                                         r"\[\(FADD_P_P, \"\"\) not in table"):
        codec.lower_text("\n".join(lines))


@pytest.mark.parametrize("n", [1, 191, 192, 193, 1000])
def test_printed_lines_keep_their_order(codec, n):
    """print_text over several runs of lines equals printing word by word."""
    variants = np.arange(n, dtype=np.uint32) * 37 % codec.table_info()[1]
    words = np.arange(16 * n, dtype=np.uint32).astype(np.uint8).reshape(n, 16)
    slots = (np.arange(8 * n, dtype=np.uint32) * 2654435761).reshape(8, n)
    form, ctrl = variants.astype(np.uint16), np.arange(n, dtype=np.uint32) << 20
    lines = codec.print_text(words, 0x100, (form, slots, ctrl))
    assert len(lines) == n
    for i in range(0, n, max(1, n // 50)):
        one = codec.print_text(words[i:i + 1], 0x100 + 16 * i, (form[i:i + 1], slots[:, i:i + 1], ctrl[i:i + 1]))
        assert one == [lines[i]]
