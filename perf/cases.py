"""The work whose speed matters to a user of this package, as cases that can be timed.

A case is a dict of plain values with a `kind`:

  word       one instruction word through the reference's single-word functions: decode, to_sass, encode
  decode     a device-resident batch of words -> records (`Codec.decode_device`)
  encode     device-resident records -> words (`Codec.encode_device`)
  roundtrip  device-resident words -> faithfulness status (`Codec.roundtrip_device`)
  host       the same three on numpy arrays (`Codec.decode_batch` / `encode_batch` / `roundtrip_batch`)
  cubin      every kernel of a multi-kernel cubin image -> records (`Codec.decode_elf`)
  listing    a cubin image -> its listing (`Codec.disassemble`, plain or re-assemblable)
  assemble   a program's text with labels and control codes -> words (`Codec.encode_text`)

Words come from the package's seeded stream generator in its three mixes (uniform over the forms, Zipf, the MMA-heavy
family mix), with a share of raw random words where `noise_ppm` says so.  Every result is whole numbers or text, and
has to be the same to the bit.
"""
import math

import numpy as np
import torch

import cubit_b200

MI = 1 << 20
MIXES = {"uniform": cubit_b200.MIX_UNIFORM, "zipf": cubit_b200.MIX_ZIPF, "family": cubit_b200.MIX_FAMILY}

# Upper ends of the ranges; the listed cases reach them.
MOST_DEVICE = 64 * MI        # words of a device-resident batch (the batch decode and encode configurations)
MOST_HOST = 9 * MI           # words of a numpy batch
MOST_KERNELS = 96            # kernels of a cubin, 20,000 words each in the median
MOST_LINES = 20000           # words of a listing, lines of a program: one kernel of median length


def listed():
    return [
        # Looking at one instruction: what an interactive user or a script over single words calls.
        {"name": "one_word", "kind": "word", "mix": "uniform", "addr": 256},
        # A short kernel that is already on the device, ragged: launch latency is what counts.
        {"name": "decode_short_kernel", "kind": "decode", "n": 4097, "mix": "uniform", "noise_ppm": 0, "counts": False},
        # The reference corpus's size, encoded from records on the device.
        {"name": "encode_corpus", "kind": "encode", "n": 47244, "mix": "uniform", "noise_ppm": 0},
        # The same size as numpy arrays, the form in which the words of one binary usually come.
        {"name": "decode_corpus_host", "kind": "host", "call": "decode", "n": 47244, "mix": "uniform", "noise_ppm": 0, "pinned": False},
        # A library's worth of code on the device, with undecodable words in it, counted.
        {"name": "decode_library", "kind": "decode", "n": 1000003, "mix": "family", "noise_ppm": 5000, "counts": True},
        # The large batch: decode, encode, and the faithfulness check with 1 % words that match no form.
        {"name": "decode_batch", "kind": "decode", "n": 64 * MI, "mix": "zipf", "noise_ppm": 0, "counts": False},
        {"name": "encode_batch", "kind": "encode", "n": 64 * MI, "mix": "zipf", "noise_ppm": 0},
        {"name": "roundtrip_batch", "kind": "roundtrip", "n": 64 * MI, "mix": "zipf", "noise_ppm": 10000, "counts": True},
        # Checking a dump that sits in ordinary host memory.
        {"name": "roundtrip_host", "kind": "host", "call": "roundtrip", "n": 9 * MI + 5, "mix": "zipf", "noise_ppm": 10000, "pinned": False},
        # A multi-kernel binary, MMA-heavy, all kernels in one call.
        {"name": "cubin_decode", "kind": "cubin", "kernels": 96, "mix": "family"},
        # Disassembling a kernel to a listing that assembles back, and assembling a program of that length.
        {"name": "listing_frozen", "kind": "listing", "n": 20000, "kernels": 3, "mix": "family", "frozen": True},
        {"name": "assemble_program", "kind": "assemble", "n": 20000, "mix": "family"},
    ]


def _log_size(rng, low, high):
    """A size spread over the logarithm of [low, high]; nearly all of them are ragged."""
    return max(low, min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(["word", "decode", "decode", "encode", "roundtrip", "host", "host", "cubin", "listing", "assemble"])
    mix = rng.choice(sorted(MIXES))
    noise = rng.choice([0, 0, 1000, 10000, 50000])
    if kind == "word":
        return {"kind": kind, "mix": mix, "addr": 16 * rng.randrange(1 << 16)}
    if kind == "decode" or kind == "roundtrip":
        return {"kind": kind, "n": _log_size(rng, 1, MOST_DEVICE), "mix": mix, "noise_ppm": noise, "counts": rng.random() < 0.5}
    if kind == "encode":
        return {"kind": kind, "n": _log_size(rng, 1, MOST_DEVICE), "mix": mix, "noise_ppm": noise}
    if kind == "host":
        call = rng.choice(["decode", "encode", "roundtrip"])
        # 54 bytes a word cross the bus for records, 17 for a status: the largest record batch costs what the largest check does.
        most = MOST_HOST if call == "roundtrip" else MOST_HOST // 8
        return {"kind": kind, "call": call, "n": _log_size(rng, 1, most), "mix": mix, "noise_ppm": noise, "pinned": rng.random() < 0.3}
    if kind == "cubin":
        return {"kind": kind, "kernels": _log_size(rng, 1, MOST_KERNELS), "mix": mix}
    if kind == "listing":
        n = _log_size(rng, 16, MOST_LINES)
        return {"kind": kind, "n": n, "kernels": rng.randint(1, max(1, min(8, n // 16))), "mix": mix, "frozen": rng.random() < 0.6}
    return {"kind": kind, "n": _log_size(rng, 16, MOST_LINES), "mix": mix}


# ---- inputs ----------------------------------------------------------------------------------

_codec = None


def codec():
    """One table on the first GPU for the whole process, as a program keeps it."""
    global _codec
    if _codec is None:
        _codec = cubit_b200.Codec(devices=(0,))
    return _codec


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _device_planes(n):
    empty = dict(dtype=torch.int32, device="cuda")
    return torch.empty(n, dtype=torch.int16, device="cuda"), torch.empty((8, n), **empty), torch.empty(n, **empty)


def _device_words(n):
    return torch.empty((n, 16), dtype=torch.uint8, device="cuda")


def _host_stream(case, seed, n):
    """(words, form, slots, ctrl) of the seeded stream as numpy arrays."""
    return codec().synth(MIXES[case["mix"]], seed, n, case.get("noise_ppm", 0))


def _host_copy(a, pinned):
    if not pinned:
        return a
    held = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True).numpy().view(a.dtype).reshape(a.shape)
    held[...] = a
    return held


def kernel_lengths(case):
    """Words of each kernel: lognormal with a median of 20,000 for a cubin, an even split for a listing."""
    k = case["kernels"]
    if case["kind"] == "listing":
        return [case["n"] // k + (i < case["n"] % k) for i in range(k)]
    drawn = np.exp(np.random.default_rng(1000 + k).normal(math.log(20000.0), 1.0, k))
    return [int(v) for v in np.clip(drawn, 2000, 200000)]


def _cubin(case, seed):
    lengths = kernel_lengths(case)
    words = _host_stream(case, seed, sum(lengths))[0]
    at = np.concatenate([[0], np.cumsum(lengths)])
    return cubit_b200.build_cubin([("kernel_%03d" % i, words[at[i]:at[i + 1]].tobytes()) for i in range(len(lengths))])


def _word(case, seed):
    """The first word of the stream whose text reads back (a sibling form's syntax does not always)."""
    for row in _host_stream(case, seed, 256)[0]:
        lo, hi = (int(v) for v in row.view(np.uint64))
        try:
            codec().encode(codec().to_sass(lo, hi, case["addr"]), case["addr"])
            return lo, hi
        except ValueError:
            continue
    raise RuntimeError("no word of the stream reads back")


def _program(case, seed):
    """Statements that assemble: lines of a re-assemblable listing, with a label and a branch every few lines."""
    n, lines, first = case["n"], [], 0
    while len(lines) < n:
        words = codec().synth(MIXES[case["mix"]], seed, 3 * n, 0, first)[0]
        first += 3 * n
        text = codec().disassemble(cubit_b200.build_cubin([("k", words.tobytes())]), frozen=True)
        lines += [t.strip() for t in text.splitlines() if t.startswith("    [") and "L_" not in t]
    rng = np.random.default_rng(seed)
    target = rng.integers(0, (n + 23) // 24, n)
    out = []
    for i, line in enumerate(lines[:n]):
        if i % 32 == 17:
            line = "[B------:R-:W-:-:S05] @P%d BRA L_%d ;" % (i % 7, target[i])
        out.append("L_%d:  %s" % (i // 24, line) if i % 24 == 0 else "    " + line)
    return "\n".join(out) + "\n"


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "word":
        state["lo"], state["hi"] = _word(case, seed)
        state.update(fields=np.zeros((32, 3), np.uint64), names=np.zeros(256, np.uint8), text=np.zeros(256, np.uint8))
    elif kind in ("decode", "roundtrip", "encode"):
        n = case["n"]
        words, (form, slots, ctrl) = _device_words(n), _device_planes(n)
        codec().synth_device(MIXES[case["mix"]], seed, n, words.data_ptr(), form.data_ptr(), slots.data_ptr(), ctrl.data_ptr(),
                             case["noise_ppm"], 0, _stream())
        if kind == "encode":
            state.update(form=form, slots=slots, ctrl=ctrl, words=torch.zeros_like(words))
        elif kind == "decode":
            state.update(words=words, form=form.zero_(), slots=slots.zero_(), ctrl=ctrl.zero_())
        else:
            state.update(words=words, status=torch.zeros(n, dtype=torch.uint8, device="cuda"))
    elif kind == "host":
        words, form, slots, ctrl = (_host_copy(a, case["pinned"]) for a in _host_stream(case, seed, case["n"]))
        state.update(dict(form=form, slots=slots, ctrl=ctrl) if case["call"] == "encode" else dict(words=words))
    elif kind in ("cubin", "listing"):
        state["image"] = _cubin(case, seed)
        if kind == "listing":
            state["text"] = np.zeros(192 * case["n"] + 4096 * case["kernels"], np.uint8)
    else:
        state["text"] = _program(case, seed)
    return state


# ---- one pass ----------------------------------------------------------------------------------

def _signed(a):
    """The same bits as a signed type, which every consumer of arrays knows."""
    return a.view(a.dtype.str.replace("u", "i")) if a.dtype.kind == "u" and a.dtype.itemsize > 1 else a


def _place(held, text):
    """Text as an array of numbers: its bytes in a buffer that is the same length whatever the text's."""
    raw = text.encode()
    held[:len(raw)] = np.frombuffer(raw, np.uint8)
    return held


def _run_word(s):
    lo, hi, addr = s["lo"], s["hi"], s["case"]["addr"]
    d = codec().decode(lo, hi, addr)
    text = codec().to_sass(lo, hi, addr)
    again = codec().encode(text, addr)
    s["fields"][:len(d["fields"])] = [(f["shift"], f["bits"], f["value"]) for f in d["fields"]]
    sched = np.array([int(v) for v in d["scheduling"].values()], np.int64)
    names = _place(s["names"], d["key"] + " " + d["mod_group"] + " " + d["opcode"])
    return _signed(s["fields"]), sched, names, _place(s["text"], text), _signed(np.array(again, np.uint64))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "word":
        return _run_word(s)
    if kind == "decode":
        counts = codec().decode_device(s["words"].data_ptr(), case["n"], s["form"].data_ptr(), s["slots"].data_ptr(),
                                       s["ctrl"].data_ptr(), _stream(), case["counts"])
        return s["form"], s["slots"], s["ctrl"], counts
    if kind == "encode":
        codec().encode_device(s["form"].data_ptr(), s["slots"].data_ptr(), s["ctrl"].data_ptr(), case["n"],
                              s["words"].data_ptr(), _stream())
        return s["words"]
    if kind == "roundtrip":
        counts = codec().roundtrip_device(s["words"].data_ptr(), case["n"], s["status"].data_ptr(), _stream(), case["counts"])
        return s["status"], counts
    if kind == "host":
        if case["call"] == "encode":
            return codec().encode_batch(s["form"], s["slots"], s["ctrl"])
        if case["call"] == "roundtrip":
            return codec().roundtrip_batch(s["words"])
        form, slots, ctrl, counts = codec().decode_batch(s["words"])
        return _signed(form), _signed(slots), _signed(ctrl), counts
    if kind == "cubin":
        sections, start, form, slots, ctrl, raw, counts = codec().decode_elf(s["image"])
        return _signed(start), _signed(form), _signed(slots), _signed(ctrl), raw, counts
    if kind == "listing":
        text, n_raw = codec().disassemble(s["image"], frozen=case["frozen"], want_raw_count=True)
        return _place(s["text"], text), n_raw
    return codec().encode_text(s["text"])


def work(case):
    """Bytes that a pass reads and writes at least once: a word is 16 bytes, a record 38, a status 1, a line of text about 64.
    Nothing here is floating-point work."""
    kind, call = case["kind"], case.get("call", case["kind"])
    n = sum(kernel_lengths(case)) if kind == "cubin" else case.get("n", 1)
    each = {"decode": 54, "encode": 54, "roundtrip": 17, "cubin": 16 + 38 + 16, "listing": 16 + 64, "assemble": 64 + 16,
            "word": 16 + 38 + 64 + 16}[call]
    return {"bytes": each * n, "flops": 0}


def tolerance(case):
    return "exact"
