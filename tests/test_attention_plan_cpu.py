"""How a decode attention launch is laid out (scratchy_b200/csrc/attention_plan.h), compiled for the host."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scratchy_b200", "csrc")
SMS = 148


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    folder = tmp_path_factory.mktemp("plan")
    source, library = folder / "plan.cpp", folder / "plan.so"
    source.write_text('#include "attention_plan.h"\nextern "C" AttPlan plan(int d, int g, int b, int h, int bs, int mb) '
                      f'{{ return att_plan(d, g, b, h, bs, mb, {SMS}); }}\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", library, source], check=True)

    class Plan(ctypes.Structure):
        _fields_ = [(n, ctypes.c_int) for n in ("nsplit", "warps", "stages", "table_cap")] + [("fixed", ctypes.c_size_t)]
    call = ctypes.CDLL(str(library)).plan
    call.restype = Plan
    return lambda d, g, batch, heads, block, blocks: call(d, g, batch, heads, block, blocks)


@pytest.mark.parametrize("d,block", [(128, 16), (64, 16), (128, 32), (128, 48), (64, 64), (128, 128)])
@pytest.mark.parametrize("g", range(1, 9))
@pytest.mark.parametrize("batch,heads", [(1, 8), (2, 8), (16, 8), (32, 8), (20, 4), (64, 8)])
def test_as_many_warps_as_fit(plan, d, block, g, batch, heads):
    """No smaller number of warps than another that has its two stages each in the same shared memory."""
    for tokens in (block, 640, 1040, 2048, 4112, 16384):
        p = plan(d, g, batch, heads, block, -(-tokens // block))
        alone = 2 * batch * heads * p.nsplit <= SMS
        room = (200 if alone else 110) * 1024 - p.fixed
        two = lambda warps: 4 * (block * d * 2) * warps <= room
        assert p.warps in ((8, 4, 2) if alone else (6, 4, 2)) and p.stages <= 3
        assert p.warps * p.stages * 2 * block * d * 2 <= room
        assert p.warps >= 4 or not two(4), (tokens, p.warps)
        assert p.stages >= 2 or not two(2)


@pytest.mark.parametrize("block", [16, 32, 48, 256])
def test_the_width_of_the_table_cuts_no_sequence(plan, block):
    """The table's width is a capacity (a server captures its step once): the cut follows the number of sequences alone."""
    for batch in range(1, 130):
        fits = [n for n in (8, 4, 2, 1) if batch * 8 * n <= 2 * SMS or n == 1][0]
        for tokens in (256, 1024, 1536, 2048, 5000, 32768):
            p = plan(128, 3, batch, 8, block, -(-tokens // block))
            assert p.nsplit == fits and p.table_cap >= -(-(-(-tokens // block)) // fits)


def test_sequences_are_dealt_evenly_to_bins_that_fit(tmp_path):
    """The packed layout: every sequence has a place, the shared memory of a CTA suffices, and falling lengths dealt back and forth leave no CTA
    with more than the mean, the longest sequence and the spread of one round allow."""
    source, library = tmp_path / "bins.cpp", tmp_path / "bins.so"
    source.write_text('#include "attention_plan.h"\nextern "C" AttBins bins(int d, int g, int b, int h, int bs, int mb, int split) '
                      f'{{ return att_bins(d, g, b, h, bs, mb, {SMS}, split); }}\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", library, source], check=True)

    class Bins(ctypes.Structure):
        _fields_ = [(n, ctypes.c_int) for n in ("bins", "items", "warps", "stages", "table_cap")] + [("smem", ctypes.c_size_t)]
    call = ctypes.CDLL(str(library)).bins
    call.restype = Bins
    for batch in range(1, 80):
        for g in range(1, 9):
            for block, blocks in ((16, 128), (32, 64), (16, 2048), (128, 16)):
                p = call(128, g, batch, 8, block, blocks, 1)
                if not p.items:
                    continue
                assert p.bins * 8 <= SMS and p.bins < batch <= p.bins * p.items and p.items <= 4
                assert p.stages >= 2 * p.warps and p.smem <= 227 * 1024 and p.table_cap >= p.items * blocks
                lens = sorted(((7919 * (i + g)) % 1500 + 500 for i in range(batch)), reverse=True)
                load, rounds = [0] * p.bins, -(-batch // p.bins)
                for r, n in enumerate(lens):
                    at = r % p.bins
                    load[p.bins - 1 - at if (r // p.bins) & 1 else at] += n
                assert max(load) <= max(lens[0], sum(load) / p.bins) + lens[0] - lens[-1]
    assert not call(128, 3, 32, 8, 16, 128, 2).items and not call(128, 3, 18, 8, 16, 128, 1).items and not call(128, 3, 73, 8, 16, 128, 1).items


def test_packed_layout_leaves_room_for_the_static_arrays(tmp_path):
    """A CTA may have 227 KB, dynamic and static together: no layout asks for more, at any width of the table."""
    source, library = tmp_path / "bins.cpp", tmp_path / "bins.so"
    source.write_text('#include "attention_plan.h"\nextern "C" size_t most(int d, int g, int b, int bs, int from, int to) {\n'
                      '    size_t most = 0;\n    for (int mb = from; mb < to; ++mb) {\n'
                      f'        const AttBins p = att_bins(d, g, b, 8, bs, mb, {SMS}, 1);\n        if (p.items && p.smem > most) most = p.smem;\n    }}\n    return most;\n}}\n'
                      'extern "C" size_t fixed_part() { return sizeof(AttMergeShared) + sizeof(AttShared); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", library, source], check=True)
    call = ctypes.CDLL(str(library))
    call.most.restype = call.fixed_part.restype = ctypes.c_size_t
    seen = 0
    for d in (64, 128):
        for g in range(1, 9):
            for batch in (20, 36, 38, 40, 44, 48, 52, 54, 55, 72):
                for block in (16, 32):
                    most = call.most(d, g, batch, block, 1, 12000)
                    assert most + call.fixed_part() <= 227 * 1024, (d, g, batch, block, most)
                    seen += most > 220 * 1024
    assert seen > 50


def test_packed_only_where_single_sequences_would_start_a_second_round(tmp_path):
    source, library = tmp_path / "bins.cpp", tmp_path / "bins.so"
    source.write_text('#include "attention_plan.h"\nextern "C" int items(int g, int b, int h, int mb) {\n'
                      f'    return att_bins(128, g, b, h, 16, mb, {SMS}, att_plan(128, g, b, h, 16, mb, {SMS}).nsplit).items;\n}}\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", library, source], check=True)
    items = ctypes.CDLL(str(library)).items
    for heads in (1, 2, 4, 8, 16):
        for blocks in (8, 128, 512):
            for batch in range(1, 500):
                one_round, three = batch * heads <= 2 * SMS, batch <= 3 * (SMS // heads)
                assert (items(3, batch, heads, blocks) > 0) == (three and not one_round), (heads, batch)
    source.write_text('#include "attention_plan.h"\nextern "C" int items(int g, int b, int h, int mb) {\n'
                      f'    return att_bins(64, g, b, h, 16, mb, {SMS}, 1).items;\n}}\n')
    narrow = tmp_path / "narrow.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", narrow, source], check=True)
    heads64 = ctypes.CDLL(str(narrow)).items                  # three CTAs to an SM up to 23 blocks, two beyond
    assert heads64(4, 48, 8, 19) == 0 and heads64(4, 48, 8, 63) == 3 and heads64(4, 37, 8, 63) == 0
    assert items(3, 37, 8, 128) == 0 and items(3, 38, 8, 128) == 3 and items(3, 54, 8, 128) == 3 and items(3, 55, 8, 128) == 0
