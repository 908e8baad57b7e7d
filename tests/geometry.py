"""The library's launch geometry (flint_b200/csrc/fb_geometry.hpp: plain C++, no CUDA) compiled for the host, so that a test can say which kernel a
call takes and fails when a changed rule takes it elsewhere."""
import ctypes
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_SHIM = """
#include "fb_geometry.hpp"
extern "C" void gemm(int M, int rows, int k, int zeros, int sms, int* o) {
  const fb::GemmGeometry g = fb::gemm_geometry(M, rows, k, zeros != 0, sms);
  o[0] = g.nt; o[1] = g.ntok; o[2] = g.ntile; o[3] = g.nsplit;
}
extern "C" void attn(int M, int pos, int n_kv, int r, int sms, int* o) {
  const fb::AttnGeometry a = fb::attn_geometry(M, pos, n_kv, r, sms);
  o[0] = a.rt; o[1] = a.groups; o[2] = a.nspan; o[3] = a.span;
}
extern "C" int tile_rt(int k) { return fb::tile_rt(k); }
extern "C" int cta_first_row(int rows, int unit, int b, int G) { return fb::cta_first_row(rows, unit, b, G); }
extern "C" void window(int width, int rank, int* o) {
  const fb::OWindow w = fb::o_window(width, rank);
  const fb::WordPairs p = fb::o_words(width, w.off);
  o[0] = w.ko; o[1] = w.off; o[2] = p.first; o[3] = p.end;
}
static const int kShapes[][5] = {
#define FB_DECODE_ENTRY(KD, KO, KF, HD, R) {KD, KO, KF, HD, R}
#include "fb_decode_shapes.h"
};
extern "C" int shapes(const int** o) { *o = &kShapes[0][0]; return (int)(sizeof(kShapes) / sizeof(kShapes[0])); }
extern "C" int draft(int blocks, int chunks, int nt, int sms) { return fb::draft_splits(blocks, chunks, nt, sms); }
"""
_lib = None


def _load():
    global _lib
    if _lib is None:
        with tempfile.TemporaryDirectory() as d:
            src, so = os.path.join(d, "geometry.cpp"), os.path.join(d, "geometry.so")
            with open(src, "w") as f:
                f.write(_SHIM)
            subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "flint_b200", "csrc"), "-o", so, src])
            _lib = ctypes.CDLL(so)
    return _lib


def _four(fn, *args):
    o = (ctypes.c_int * 4)()
    fn(*args, o)
    return tuple(o)


def gemm(M, rows, k, zeros=False, sms=148):
    """(tile, tokens of a tile, tiles, CTAs that share K)"""
    return _four(_load().gemm, M, rows, k, int(zeros), sms)


def matrices(cfg, M, asym=False, sms=148):
    """The same for the five matrices of a model."""
    d, ko, f = cfg.dim, cfg.n_head * cfg.head_dim, cfg.ffn_padded
    return {n: gemm(M, rows, k, asym, sms) for n, rows, k in (("qkv", cfg.qkv_rows, d), ("o", d, ko), ("gu", 2 * f, d), ("d", d, f),
                                                               ("lm", cfg.vocab_size, d))}


def attn(M, pos, n_kv, r, sms=148):
    """(row tiles of a CTA, row groups, spans, positions of a span)"""
    return _four(_load().attn, M, pos, n_kv, r, sms)


def draft(rows, k, T, pair=False, sms=148):
    """CTAs that share K in a draft linear over T tokens (at most 32); rows: the rows of its one to three matrices; pair: gate and up together."""
    nt = 1 if T <= 8 else (2 if T <= 16 else 4)
    per = 16 if nt == 1 or pair else 32
    return _load().draft(sum(-(-r // per) for r in rows), -(-k // 32), nt, sms)


def decode_shapes():
    """(model width, O columns of a rank, FFN width of a rank, head dimension, query heads per kv head) of every decode kernel"""
    p = ctypes.POINTER(ctypes.c_int)()
    n = _load().shapes(ctypes.byref(p))
    return [tuple(p[5 * i:5 * i + 5]) for i in range(n)]


def tile_rt(k):
    return _load().tile_rt(k)


def cta_rows(rows, unit, sms=148):
    """First and end row of every CTA's share of a decode phase"""
    at = [_load().cta_first_row(rows, unit, b, sms) for b in range(sms + 1)]
    return list(zip(at[:-1], at[1:]))


def o_window(width, rank):
    """(columns of the O projection that a rank reads, where its own start in them, first and end pair of tagged words of its own)"""
    return _four(_load().window, width, rank)
