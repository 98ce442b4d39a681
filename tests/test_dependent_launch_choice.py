"""Which launches a driver with two contexts makes (csrc/lstm_rec_api.h): the caller's choice of dependent launches holds for both of them, whichever it is, and the
driver's own rule where there is none; both contexts are left as they were found. Built with a stand-in for the library's setting."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "dynet_b200" / "csrc"
CODE = r"""
#include "lstm_rec_api.h"
#include <cstdio>
struct dyb200_ctx { int pdl, chosen; };
extern "C" int dyb200i_dependent_launch(dyb200_ctx* c, int set) {   /* as the library's: a setting that the caller has chosen stays */
  const int was = c->pdl;
  if (set >= 0 && !c->chosen) c->pdl = set;
  return was;
}
int main() {
  for (int chosen = 0; chosen < 2; ++chosen)
    for (int pdl = 0; pdl < 2; ++pdl)
      for (int rule = 0; rule < 2; ++rule) {
        dyb200_ctx caller = {pdl, chosen}, own = {1, 0};
        const int want = chosen ? pdl : rule;
        {
          const dyb200i_both_launches in_force(&caller, &own, rule);
          if (caller.pdl != want || own.pdl != want) { printf("chosen %d (%d), rule %d: %d %d\n", chosen, pdl, rule, caller.pdl, own.pdl); return 1; }
        }
        if (caller.pdl != pdl || own.pdl != 1) { printf("not put back\n"); return 1; }
      }
  return 0;
}
"""


def test_the_callers_choice_holds_for_both_contexts(tmp_path):
    (tmp_path / "t.cc").write_text(CODE)
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-o", str(tmp_path / "t"), str(tmp_path / "t.cc"), "-I", str(CSRC)])
    p = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout


def test_the_tagger_goes_by_it():
    text = (CSRC.parent / "host" / "tagger.cc").read_text()
    assert text.count("dyb200i_both_launches ") == 1 and "dyb200i_ordinary_launches second" not in text
