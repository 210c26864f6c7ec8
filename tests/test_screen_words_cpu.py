"""A screen's list items name their table word in 3 bits, relative to the first
word of the listing CTA's share: whatever the number of SMs, the planned words
leave every share within 8 words."""
import random

import pytest


@pytest.mark.parametrize("sms", [1, 18, 60, 108, 109, 110, 152])
def test_words_of_a_share(P, built, sms):
    rng = random.Random(sms)
    planned = []
    for spacer, pam, guides, mm in ((20, "NGG", 5000, 4), (20, "NGG", 700, 8), (24, "NNGRRT", 40, 5)):
        text = f"g\n{'N' * spacer}{pam}\n" + "".join(
            "".join(rng.choice("ACGT") for _ in range(spacer)) + "N" * len(pam) + f" {mm}\n" for _ in range(guides))
        for level in range(-1, 9):
            s = P.screen_plan(text, level, sms)
            if s is None:
                continue
            planned.append(s["words"])
            # The shares of the launch's CTAs: `spans` warp shares per word, word by word.
            for spans in (1, 2, 3, 64, 997, 1 << 20):
                total = spans * s["words"]
                for b in range(sms):
                    begin, end = total * b // sms, total * (b + 1) // sms
                    if begin < end:
                        assert (end - 1) // spans - begin // spans <= 7, (guides, level, s["words"], spans, b)
    assert planned
    assert max(planned) > 4 * min(sms, 100)  # large screens are still planned
