// The host's wait for handed-over words (wrapd_b200/csrc/hand_over.hpp).
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>

#include "../../wrapd_b200/csrc/hand_over.hpp"

using Word = unsigned long long;
static const Word U = 0x7ff45a5a5a5a5a5aull;
static int failures = 0;
static void expect(bool ok, const char* what) {
    if (!ok) { std::printf("FAILED: %s\n", what); ++failures; }
}

int main() {
    // all there: taken without asking whether the writer has ended
    {
        const Word in[3] = {1, 0, ~0ull};
        Word out[3] = {U, U, U};
        int asked = 0;
        expect(wrapd::take_words(in, 3, U, out, [&] { ++asked; return false; }) && asked == 0, "set words");
        expect(out[0] == 1 && out[1] == 0 && out[2] == ~0ull, "set words' values");
    }
    // a word that never comes, first, in the middle and last: reported, not returned as a value
    for (int miss = 0; miss < 3; ++miss) {
        Word in[3] = {5, 6, 7}, out[3] = {0, 0, 0};
        in[miss] = U;
        expect(!wrapd::take_words(in, 3, U, out, [] { return true; }), "missing word");
        expect(out[miss] != U, "missing word is not handed on");
    }
    // a word that the writer stores as its last act: found after it has ended
    {
        volatile Word in[2] = {3, U};
        Word out[2] = {0, 0};
        int asked = 0;
        const bool ok = wrapd::take_words(in, 2, U, out, [&] { if (++asked == 3) in[1] = 9; return asked == 3; });
        expect(ok && out[1] == 9 && asked == 3, "word stored just before the end");
    }
    // words stored one by one, backwards, by another thread
    {
        volatile Word in[8];
        for (auto& w : in) w = U;
        std::atomic<bool> over{false};
        std::thread t([&] {
            for (int k = 7; k >= 0; --k) {
                std::this_thread::sleep_for(std::chrono::milliseconds(1));
                in[k] = 100 + k;
            }
            over = true;
        });
        Word out[8];
        expect(wrapd::take_words(in, 8, U, out, [&] { return over.load(); }), "words stored later");
        t.join();
        for (int k = 0; k < 8; ++k) expect(out[k] == Word(100 + k), "values stored later");
    }
    // an error that the question raises ends the wait
    {
        const Word in[1] = {U};
        Word out[1];
        bool thrown = false;
        try {
            wrapd::take_words(in, 1, U, out, []() -> bool { throw 1; });
        } catch (int) {
            thrown = true;
        }
        expect(thrown, "error of the writer");
    }
    if (failures == 0) std::printf("ok\n");
    return failures != 0;
}
