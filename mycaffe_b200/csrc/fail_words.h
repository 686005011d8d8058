// Failure words in pinned host memory, visible to every device: a kernel that writes a failure into its device's status
// words also raises the word of its family in that device's row here, so that a synchronous call learns from a plain host
// load behind its one stream synchronisation that nothing failed.  (Copying the status words back after every call cost a
// 3 us transfer and its launch on each.)  A device's kernels know their row's address by a symbol of each translation
// unit, set when a kernel index is initialised; null (raw callers) means no word is raised.
// The rows are per device because the status words are: a call lowers a word before it reads the status array behind it, and
// the array it reads is its own device's.
#pragma once

enum McaFailWord : int { MCA_FAIL_TC = 0, MCA_FAIL_DECODE = 1, MCA_FAIL_PROJ = 2, MCA_FAIL_WORDS = 4 };
constexpr int MCA_FAIL_DEVICES = 64;

struct McaFailTable {
  int* words = nullptr;   // MCA_FAIL_DEVICES rows of MCA_FAIL_WORDS, or null
  static constexpr int SIZE = MCA_FAIL_DEVICES * MCA_FAIL_WORDS;
  int* row(int device) const { return words + device * MCA_FAIL_WORDS; }
  bool raised(int device, McaFailWord family) const { return *static_cast<volatile int*>(row(device) + family) != 0; }
  void lower(int device, McaFailWord family) const { *static_cast<volatile int*>(row(device) + family) = 0; }
};
